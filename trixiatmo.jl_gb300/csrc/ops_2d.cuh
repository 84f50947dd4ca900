// Launchers of the 2D Cartesian kernels (included by the ops_*.cu units).
#pragma once
#include "dg2d_kernels.cuh"
#include "handle.cuh"

// Largest multiple of 32 threads both element kernels (stage and rhs mode) of
// one instantiation can be launched with.
template <class K1, class K2>
int launch_thread_cap(K1 k1, K2 k2, int& cap) {
  cudaFuncAttributes a, b;
  TAG_CUDA(cudaFuncGetAttributes(&a, k1));
  TAG_CUDA(cudaFuncGetAttributes(&b, k2));
  cap = (std::min(a.maxThreadsPerBlock, b.maxThreadsPerBlock) / 32) * 32;
  return TAG_OK;
}

template <class Phys>
const typename Phys::Params& params_of(tag_handle h);
template <>
inline const PhysEnergy2D::Params& params_of<PhysEnergy2D>(tag_handle h) {
  return h->p_energy;
}
template <>
inline const PhysEnergy3D::Params& params_of<PhysEnergy3D>(tag_handle h) {
  return h->p_energy3d;
}
template <>
inline const PhysRainy2D::Params& params_of<PhysRainy2D>(tag_handle h) {
  return h->p_rainy;
}
template <>
inline const PhysMoist2D::Params& params_of<PhysMoist2D>(tag_handle h) {
  return h->p_moist;
}
template <>
inline const PhysPT2D::Params& params_of<PhysPT2D>(tag_handle h) {
  return h->p_pt;
}
template <>
inline const PhysPT3D::Params& params_of<PhysPT3D>(tag_handle h) {
  return h->p_pt3d;
}
template <>
inline const PhysIE2D::Params& params_of<PhysIE2D>(tag_handle h) {
  return h->p_ie;
}

template <class Phys, int n, int VOL = kVolFluxDiff>
struct OpsImpl {
  using S = ElemSmem<Phys, n>;
  static int interface(tag_handle h, const double* u) {
    const int total = (h->nif + h->nbd) * n;
    if (total == 0) return TAG_OK;
    const int threads = interface_threads(total);
    if (h->need_bvals && !h->bvals_set)
      return fail(TAG_E_INVALID, "Dirichlet boundary faces without states (tag_set_boundary_values)");
    TAG_CUDA(launch_overlapped(
        h->overlap(), k_interface<Phys, n>, (total + threads - 1) / threads, threads, 0, h->stream,
        params_of<Phys>(h), u, h->d_Ja, h->d_invJ, h->d_if_e, h->d_if_f, h->d_if_flip, h->nif,
        h->d_bd_e, h->d_bd_f, h->d_bd_kind, h->nbd, h->d_sfv, h->d_bvals));
    return TAG_OK;
  }
  static int element(tag_handle h, int mode, double* u, double* du, int stage, bool last,
                     double t) {
    const int epb = h->epb > 0 ? h->epb : 4;
    const int blocks = (h->nelem + epb - 1) / epb;
    const int threads = launch_threads(h);
    const size_t smem = S::bytes(epb);
    StageArgs st{};
    st.member = h->d_member;
    st.xy = h->d_xy;
    st.t_rhs = t;
    if (mode == kModeStage) {
      set_stage(st, h->scheme, stage);
      st.t_member = h->d_mscal;
      st.dt = h->d_mscal + h->nmembers;
      st.max_speed = last ? h->d_mscal + 2 * h->nmembers : nullptr;
      st.sink = last && h->capturing_steps ? h->sink : nullptr;
      TAG_CUDA(launch_overlapped(h->overlap(), k_element<Phys, n, kModeStage, VOL>, blocks, threads,
                                 smem, h->stream, params_of<Phys>(h), h->basis, u, du, h->d_k,
                                 h->d_Ja, h->d_invJ, h->d_sfv, h->nelem, epb, st, h->d_status));
    } else {
      TAG_CUDA(launch_overlapped(h->overlap(), k_element<Phys, n, kModeRhs, VOL>, blocks, threads,
                                 smem, h->stream, params_of<Phys>(h), h->basis, u, du, h->d_k,
                                 h->d_Ja, h->d_invJ, h->d_sfv, h->nelem, epb, st, h->d_status));
    }
    return TAG_OK;
  }
  static int max_speed(tag_handle h, const double* u) {
    using K = MaxSpeedTile<n>;
    k_max_speed<Phys, n><<<(h->nelem + K::EPB - 1) / K::EPB, K::T, 0, h->stream>>>(
        params_of<Phys>(h), u, h->d_Ja, h->d_invJ, h->nelem, h->d_member,
        h->d_mscal + 2 * h->nmembers);
    TAG_CUDA(cudaGetLastError());
    return TAG_OK;
  }
  // opt the element kernels into the device's full dynamic shared memory once,
  // outside any stream capture
  static int init(int max_smem) {
    TAG_CUDA(cudaFuncSetAttribute(k_element<Phys, n, kModeStage, VOL>,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem));
    TAG_CUDA(cudaFuncSetAttribute(k_element<Phys, n, kModeRhs, VOL>,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem));
    return launch_thread_cap(k_element<Phys, n, kModeStage, VOL>, k_element<Phys, n, kModeRhs, VOL>,
                             cap());
  }
  static int& cap() {
    static int c = 1024;
    return c;
  }
  static int max_threads() { return cap(); }
  static int launch_threads(tag_handle h) {
    return std::min(cap(), cta_threads((h->epb > 0 ? h->epb : 4) * S::TPE, h->tile_div));
  }
  static size_t smem_bytes(int epb) { return S::bytes(epb); }
  static const Ops* get() {
    static const Ops ops{&interface, &element, &max_speed, nullptr, &init, &smem_bytes,
                         S::TPE, &max_threads, &launch_threads};
    return &ops;
  }
};

template <class Phys, int VOL = kVolFluxDiff>
const Ops* ops_for_n(int n) {
  switch (n) {
    case 2: return OpsImpl<Phys, 2, VOL>::get();
    case 3: return OpsImpl<Phys, 3, VOL>::get();
    case 4: return OpsImpl<Phys, 4, VOL>::get();
    case 5: return OpsImpl<Phys, 5, VOL>::get();
    case 6: return OpsImpl<Phys, 6, VOL>::get();
    case 7: return OpsImpl<Phys, 7, VOL>::get();
    case 8: return OpsImpl<Phys, 8, VOL>::get();
    default: return nullptr;
  }
}
