// Launchers of the 3D kernels (included by the ops_*.cu units).
#pragma once
#include "dg3d_kernels.cuh"
#include "ops_2d.cuh"

template <class Phys, int n>
struct OpsImpl3D {
  using S = ElemSmem3D<Phys, n>;
  static int interface(tag_handle h, const double* u) {
    const int total = (h->nif + h->nbd) * n * n;
    if (total == 0) return TAG_OK;
    const int threads = interface_threads(total);
    TAG_CUDA(launch_overlapped(
        h->overlap(), k_interface3d<Phys, n>, (total + threads - 1) / threads, threads, 0,
        h->stream, params_of<Phys>(h), u, h->d_Ja, h->d_invJ, h->d_if_e, h->d_if_f, h->d_if_flip,
        h->nif, h->d_bd_e, h->d_bd_f, h->nbd, h->d_sfv));
    return TAG_OK;
  }
  static int element(tag_handle h, int mode, double* u, double* du, int stage, bool last,
                     double) {
    const int epb = h->epb > 0 ? h->epb : 1;
    const int blocks = (h->nelem + epb - 1) / epb;
    const int threads = launch_threads(h);
    const size_t smem = S::bytes(epb);
    StageArgs st{};
    st.member = h->d_member;
    if (mode == kModeStage) {
      set_stage(st, h->scheme, stage);
      st.dt = h->d_mscal + h->nmembers;
      st.max_speed = last ? h->d_mscal + 2 * h->nmembers : nullptr;
      st.sink = last && h->capturing_steps ? h->sink : nullptr;
      TAG_CUDA(launch_overlapped(h->overlap(), element3d_kernel<Phys, n, kModeStage>(), blocks, threads,
                                 smem, h->stream, params_of<Phys>(h), h->basis, u, du, h->d_k,
                                 h->d_Ja, h->d_invJ, h->d_sfv, h->nelem, epb, st, h->d_status));
    } else {
      TAG_CUDA(launch_overlapped(h->overlap(), element3d_kernel<Phys, n, kModeRhs>(), blocks, threads,
                                 smem, h->stream, params_of<Phys>(h), h->basis, u, du, h->d_k,
                                 h->d_Ja, h->d_invJ, h->d_sfv, h->nelem, epb, st, h->d_status));
    }
    return TAG_OK;
  }
  static int max_speed(tag_handle h, const double* u) { return speeds(h, u, nullptr); }
  // the state from mapped host memory into the device copy, speeds on the way
  static int load_state(tag_handle h, const double* u_mapped) {
    return speeds(h, u_mapped, h->d_u);
  }
  static int speeds(tag_handle h, const double* u, double* copy_to) {
    const int threads = 256, warps = threads / 32;  // one warp per element
    k_max_speed3d<Phys, n><<<(h->nelem + warps - 1) / warps, threads, 0, h->stream>>>(
        params_of<Phys>(h), u, h->d_Ja, h->d_invJ, h->nelem, h->d_member,
        h->d_mscal + 2 * h->nmembers, copy_to);
    TAG_CUDA(cudaGetLastError());
    return TAG_OK;
  }
  static int init(int max_smem) {
    TAG_CUDA(cudaFuncSetAttribute(element3d_kernel<Phys, n, kModeStage>(),
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem));
    TAG_CUDA(cudaFuncSetAttribute(element3d_kernel<Phys, n, kModeRhs>(),
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem));
    return launch_thread_cap(element3d_kernel<Phys, n, kModeStage>(), element3d_kernel<Phys, n, kModeRhs>(),
                             cap());
  }
  static int& cap() {
    static int c = 1024;
    return c;
  }
  static int max_threads() { return 1024; }  // of a tile; the kernel strides over its work
  static int launch_threads(tag_handle h) {
    return std::min(cap(), tile_threads((h->epb > 0 ? h->epb : 1) * S::TPE, h->tile_div));
  }
  static size_t smem_bytes(int epb) { return S::bytes(epb); }
  static const Ops* get() {
    static const Ops ops{&interface, &element, &max_speed, &load_state, &init, &smem_bytes,
                         S::TPE, &max_threads, &launch_threads};
    return &ops;
  }
};

template <class Phys>
const Ops* ops3d_for_n(int n) {
  switch (n) {
    case 3: return OpsImpl3D<Phys, 3>::get();
    case 4: return OpsImpl3D<Phys, 4>::get();
    case 5: return OpsImpl3D<Phys, 5>::get();
    case 6: return OpsImpl3D<Phys, 6>::get();
    case 7: return OpsImpl3D<Phys, 7>::get();
    case 8: return OpsImpl3D<Phys, 8>::get();
    default: return nullptr;
  }
}
