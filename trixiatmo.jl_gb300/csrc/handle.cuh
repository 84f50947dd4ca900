// The handle behind the C ABI and the launchers of one equation system's
// kernels.  The kernels of each system are compiled in a unit of their own
// (ops_*.cu), so that the build runs them in parallel.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <string>

#include "cov_params.cuh"
#include "dg2d_kernels.cuh"
#include "newton_rainy.cuh"
#include "phys_euler_energy_2d.cuh"
#include "phys_euler_energy_3d.cuh"
#include "phys_ie_2d.cuh"
#include "phys_moist_2d.cuh"
#include "phys_pt_2d.cuh"
#include "phys_pt_3d.cuh"
#include "phys_rainy_2d.cuh"

inline int fail(int code, const std::string& msg) {
  tag::set_last_error(msg);
  return code;
}

#define TAG_CUDA(call)                                                                    \
  do {                                                                                    \
    cudaError_t err_ = (call);                                                            \
    if (err_ != cudaSuccess)                                                              \
      return fail(TAG_E_CUDA, std::string(#call) + ": " + cudaGetErrorString(err_));      \
  } while (0)

using namespace tag;

struct Ops;

// Threads of an element-kernel CTA: `items` work items split `div` ways,
// rounded up to whole warps.
inline int cta_threads(int items, int div) { return ((items + div - 1) / div + 31) / 32 * 32; }
// Threads of an interface-kernel CTA for `total` interface nodes: the largest of
// 256 to 32 that still gives each of the 152 SMs a CTA.  A small mesh's few CTAs
// of 256 would queue eight warps on one SM's FP64 pipe and leave the others idle:
// 60 x 8 elements, polydeg 3 (3,936 nodes): 80 stages 1.68 ms with 16 CTAs of
// 256, 1.60 ms with 123 of 32; dry 64 x 32 elements, 100 stages: 2.17 -> 2.01 ms.
inline int interface_threads(long total) {
  int t = 256;
  while (t > 32 && total <= 152L * t) t /= 2;
  return t;
}
// Meshes whose stages are overlapped launches: a stage is two dependent kernels
// of 5 to 13 us each on a mesh this small, and the gap between them and the
// loads of geometry are a fifth of it.  Measured, launches in order against
// overlapped: 10 to 20 steps of 3,840 nodes (potential temperature) 1.60 -> 1.37
// ms, 15,840 (dry) 1.87 -> 1.77 ms, shallow water 24,576 nodes 0.93 -> 0.87 ms;
// above, CTAs that start early fill the SMs unevenly: 32,768 nodes 1.97 -> 2.01
// ms, 131,072 nodes 4.65 -> 5.07 ms.
constexpr long kOverlapNodes = 24576;

// Launches a kernel that, with `overlap`, may start before the stream's previous
// kernel has ended (it waits for it by wait_for_previous).
template <class Kernel, class... Args>
cudaError_t launch_overlapped(bool overlap, Kernel kernel, int blocks, int threads, size_t smem,
                              cudaStream_t stream, Args&&... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = dim3(blocks);
  c.blockDim = dim3(threads);
  c.dynamicSmemBytes = smem;
  c.stream = stream;
  c.attrs = &attr;
  c.numAttrs = overlap ? 1 : 0;
  return cudaLaunchKernelEx(&c, kernel, std::forward<Args>(args)...);
}
// Tiles of the 3D kernels: div 1 to 3 as above; 4 to 6 the same rounded up to
// whole groups of four warps, one for each of the SM's sub-partitions (their
// registers are separate, so an odd warp can cost a CTA's place on all four).
inline int tile_threads(int items, int div) {
  const int t = cta_threads(items, div > 3 ? div - 3 : div);
  return div > 3 ? (t + 127) / 128 * 128 : t;
}

struct tag_handle_s {
  int eq = 0, n = 0, nelem = 0, nif = 0, nbd = 0, nv = 0, na = 0;
  int dim = 2, npe = 0, nface = 4, jpn = 4;  // nodes per element, faces, Ja doubles per node
  long nodes = 0;                            // solution nodes (all elements)
  int dt_n = 0;                              // n in dt = cfl 2 / (n max_speed); 1 when
                                             // the kernels reduce n-scaled speeds
  // covariant equations: element groups, geometry, packed element data
  CovParams p_cov{};

  CovGroups h_groups{};
  CovGroups* d_groups = nullptr;
  BasisDev* d_bases = nullptr;
  double *d_aux = nullptr, *d_pk = nullptr, *d_ipk = nullptr;
  long cov_if_nodes = 0;  // interface nodes packed in d_ipk
  int cov_blocks = 0, cov_iblocks = 0, cov_threads = 0;
  size_t cov_smem = 0;
  PhysEnergy2D::Params p_energy{};
  PhysEnergy3D::Params p_energy3d{};
  PhysRainy2D::Params p_rainy{};
  PhysMoist2D::Params p_moist{};
  PhysPT2D::Params p_pt{};
  PhysPT3D::Params p_pt3d{};
  PhysIE2D::Params p_ie{};
  // rainy: Newton stage limiter settings, MLP parameters, statistics counters
  bool has_limiter = false;
  int scheme = TAG_RK_CK2N54;  // time integrator of tag_rk_steps
  NewtonArgs newton{0, 20, 0, 0, 8, 1e-9, nullptr, nullptr, nullptr};
  float* d_mlp = nullptr;
  unsigned long long* d_counters = nullptr;
  int* d_iters = nullptr;
  // the stage limiter inside tag_rk_steps: its start (NewtonArgs::learned)
  // and counters accumulated over the run ([0] updates, [1] fallbacks,
  // [2] not converged), with the number of node solves they cover
  int newton_start = 0;
  unsigned long long* d_run_counters = nullptr;
  long long run_node_solves = 0;
  BasisDev basis{};
  cudaStream_t stream = nullptr;
  double *d_u = nullptr, *d_k = nullptr, *d_Ja = nullptr, *d_invJ = nullptr, *d_xy = nullptr,
         *d_sfv = nullptr, *d_tmp_u = nullptr, *d_tmp_du = nullptr;
  // adaptive SSPRK43: the stage value entering the last stage, error partials
  double *d_u3 = nullptr, *d_err = nullptr;
  int *d_if_e = nullptr, *d_if_f = nullptr, *d_if_flip = nullptr, *d_bd_e = nullptr,
      *d_bd_f = nullptr, *d_bd_kind = nullptr;
  // states of the TAG_BC_DIRICHLET faces [B][n][nv] (allocated when the mesh has
  // such faces; the interface kernel reads them)
  double* d_bvals = nullptr;
  bool need_bvals = false, bvals_set = false;
  int nmembers = 1;
  int* d_member = nullptr;        // [E] or null
  double* d_mscal = nullptr;      // [3 * nmembers]: t, dt, max_speed
  StepCtl* d_ctl = nullptr;
  double* h_pin = nullptr;        // pinned staging, 3 * nmembers + 2 doubles
  unsigned* d_status = nullptr;
  cudaGraphExec_t graph = nullptr;
  int graph_epb = -1;
  // 3D: mapped host array that the last stage of every tag_rk_steps step also
  // stores the new state into (tag_set_state_sink); armed only while the step
  // graph is captured, so that no other stage sequence writes it
  double* sink = nullptr;
  double* graph_sink = nullptr;
  bool capturing_steps = false;
  bool overlap() const { return nodes <= kOverlapNodes; }
  bool speed_valid = false;
  int epb = 0;
  // threads of a CTA = its elements' work items / tile_div, rounded up to
  // whole warps (one to three items per thread and phase; 3D: tile_threads), and
  // no more than the kernel's registers allow (Ops::launch_threads)
  int tile_div = 1;
  const Ops* ops = nullptr;
  // analysis (allocated by the first analysis call)
  bool an_ready = false;
  int an_m = 0, an_chunks = 0;
  long an_chunk = 0;
  double *d_an_wj = nullptr, *d_an_V = nullptr, *d_an_wa = nullptr, *d_an_rows = nullptr,
         *d_an_erows = nullptr, *d_an_out = nullptr, *d_an_uex = nullptr, *d_an_x = nullptr;
  long* d_an_rng = nullptr;  // [4][nmembers]: node begin, node end, element begin, element end
  size_t an_uex_cap = 0;
};

// Launchers for one (physics, n) instantiation.
struct Ops {
  int (*interface)(tag_handle h, const double* u);
  int (*element)(tag_handle h, int mode, double* u, double* du, int stage, bool last, double t);
  int (*max_speed)(tag_handle h, const double* u);
  // optional: u from mapped host memory into d_u with the CFL speeds reduced
  int (*load_state)(tag_handle h, const double* u_mapped);
  int (*init)(int max_smem);
  size_t (*smem_bytes)(int epb);
  int threads_per_element;
  int (*max_threads)();  // a tile's largest number of work items for one CTA
  int (*launch_threads)(tag_handle h);  // threads that an element kernel's CTA is launched with
};

// The launchers of each system for n nodes per direction (null: not built).
const Ops* ops_energy2d(int n);
const Ops* ops_energy3d(int n);
const Ops* ops_pt2d(int n);
const Ops* ops_pt3d(int n);
const Ops* ops_ie2d(int n);
const Ops* ops_moist2d(int n, bool weak);
const Ops* ops_rainy2d(int n, bool weak);
