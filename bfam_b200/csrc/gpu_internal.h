// Host-side declarations shared by the translation units of the bfam_gpu
// C-ABI (internal; the public interface is include/bfam_gpu.h).
#pragma once

#include "bfam_gpu.h"
#include "dg_common.cuh"

#include <atomic>
#include <cstdint>
#include <vector>

namespace bfam_b200
{
namespace host
{

// records the message for bfam_gpu_last_error and returns code
int fail(int code, const char *fmt, ...);
// kernels launched by the library (bfam_gpu_launch_count)
extern std::atomic<uint64_t> g_launches;
// stage kernels set up for launching (bfam_gpu_prepare_count)
extern std::atomic<uint64_t> g_prepares;

#define CUDA_TRY(call)                                                         \
  do                                                                           \
  {                                                                            \
    cudaError_t e_ = (call);                                                   \
    if (e_ != cudaSuccess)                                                     \
      return fail(BFAM_GPU_ECUDA, "%s: %s (%s:%d)", #call,                     \
                  cudaGetErrorString(e_), __FILE__, __LINE__);                 \
  } while (0)

// Launch as a programmatic dependent of the kernel before it in the stream:
// its CTAs may start while that kernel drains and wait for its completion in
// grid_dependency_wait, so that launch, scheduling and set-up overlap the
// drain.  The kernel must call grid_dependency_wait in every CTA before it
// touches anything an earlier kernel writes.  A step of a small mesh is a
// chain of such latencies: 2D N = 4 on 16 x 16 elements 18.5 -> 16.4 us per
// step of five launches replayed from a graph, and eagerly 30.7 -> 15.4 where
// the steps are waited for (13.6 -> 12.5 in a stream of steps, which the host's
// launch calls bound), 3D N = 5 on 211 elements 71.7 -> 69.9 and 92.2 -> 66.1 us
// per ten launches.
// overlap false: an ordinary launch (kernels among others on other streams).
template <typename... P, typename... A>
cudaError_t launch_dependent(bool overlap, void (*kernel)(P...), dim3 grid,
                             int threads, size_t smem, cudaStream_t stream,
                             A &&...args)
{
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = overlap;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = overlap ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// sp with StageParams::early for a stage whose widest launch has `ctas` CTAs
// (from: see late_from).  A stage of less than a wave of CTAs leaves
// places free on its SMs.  If the next launch's CTAs take them early, the SMs
// that finish first take more than their share of them, and the slowest SM of
// the next launch, with one CTA more than it need have, sets its time.  So from
// `from` per cent of a wave (there is room for the next launch's CTAs beside them
// below) to 85 % (hardly a place is free above), and not on meshes of at most a
// CTA per SM, the next launch's CTAs wait for the end, and only its launch
// overlaps it.  Us per step, ordinary launches -> early -> by this rule, replayed
// from a graph: 3D N = 5 FP64, 440 conforming elements (0.59 of a wave)
// 45.6 -> 50.7 -> 42.1, 528 49.7 -> 53.6 -> 47.6, 651 with hanging faces
// 93.0 -> 96.1 -> 90.2; N = 4, 528 38.4 -> 43.5 -> 35.3; N = 6, 256
// 48.7 -> 59.9 -> 46.5.  Waiting always costs
// small meshes 0.2 to 0.4 us a launch (2D N = 4, 256 16.9 -> 18.9).
inline StageParams with_early(int ctas, StageParams sp, int from)
{
  sp.early = ctas <= sp.sms || 100 * (int64_t)ctas <= from * (int64_t)sp.slots ||
             100 * (int64_t)ctas >= 85 * (int64_t)sp.slots;
  return sp;
}

// the kernels that serve the shapes: a thread per node, several elements per
// CTA, the matrix instruction
enum
{
  KERNEL_NODE = 0,
  KERNEL_PACK = 1,
  KERNEL_MMA = 2
};

// per-order launchers (the kernels' parameter lists depend on the order);
// which kernel serves a launch of n elements, and its set-up: shared-memory
// opt-in, resident CTAs per SM
typedef cudaError_t (*stage_launch_fn)(const DomainView &, int n,
                                const StageParams &, const double *D,
                                int mode, int kernel, cudaStream_t,
                                bool overlap);
typedef int (*stage_kernel_fn)(int n, const double *hops, int sms, int mode);
typedef cudaError_t (*prepare_fn)(int kernel, int mode, int *occ);
typedef void (*energy_fn)(const double *, size_t, const ElemData *,
                          const double *, double *);

struct KernelSet
{
  stage_launch_fn launch = nullptr;
  stage_kernel_fn kernel = nullptr;
  prepare_fn prepare = nullptr;
  energy_fn energy = nullptr;
  int NT = 0;
  int occ[3][4] = {}; // resident CTAs per SM by kernel and mode (0: not set up)
  int elements = 1;   // elements per CTA of the packed kernel
  int lookahead = 2;  // L2 lookahead: that part of a wave of resident CTAs
};

// a launch of a domain's stages: elements, mode, kernel, its resident CTAs on the
// device and its L2 lookahead
struct LaunchPlan
{
  int n = 0, mode = 0, kernel = 0, slots = 0, ahead = 0;
};

// the kernels of one (dim, order, precision)
bool kernel_set(int dim, int N, int precision, KernelSet *out);

// hops: host copy of the operator block Dr | interp[3] | proj[3] | w
template <int N, typename CT>
DiffOp<N, CT> make_diffop(const double *hops)
{
  constexpr int n2 = (N + 1) * (N + 1);
  DiffOp<N, CT> dop;
  for (int i = 0; i < n2; ++i)
  {
    dop.D[i] = CT(hops[i]);
    dop.Ib[i] = CT(hops[2 * n2 + i]); // interpolation[1]: refine to bottom
    dop.Pb[i] = hops[5 * n2 + i];     // projection[1]: coarsen from bottom
  }
  dop.iwend = 1.0 / hops[7 * n2];
  return dop;
}

} // namespace host
} // namespace bfam_b200

struct bfam_gpu_domain
{
  int dim = 0, N = 0, Nq = 0, Np = 0, Nfp = 0, NF = 0, NFLD = 0;
  int32_t K = 0, Kg = 0;
  int device = 0, sms = 0;
  int flux = 0, precision = 0;
  size_t fs = 0;
  bfam_b200::host::KernelSet ks;
  // per launch level; of the right-hand side once it is called
  std::vector<bfam_b200::host::LaunchPlan> stage_plan, rhs_plan;
  int widest = 0; // elements of the largest level
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  double *q[2] = {nullptr, nullptr};
  double *dq = nullptr;
  double *rhs = nullptr;
  double *energy = nullptr;
  bfam_b200::ElemData *ed = nullptr;
  int2 *fdesc = nullptr;
  double4 *fcE = nullptr;
  int *fslot = nullptr;  // [K][NF] mortar slot of each fine face (-1: none)
  double *mbuf = nullptr; // [slots][2 dim][Nfp] projected coarse-side jumps
  // launch levels (meshes with hanging faces): elements of level l are
  // elist[level_off[l] .. level_off[l+1])
  int nlevels = 1;
  std::vector<int32_t> level_off;
  int32_t *elist = nullptr;
  std::vector<int32_t> helist; // host copy of elist
  double *ops = nullptr;
  // host copy of Dr | interp[3] | proj[3] | w; the 1-D operators are passed
  // by value (kernel parameter bank) to each launch
  std::vector<double> hops;
  int *err = nullptr;
  int cur = 0;
  size_t bytes = 0, budget = 0;
  std::vector<void *> allocs;
  std::vector<size_t> alloc_bytes;
  // host copies for locating sources and receivers: element lower corners
  // and edge lengths [K][3], LGL nodes and weights [Nq]
  std::vector<double> hx0, hh, hr, hw;
  // element boxes computed on the device from quadrant data ([K][3] each;
  // null when the boxes came from the host)
  double *gx0 = nullptr, *gh = nullptr;
  // boundary list: element, face and (glued faces) mortar slot per entry;
  // glued faces are filled by the glue between domains
  std::vector<int32_t> bE, bslot;
  std::vector<int8_t> bF;
  int nglued = 0;
  // time-dependent extras: device clock, Ricker point source, receivers
  bfam_b200::DomainClock *clock = nullptr;
  bool clock_valid = false; // device clock holds the stepper's time
  bfam_b200::PointSource src{-1, nullptr, {0, 0, 0}, 0, 0};
  void *src_w_alloc = nullptr; // device copy of src.w
  int nrecv = 0, max_samples = 0;
  int *recv_elem = nullptr;
  double *recv_w = nullptr;
  double *seis = nullptr;
  unsigned extras_gen = 0;   // bumped when the source or receivers change
  // opt-in per-launch timing (bfam_gpu_domain_profile): an event pair
  // around every stage launch, drained into per-level totals
  bool prof = false;
  struct ProfLaunch
  {
    cudaEvent_t t0, t1;
    int level;
    double bytes; // algorithmic bytes of the launch
    int64_t elements;
  };
  std::vector<ProfLaunch> prof_pending;
  std::vector<cudaEvent_t> prof_free;
  std::vector<double> prof_ms, prof_bytes;
  std::vector<int64_t> prof_launches, prof_elements;
};

struct bfam_ts_lsrk
{
  bfam_gpu_domain_t *dom = nullptr;
  int ns = 0;
  double A[6] = {0}, B[6] = {0}, C[7] = {0};
  double t = 0;
  cudaGraphExec_t graph[2] = {nullptr, nullptr};
  double graph_dt[2] = {0, 0};
  bool graph_post[2] = {false, false};
  unsigned graph_gen[2] = {0, 0};
};

namespace bfam_b200
{
namespace host
{

// device allocation counted against the domain's budget, freed with it
int dev_alloc(bfam_gpu_domain_t *d, void **p, size_t bytes);
// the library's own stream-ordered memory pool of a device (created once,
// keeps freed blocks for reuse), and an allocation from it on a stream
cudaMemPool_t library_pool(int device);
cudaError_t pool_alloc(void **p, size_t bytes, int device, cudaStream_t stream);
// fills the host copies of the element boxes (read back from the device
// when the domain computed them from quadrant data)
int host_geometry(bfam_gpu_domain_t *d);
// frees one allocation made by dev_alloc before the domain is freed
void dev_free(bfam_gpu_domain_t *d, void *p);

template <typename T>
int upload(bfam_gpu_domain_t *d, T **dst, const T *src, size_t n)
{
  int rc = dev_alloc(d, (void **)dst, n * sizeof(T));
  if (rc)
    return rc;
  if (n)
    CUDA_TRY(cudaMemcpy(*dst, src, n * sizeof(T), cudaMemcpyHostToDevice));
  return 0;
}

// the stage kernel's view of a domain whose stage input is q[in]
DomainView view(bfam_gpu_domain_t *d, int in);
// one launch of a plan over v, the domain's view
int launch_planned(bfam_gpu_domain_t *d, const DomainView &v,
                   const LaunchPlan &p, StageParams sp, cudaStream_t stream,
                   bool overlap);
int launch_stage(bfam_gpu_domain_t *d, int in, double A, double B, double C,
                 double dt, int first, int mode);

// point source or receivers present
inline bool has_extras(const bfam_gpu_domain_t *d)
{
  return d->src.elem >= 0 || d->nrecv > 0;
}
// set the device clock to t (and reset the sample count), on the domain's
// stream
int set_clock(bfam_gpu_domain_t *d, double t, int reset);
// the post-step kernel of one domain whose state after the step is q[cur]
int launch_post(bfam_gpu_domain_t *d, int cur, double dt);

} // namespace host
} // namespace bfam_b200
