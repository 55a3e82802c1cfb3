// kura_resident.cu -- the resident integrator (kura_resident.cuh) for one volcano network and its
// batch of trajectories, or one trajectory of a stored adjacency: kernels, the choice of shape, and
// the launch.  Stands in for the persistent
// kernel in MODE_INTEGRATE wherever a CTA's share of the state fits in shared memory.
#include "kura_resident.cuh"

namespace kura {
namespace {

constexpr int NT = 512;
// 18 warps for the float product: 33 rows per CTA (N = 5000) are two rows per warp, where 16 warps
// would wait for the one that has three
constexpr int NT_F32 = 576;
__host__ __device__ constexpr int threads_of(int den) { return den == RES_F32 ? NT_F32 : NT; }
constexpr size_t SMEM_CAP = 227 * 1024 - 256;  // dynamic, beside the ResNet
static_assert(sizeof(ResNet) <= 256, "SMEM_CAP");

template <int MODE, bool HL, int DEN = 0>
__global__ void __launch_bounds__(threads_of(DEN), 1) k_resident(const KParams p, const ResSplit split) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ ResNet net;
  if (threadIdx.x == 0) {
    net.n = p.n; net.k = split.k; net.B = p.batch; net.seed = p.seed; net.split = split;
    net.omega = p.omega;
    net.hi = p.ph_hi; net.lo = p.ph_lo; net.w = p.ph_w; net.g = p.g;
    net.ld = p.ld;
    net.atol = p.atol; net.rtol = p.rtol; net.fixed = p.fixed; net.dense_level = p.dense_level;
    net.t_eval = p.t_eval; net.n_eval = p.n_eval;
    net.out_r = p.out_r; net.out_idx = p.out_idx; net.out_theta = p.out_theta; net.out_coup = p.out_coup;
    net.out_ld = p.ld; net.ring = p.ring;
    net.log_t = p.log_t; net.log_h = p.log_h; net.log_cap = p.log_cap;
    net.max_attempts = p.max_attempts;
    net.adj = p.adj; net.adj8 = p.adj8; net.invn = p.invn; net.x = p.xbuf; net.xdig = p.xdig;
  }
  __syncthreads();
  Resident<MODE, HL, threads_of(DEN), DEN> e(net, smem, blockIdx.x, gridDim.x);
  e.bar = p.bar;
  e.bar_extra = p.bar_extra;
  e.err = p.err;
  e.part = p.part;
  e.timeout_ns = p.timeout_ns;
  e.fix = p.fix;
  if (threadIdx.x < p.batch) e.tr[threadIdx.x] = p.traj[threadIdx.x];
  __syncthreads();
  if (MODE == RES_CLUSTER) {  // every CTA runs before a peer writes into its shared memory
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
  if (!e.run()) return;
  if (blockIdx.x == 0) {
    if (threadIdx.x < p.batch) p.traj[threadIdx.x] = e.tr[threadIdx.x];
    if (threadIdx.x == 0) atomicAdd((unsigned long long*)p.counters, (unsigned long long)e.nbar);
  }
}

const void* pick(int mode, int hl, int den) {
  if (den == RES_F32) return (const void*)&k_resident<RES_GRIDX, true, RES_F32>;
  if (den == RES_I8) return (const void*)&k_resident<RES_GRIDX, true, RES_I8>;
  if (den == RES_IMMA) return (const void*)&k_resident<RES_GRIDX, true, RES_IMMA>;
  if (mode == RES_ONE) return hl ? (const void*)&k_resident<RES_ONE, true> : nullptr;
  if (mode == RES_CLUSTER) return hl ? (const void*)&k_resident<RES_CLUSTER, true> : nullptr;
  if (mode == RES_GRIDX) return hl ? (const void*)&k_resident<RES_GRIDX, true> : nullptr;
  return hl ? (const void*)&k_resident<RES_GRID, true> : (const void*)&k_resident<RES_GRID, false>;
}

cudaError_t configure(cudaLaunchConfig_t* cfg, cudaLaunchAttribute* attr, const ResPlan& r, cudaStream_t st) {
  const void* f = pick(r.mode, r.hl, r.split.den);
  // the limit is the kernel's, for every launch of it: always the same one, so that a thread that launches
  // a small network does not lower it under another thread's large one
  cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_CAP);
  if (e == cudaSuccess && r.mode == RES_CLUSTER && r.grid > 8)
    e = cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  cfg->gridDim = dim3((unsigned)r.grid);
  cfg->blockDim = dim3(threads_of(r.split.den));
  cfg->dynamicSmemBytes = r.smem;
  cfg->stream = st;
  cfg->attrs = attr;
  cfg->numAttrs = 0;
  if (r.mode == RES_CLUSTER) {
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = r.grid;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg->numAttrs = 1;
  } else if (r.mode >= RES_GRID) {
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg->numAttrs = 1;
  }
  return e;
}

// fills *r for a launch of `ctas` CTAs; blocks, rows: the grid of the persistent kernel and its rows
// per CTA.  False when the state does not fit.
bool shape(ResPlan* r, int B, int k, int blocks, int rows, int mode, int ctas, int hl, int den = 0, int ld = 0) {
  r->mode = mode;
  r->hl = hl;
  r->grid = ctas;
  r->split = {B, k, mode == RES_GRID ? rows : (blocks + ctas - 1) / ctas * rows, rows, blocks, ctas, den, ld};
  int off[18];
  r->smem = res_layout(r->split, hl, mode, threads_of(den), off);
  return r->smem <= SMEM_CAP && (mode == RES_GRID || r->split.rows < 65536);
}

}  // namespace

// Which form, by measured time per attempt (K = 5, Cauchy frequencies; the persistent kernel in
// brackets):
//   n x batch      one CTA   cluster (CTAs)   grid, same order   grid, fixed point
//   128             15.2     17.1 (2)
//   256             15.7     17.1 (4)
//   300             16.5     17.0 (4)          26.2              21.4   [44]
//   400             17.4     17.0 (4)
//   1000            23.4     17.5 (8)          26.4              25.1   [48]
//   4000             -       21.4 (16)         29.3              25.6   [48]
//   8000             -       23.9 (16)         31.1              25.7   [48]
//   16000            -       35.5 (16)         33.1              27.4   [50]
//   1000 x 8         -       25.4 (16)         33.4              30.2   [56]
//   4000 x 8         -       51.6 (16)         36.7              30.0   [56]
//   200000 x 5       -        -                 -                61.6   [139]
// One CTA and a cluster of four cross between 350 and 400 pairs and differ by 3 % from 300 to 400; the
// line is drawn below that, at 256.  A cluster pays for its rows, a grid for its barrier.  Fixed point serves from 12000 oscillators
// on, where it no longer matters in which order the sums are formed (kura_resident.cuh).
constexpr int64_t ONE_PAIRS = 256, CLUSTER_PAIRS = 12288, FIXED_N = 12000;

int resident_threads(const ResPlan& r) { return threads_of(r.split.den); }

ResPlan resident_plan(int64_t n, int B, int k, int blocks, int rows) {
  ResPlan r;
  if (k > RES_KMAX || B > 8) return r;
  const int64_t pairs = n * B;
  if (pairs <= ONE_PAIRS && shape(&r, B, k, blocks, rows, RES_ONE, 1, 1)) return r;
  if (pairs <= CLUSTER_PAIRS) {
    int cs = pairs <= 512 ? 4 : pairs <= 2048 ? 8 : RES_MAX_CLUSTER;
    while (cs > blocks) cs /= 2;
    for (; cs >= 2; cs /= 2) {
      if (!shape(&r, B, k, blocks, rows, RES_CLUSTER, cs, 1)) break;
      cudaLaunchConfig_t cfg = {};
      cudaLaunchAttribute attr[1];
      int fit = 0;
      if (configure(&cfg, attr, r, nullptr) == cudaSuccess &&
          cudaOccupancyMaxActiveClusters(&fit, pick(r.mode, r.hl, r.split.den), &cfg) == cudaSuccess && fit >= 1)
        return r;
      cudaGetLastError();
    }
  }
  if (n < FIXED_N) return rows < 1024 && shape(&r, B, k, blocks, rows, RES_GRIDX, blocks, 1) ? r : ResPlan();
  for (int hl = 1; hl >= 0; --hl)
    if (shape(&r, B, k, blocks, rows, RES_GRID, blocks, hl)) return r;
  return ResPlan();
}

// One trajectory of a stored adjacency: wherever the state fits beside the x tile and the ring (N up
// to about 80000 in float32, 70000 in int8) and a CTA has fewer than 1024 rows, from where on the
// persistent kernel forms its sums in another order.
// int8: the integer product from 12000 oscillators on (FIXED_N above; it adds in another order than
// the float one): us per attempt at N = 16384 377 -> 286, 40009 2347 -> 1607, 65536 4992 -> 3800.
ResPlan resident_plan_dense(int den, int64_t n, int ld, int blocks, int rows) {
  ResPlan r;
  if (den == RES_I8 && n >= FIXED_N && n <= 131072) {
    if (rows < 1024 && shape(&r, 1, 0, blocks, rows, RES_GRIDX, blocks, 1, RES_IMMA, ld)) return r;
  }
  if (rows < 1024 && shape(&r, 1, 0, blocks, rows, RES_GRIDX, blocks, 1, den, ld)) return r;
  return ResPlan();
}

cudaError_t launch_resident(const KParams& p, const ResPlan& r, cudaStream_t st) {
  KParams q = p;
  ResSplit split = r.split;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  cudaError_t e = configure(&cfg, attr, r, st);
  if (e != cudaSuccess) return e;
  void* args[] = {&q, &split};
  return cudaLaunchKernelExC(&cfg, pick(r.mode, r.hl, r.split.den), args);
}

}  // namespace kura
