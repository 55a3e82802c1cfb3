// kura_tensor_split.cuh -- the coupling GEMM of a small or middle-sized ensemble: one unit of MT
// 128-row tiles and NCOL columns per thread-block cluster, the K range split over the cluster.
//
// The persistent GEMM (kura_tensor_gemm.cuh) gives a unit of rows to a CTA, which leaves most of
// the 152 SMs idle when n is below about 39000: at n = 3000 it ran on 12 of them and took 52 us,
// at n = 6007 (general adjacency) on 24 and took 120 us + 39 us for the pass over A_lo.  Here S
// CTAs of a cluster each accumulate K/S of the same unit in their own TMEM, leave the sums in
// shared memory and finish 1/S of the unit's (row, trajectory) pairs each, adding the S parts in
// rank order out of the peers' shared memory.  The A_lo pass of a general adjacency runs in the
// same K loop and accumulates into the X_lo columns, whose small sums it joins.  split_shape below
// gives the measured times.
//
// Roles (256 threads): warp 0 lane 0 feeds the ring with TMA, warp 1 lane 0 issues the MMAs; then
// all eight warps read TMEM (warp w owns lanes 32 (w % 4).., and half of the trajectories) and
// share the epilogue.  Every mbarrier wait is bounded; a CTA that gave up records the error and
// still arrives at both cluster barriers, so that its peers end too.
#pragma once
#include "kura_tensor_gemm.cuh"

namespace kura {

constexpr int TS_THREADS = 256;
constexpr int TS_BK = 64;
constexpr int TS_MAX_SPLIT = 8;  // portable cluster size

template <int NCOL, int MT> struct TSCfg {
  static constexpr int BP = NCOL / 4;  // trajectories per unit: [hi cos | hi sin | lo cos | lo sin]
  static constexpr int A1_BYTES = TG_BM * TS_BK * 2;
  static constexpr int A_BYTES = MT * A1_BYTES;
  static constexpr int X_BYTES = NCOL * TS_BK * 2;
  static constexpr int STAGE_BYTES = A_BYTES + X_BYTES;
  static constexpr int STAGES = (216 * 1024) / STAGE_BYTES > 8 ? 8 : (216 * 1024) / STAGE_BYTES;
  static constexpr int PART_BYTES = MT * 2 * BP * TG_BM * 4;  // the unit's sums, over the ring
  static constexpr int TMEM_COLS = MT * NCOL < 32 ? 32 : MT * NCOL;
  static constexpr int SMEM = STAGES * STAGE_BYTES + 1024 /* align */ + 256 /* barriers */;
  static_assert(PART_BYTES <= STAGES * STAGE_BYTES && MT * NCOL <= 512 && STAGES >= 2, "shape");
};

__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ float4 ld_peer4(uint32_t saddr, uint32_t rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(saddr), "r"(rank));
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(a)
               : "memory");
  return v;
}

// ktiles: K tiles of 64; S: cluster size (1 <= S <= ktiles); nsplit column blocks of xstride rows
// of X; has_lo: a second run over the K range with A_lo and the X_hi half of the columns.
// Epi::rows4(i, b, Fc, Fs): the couplings (times N) of rows i..i+3 of trajectory b.
template <int NCOL, int MT, class Epi>
__global__ void __launch_bounds__(TS_THREADS, 1)
    k_split_gemm(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmAlo,
                 const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmXhi, int ktiles, int S,
                 int nsplit, int xstride, int has_lo, Epi epi, int* err, unsigned long long limit_ns,
                 const int* run_flag) {
  using C = TSCfg<NCOL, MT>;
  constexpr int BP = C::BP;
  pdl_launch();
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* full = (uint64_t*)(smem + C::STAGES * C::STAGE_BYTES);
  uint64_t* empty = full + C::STAGES;
  uint64_t* accfull = empty + C::STAGES;
  uint32_t* tmem_slot = (uint32_t*)(accfull + 1);
  volatile int* sabort = (volatile int*)(tmem_slot + 1);
  const int unit = blockIdx.x / S, rank = blockIdx.x % S;
  const int rt0 = (unit / nsplit) * MT, sp = unit % nsplit;
  const int k0 = (int)((long long)rank * ktiles / S), nk = (int)((long long)(rank + 1) * ktiles / S) - k0;
  const int total = has_lo ? 2 * nk : nk;  // stages of this CTA: its K tiles with A_hi, then with A_lo
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (tid == 0) {
    for (int s = 0; s < C::STAGES; ++s) {
      umma::mbar_init(&full[s], 1);
      umma::mbar_init(&empty[s], 1);
    }
    umma::mbar_init(accfull, 1);
    *sabort = 0;
    umma::fence_barrier_init();
    umma::prefetch_tmap(&tmA);
    umma::prefetch_tmap(&tmX);
  }
  // One stage's loads.  A does not depend on the launch before this one (the stage kernel), so the
  // first stages' A tiles, like the setup, are on their way while that one still runs; X follows.
  // (Setup and A after the wait: runs of 3000 x 24 take 2.5 % longer, of 6007 x 64 1.5 %.)
  auto kcol = [&](int q) { return (k0 + (q >= nk ? q - nk : q)) * TS_BK; };
  auto load_a = [&](int q, int s) {
    const bool lo = q >= nk;
    umma::mbar_arrive_expect_tx(&full[s], C::A_BYTES + (lo ? C::X_BYTES / 2 : C::X_BYTES));
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
      umma::tma_load_2d(smem + s * C::STAGE_BYTES + mt * C::A1_BYTES, lo ? &tmAlo : &tmA, &full[s], kcol(q),
                        (rt0 + mt) * TG_BM);
  };
  auto load_x = [&](int q, int s) {
    umma::tma_load_2d(smem + s * C::STAGE_BYTES + C::A_BYTES, q >= nk ? &tmXhi : &tmX, &full[s], kcol(q), sp * xstride);
  };
  const int early = total < C::STAGES ? total : C::STAGES;
  if (tid == 0)  // the thread that initialised the barriers
    for (int q = 0; q < early; ++q) load_a(q, q);
  __syncwarp();
  if (warp == 2) umma::tmem_alloc(tmem_slot, C::TMEM_COLS);  // warp 2 also frees it
  umma::tc_fence_before();
  __syncthreads();
  umma::tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  pdl_wait();
  const bool skip = run_flag && *run_flag == 0;  // nothing to compute: the same for every CTA of the cluster
  if (skip) {
    if (tid == 0) {  // complete the early stages: no copy may outlive the CTA
      for (int q = 0; q < early; ++q) load_x(q, q);
      for (int q = 0; q < early; ++q) umma::mbar_wait(&full[q], 0, limit_ns, nullptr);
    }
    __syncthreads();
    if (warp == 2) umma::tmem_dealloc(tmem, C::TMEM_COLS);
    return;
  }

  if (warp == 0) {
    if (lane == 0) {
      int s = 0;
      uint32_t ph = 0;
      int issued = 0;
      for (int q = 0; q < total && (q < early || !*sabort); ++q) {
        if (q >= early) {
          if (!umma::mbar_wait(&empty[s], ph ^ 1, limit_ns, sabort)) {
            *sabort = 1;
            break;
          }
          load_a(q, s);
        }
        load_x(q, s);
        ++issued;
        if (++s == C::STAGES) { s = 0; ph ^= 1; }
      }
      // no copy may be in flight when the ring's memory is used again
      int ds = s;
      uint32_t dph = ph;
      for (int q = 0; q < C::STAGES && issued - q > 0; ++q) {
        if (--ds < 0) { ds = C::STAGES - 1; dph ^= 1; }
        umma::mbar_wait(&full[ds], dph, limit_ns, nullptr);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t id_hi = umma::idesc_f32(epi.f16(), TG_BM, NCOL), id_lo = umma::idesc_f32(epi.f16(), TG_BM, NCOL / 2);
      int s = 0;
      uint32_t ph = 0;
      for (int q = 0; q < total && !*sabort; ++q) {
        if (!umma::mbar_wait(&full[s], ph, limit_ns, sabort)) {
          *sabort = 1;
          break;
        }
        umma::tc_fence_after();
        const uint32_t a0 = umma::smem_u32(smem + s * C::STAGE_BYTES);
        const uint32_t x0 = a0 + C::A_BYTES;
        const uint32_t idesc = q >= nk ? id_lo : id_hi;
        const uint32_t acc = tmem + (q >= nk ? NCOL / 2 : 0);
#pragma unroll
        for (int kk = 0; kk < TS_BK / 16; ++kk)
#pragma unroll
          for (int mt = 0; mt < MT; ++mt)
            umma::mma_16(acc + mt * NCOL, umma::sw128_desc(a0 + mt * C::A1_BYTES + kk * 32),
                           umma::sw128_desc(x0 + kk * 32), idesc, (q > 0 || kk > 0) ? 1u : 0u);
        umma::mma_commit(&empty[s]);
        if (++s == C::STAGES) { s = 0; ph ^= 1; }
      }
      umma::mma_commit(accfull);
    }
    __syncwarp();
  }
  // ---- the unit's partial sums -> shared memory, over the ring (every MMA has read its operands)
  const bool ok = __all_sync(0xffffffffu, umma::mbar_wait(accfull, 0, limit_ns, sabort));
  if (!ok && lane == 0) *sabort = 1;
  __syncthreads();  // the producer has drained its copies
  umma::tc_fence_after();
  float* part = reinterpret_cast<float*>(smem);  // [mt][cos, sin][trajectory][128 rows]
  if (!*sabort) {
    const int row = (warp & 3) * 32 + lane;
    const uint32_t trow = tmem + ((uint32_t)((warp & 3) * 32) << 16);
#pragma unroll 1
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll 1
      for (int b0 = (warp >> 2) * (BP / 2); b0 < ((warp >> 2) + 1) * (BP / 2); b0 += 8) {
        float hc[8], hs[8], lc[8], ls[8];
        const uint32_t t = trow + mt * NCOL + b0;
        umma::tmem_ld8(t, hc);
        umma::tmem_ld8(t + BP, hs);
        umma::tmem_ld8(t + 2 * BP, lc);
        umma::tmem_ld8(t + 3 * BP, ls);
        umma::tmem_ld_wait();
        float* pc = part + ((size_t)(mt * 2) * BP + b0) * TG_BM + row;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          pc[j * TG_BM] = hc[j] + lc[j];
          pc[(BP + j) * TG_BM] = hs[j] + ls[j];
        }
      }
  }
  umma::tc_fence_before();
  if (S > 1) {
    cluster_arrive();
    cluster_wait();
  } else {
    __syncthreads();
  }
  // ---- this CTA's share of the unit: groups of four rows of one trajectory, a warp per 128 rows
  const int groups = MT * BP * (TG_BM / 4);
  const int g0 = (int)((long long)rank * (groups / 32) / S) * 32, g1 = (int)((long long)(rank + 1) * (groups / 32) / S) * 32;
  const uint32_t part_s = umma::smem_u32(part);
  if (!*sabort)
    for (int t = g0 + tid; t < g1; t += TS_THREADS) {
      const int rg = t & 31, mt = (t >> 5) % MT, bl = (t >> 5) / MT;
      const int b = sp * BP + bl;
      if (!epi.wants(b)) continue;
      const uint32_t ac = part_s + 4u * ((uint32_t)((mt * 2) * BP + bl) * TG_BM + rg * 4), as = ac + 4u * BP * TG_BM;
      float4 pc[TS_MAX_SPLIT], ps[TS_MAX_SPLIT];  // every peer's part is on its way before the first is added
#pragma unroll
      for (int r = 0; r < TS_MAX_SPLIT; ++r)
        if (r < S) {
          pc[r] = ld_peer4(ac, r);
          ps[r] = ld_peer4(as, r);
        }
      float4 c = pc[0], s4 = ps[0];
#pragma unroll
      for (int r = 1; r < TS_MAX_SPLIT; ++r)
        if (r < S) {
          c.x += pc[r].x; c.y += pc[r].y; c.z += pc[r].z; c.w += pc[r].w;
          s4.x += ps[r].x; s4.y += ps[r].y; s4.z += ps[r].z; s4.w += ps[r].w;
        }
      epi.rows4((rt0 + mt) * TG_BM + rg * 4, b, c, s4);
    }
  if (*sabort && tid == 0 && err) atomicCAS(err, 0, -4);
  if (S > 1) {  // the peers have read this CTA's sums before its shared memory goes away
    cluster_arrive();
    cluster_wait();
  }
  __syncthreads();
  if (warp == 2) {
    umma::tc_fence_after();
    umma::tmem_dealloc(tmem, C::TMEM_COLS);
  }
}

// ---------------------------------------------------------------- which shape
struct SplitShape {
  int mt = 0, s = 0;  // mt = 0: the persistent kernel
};
// The shape with the shortest predicted time, in clocks, for `tiles` 128-row tiles, nsplit column
// blocks of ncol columns and ktiles K tiles; fits(mt, s) is the number of clusters of s CTAs that run
// at once (fewer than sms / s: a cluster stays inside a GPC, and one cluster too many is a second
// wave).  A K tile of a CTA costs the larger of its MMAs (ncol 256: 142 clocks per 128 rows and 16 of
// K) and its operand bytes at the rate an SM draws from L2 when all of them do (about 55 bytes a
// clock).  A cluster adds its launch, the fill of the ring and the exchange of the sums.  The
// persistent kernel takes `waves` times a two-tile unit and pays its fill once.  Measured per launch
// (us), chosen against the persistent kernel: n = 1000 with 16 trajectories 10.4 (1 tile x 8) / 28.0;
// 3000 x 24 14.5 (1 x 4) / 45.3; 6007 x 64 28.0 (1 x 3) / 117.7, general 43.6 / 200.0; 20000 x 128
// 303 (2 x 4) / 467; 30000 x 20 292 (2 x 1) / 310; 65536 x 128 stays with the persistent kernel.
template <class Fits>
inline SplitShape split_shape(int tiles, int nsplit, int ncol, int ktiles, double waves0, Fits fits) {
  SplitShape best;
  const double mma2 = 8.0 * 142.0 * ncol / 256.0, load2 = (2 * 16384.0 + ncol * 128.0) / 55.0;
  double tbest = waves0 * ktiles * (mma2 > load2 ? mma2 : load2) + 6000.0;
  for (int mt = 1; mt <= 2; ++mt) {
    if (mt * ncol > 512) continue;
    const int units = (tiles + mt - 1) / mt * nsplit;
    const double mma = 4.0 * mt * 142.0 * ncol / 256.0;
    const double load = (mt * 16384.0 + ncol * 128.0) / 55.0;
    for (int s = 1; s <= TS_MAX_SPLIT && s <= ktiles; ++s) {
      const int at_once = fits(mt, s);
      if (at_once < 1) continue;
      const int waves = (units + at_once - 1) / at_once;
      const double exchange = 1500.0 + (s > 1 ? 1500.0 + mt * 128.0 * (ncol / 4) * 8.0 / 40.0 : 0.0);
      const double t = waves * (((ktiles + s - 1) / s) * (mma > load ? mma : load) + 4000.0 + exchange);
      if (t < tbest) {
        tbest = t;
        best.mt = mt;
        best.s = s;
      }
    }
  }
  return best;
}

}  // namespace kura
