// kura_resident.cuh -- DP45 with the state of a CTA's rows held in shared memory for the whole launch.
//
// The persistent kernel (kura_kernels.cu) keeps phases and slopes in L2 and reads up to nine values
// per oscillator and stage from there; with 64-bit addressing, a second pass over the rows for the
// projections and a third one for the slopes it spends 111 warp instructions per oscillator-step and
// 15.5 us per stage at 5 x 200000 oscillators (9.1 us of it in the rows); at n = 1000 a stage is a
// chain of latencies through L2, 6.9 us.  Now 8.8 us and 2.5 us: per attempt 139 -> 62 us and
// 48 -> 17 us.  Issue slots bound the large network, the chain of a stage (row, sums, exchange,
// table) the small one.  Here
//   * the slopes, the (cos, sin) and, where they fit, the phases of the CTA's (row, trajectory)
//     pairs stay in shared memory: 32 or 40 bytes per pair.  k2 and k7 share a slot (k2 has no
//     weight in stage 7, the error and the dense output), so six slots hold the seven slopes;
//   * one pass over the pairs per stage computes the slope of the stage before, the argument of the
//     next, its sine and cosine and the projections.  Warps take contiguous runs of 32-row chunks,
//     so that a warp meets at most two trajectories and reduces its projections once for each;
//   * the candidate y of an accepted step is formed again from the slopes when the next attempt
//     starts (and after the records of the step, which need the old y), not stored by stage 7.
//
// The sums cross CTAs in one of four ways (template MODE): not at all (one CTA), through the
// distributed shared memory of one cluster, or through L2 with a grid barrier, in two forms.  All
// are deterministic, and every CTA takes the same decisions from the same sums.  RES_ONE,
// RES_CLUSTER and RES_GRIDX add in the order of the persistent kernel and give its bits: with
// heavy-tailed frequencies the controller of a small network amplifies a rounding of its sums
// (1e-8 becomes 1e-6 of the phases within a hundred steps at n = 1000), so another order, although
// as exact, would be another run.  RES_GRID, for large networks, adds in fixed point.
//
// One trajectory of a stored adjacency runs the same way (template DEN) in the RES_GRIDX form: the
// CTAs publish (cos, sin) instead of sums, and after the barrier each forms its rows' couplings with
// kura_matvec.cuh in the place of the table.  Per attempt, against the persistent kernel: 49 -> 36 us
// at N = 997, 106 -> 89 at 5000 (A from L2 at 12 TB/s is 58 of them), 14.9 -> 14.1 ms at 65536
// (7.3 TB/s of A).
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include "kura.h"
#include "kura_device.cuh"
#include "kura_kernels.cuh"
#include "kura_matvec.cuh"

namespace kura {

constexpr int RES_KMAX = 8;
constexpr int RES_RED = 2 * RES_KMAX + 2;  // a warp's sums: 16 projections, sum cos, sum sin
constexpr int RES_WT = 12;                 // floats per weight row: W[0..6], time offset hi, lo, padding
// weight rows: stages 2..7, the error weights, the commit of the accepted step, a record, zeros
enum { RW_ERR = 6, RW_COMMIT = 7, RW_REC = 8, RW_ZERO = 9, RES_ROWS_WT = 10 };
constexpr int RES_MAX_CLUSTER = 16;
enum ResMode { RES_ONE = 0, RES_CLUSTER = 1, RES_GRID = RES_MODE_FIXED, RES_GRIDX = 3 };

// One network of up to 8 trajectories: where its state lies and what it writes.
struct ResNet {
  int n, k, B, seed;
  ResSplit split;
  const float* omega;
  float *hi, *lo;      // [2][B][ld] wrapped phase
  long long* w;        // [2][B][ld] windings
  float* g;            // [7][B][ld] slopes minus omega
  long long ld;
  double atol, rtol;
  int fixed, dense_level;
  const float* t_eval;  // output grid
  int n_eval;
  float* out_r;  // [B][ring]
  int* out_idx;  // [B][ring]
  float* out_theta;
  float* out_coup;
  long long out_ld;
  int ring;
  double *log_t, *log_h;
  int log_cap;
  long long max_attempts;
  // stored adjacency
  const float* adj;
  const int8_t* adj8;
  float invn;
  float2* x;  // [2][ld] (cos, sin) of all rows, by parity of the exchange
  int8_t* xdig;  // [2][8][ld] their digits (RES_IMMA)
};
// RES_IMMA takes the float product's x tile and ring where digits do not hold the components
static_assert(IM_SMEM_X + IM_SMEM_ACC >= CT_I8 / 16 * I8_CHUNK4 * 16 && 2 * IM_SLOTS >= I8_SLOTS, "shared memory of both products");
constexpr int RES_CTF = 7168;  // columns per x tile of the float product: leaves room for the state at N = 65536

// How the rows of a network are split and summed.  RES_GRID: CTA i owns rows i * rows ..; the
// others: the sums are formed over blocks of vrows rows, vblocks of them, as a grid of vblocks CTAs
// of the persistent kernel forms them, and CTA i owns the blocks i * vblocks / ctas ...  (ResSplit, kura_kernels.cuh)
// warps that the persistent kernel gives to one trajectory of a batch, below 1024 rows per CTA
__host__ __device__ inline int res_vwarps(int B) { return 16 / B; }
// the ones of them that have rows
__host__ __device__ inline int res_units(const ResSplit& s) {
  const int c = (s.vrows + 31) / 32, w = res_vwarps(s.B);
  return c < w ? c : w;
}
// Where CTA `cta` leaves its nv partial sums of the exchange of parity `par` (RES_GRIDX).  A CTA may
// still read the half of one exchange while another writes for the next (a half is written again only
// after a further barrier), and the number of sums differs from one exchange to the next: the halves
// lie PW_MAX sums of every CTA apart, whatever nv is.
__host__ __device__ inline size_t res_part(const ResSplit& s, int par, int cta, int nv) {
  return (size_t)par * s.vblocks * s.B * PW_MAX + (size_t)cta * nv;
}
// The sums that leave the pass of a kind (rows() below): values v0 .. v0 + nv - 1 of every trajectory,
// projections among them or not, and `npw`, the values that the persistent kernel would gather at once.
// rec_r: the pass over y (kind 0) records r; coup: records keep the couplings (dense level 2)
struct ResSums {
  int v0, nv, npw;
  bool proj;
};
__host__ __device__ inline ResSums res_sums(int kind, int k, bool den, bool rec_r, bool coup) {
  const bool stage = kind >= 2 && kind <= 7;
  if (den) {
    const bool sums = kind >= 8 || (kind == 0 && rec_r);
    return {2 * RES_KMAX, !sums ? 0 : kind == 8 ? 1 : 2, kind == 8 ? 1 : 2, false};
  }
  const bool all = kind == 0 || (kind == 9 && coup), proj = stage || all;
  const int np1 = 2 * k > 1 ? 2 * k : 1;
  const int npw = kind == 8 ? 1 : 2 * k + (kind == 9 || (kind == 0 && rec_r) ? 2 : 0);
  return {proj ? 0 : 2 * RES_KMAX, stage ? np1 : all ? RES_RED : kind == 8 ? 1 : 2, npw > 1 ? npw : 1, proj};
}
// Slices of blocks that the ordered sums are formed in, each at most 16 blocks where 128 threads
// allow: as the persistent kernel's, whose bits depend on it
__host__ __device__ inline int res_slices(int blocks, int npw) {
  int S = 128 / npw;
  if (S < 1) S = 1;
  return S < (blocks + 15) / 16 ? S : (blocks + 15) / 16;
}
// floats of the buffer of slices: every value of every slice.  (The number of slices follows npw, the
// number of values nv, which is larger in kind 0 and in a record with couplings.)
__host__ __device__ inline int res_slice_floats(const ResSplit& s) {
  const int most = res_slices(s.vblocks, 1) * s.B * RES_RED;
  return most > 1024 ? most : 1024;  // RES_GRID cuts its own to 1024
}
__host__ __device__ inline int res_align(int b) { return (b + 15) & ~15; }
// shared memory of a CTA in bytes; off[] as used by the kernel
__host__ __device__ inline size_t res_layout(const ResSplit& s, int hl, int mode, int nt, int* off) {
  const int np = s.B * s.rows, B = s.B, nvb = mode == RES_GRID ? 0 : (s.vblocks + s.ctas - 1) / s.ctas;
  const int nu = nvb * res_units(s);
  int o = 0, i = 0;
  auto take = [&](int bytes) {
    off[i++] = o;
    o += res_align(bytes);
  };
  take(B * (int)sizeof(TrajG));            // 0 controllers
  take(B * RES_ROWS_WT * RES_WT * 4);      // 1 weights
  take(B * 8);                             // 2 next output time
  take((mode == RES_GRID ? (nt / 32) * 2 : B * nu) * RES_RED * 4);  // 3 warps' or units' sums
  take(B * RES_RED * 4);                   // 4 totals
  take(mode >= RES_GRID ? 0 : (mode == RES_CLUSTER ? 2 : 1) * s.vblocks * B * RES_RED * 4);  // 5 totals of every block
  take(mode == RES_ONE ? 0 : res_slice_floats(s) * 4);  // 6 sums of slices of blocks or CTAs (RES_ONE: one slice)
  take((B << s.k) * 8);                    // 7 sign-pattern table
  take(64 + B * 28);                       // 8 flags, per-trajectory state of the run, its warps
  take(nu * 4);                            // 9 rows of the units
  take(s.rows * 4);                        // 10 omega
  take(s.rows);                            // 11 factor bits
  take(np * 8);                            // 12 (cos, sin)
  take(6 * np * 4);                        // 13 slopes
  take(hl ? np * 8 : 0);                   // 14 phases (hi, lo)
  if (s.den) {
    const int warps = nt / 32, cf = s.ld < RES_CTF ? s.ld : RES_CTF, ci = s.ld < CT_I8 ? s.ld : CT_I8;
    take(s.rows * 8);                                                                    // 15 couplings
    o = (o + 127) & ~127;  // copies into the ring are faster from a line boundary (1.2x at N = 65536)
    take(s.den == RES_F32    ? (cf + 3) / 4 * F_CHUNK * 8
         : s.den == RES_IMMA ? IM_SMEM_X + IM_SMEM_ACC
                             : (ci + 15) / 16 * I8_CHUNK4 * 16);  // 16 x tile
    o = (o + 127) & ~127;
    take(warps * 32 * 16 * (s.den == RES_F32 ? A_STAGES * A_ROWS : s.den == RES_IMMA ? 2 * IM_SLOTS : I8_SLOTS));             // 17 ring of A
  }
  return (size_t)o;
}

template <int MODE, bool HL, int NT, int DEN = 0>
struct Resident {
  static constexpr int NW = NT / 32;
  static constexpr bool EX = MODE != RES_GRID;  // sums in the persistent kernel's order
  const ResNet& N;
  TrajG* tr;
  float *wt, *red, *rsum, *ex, *slice;
  uint32_t* ut;  // of a unit: first row and the end of its block
  float2* tab;
  float2* Fr;  // DEN: couplings of the rows
  float4 *xt, *ring;
  double* te;  // per trajectory: the next output time
  int* flag;
  int* ps;  // per trajectory: phase buffer, candidate state, record slot, record index
  int* wr;  // per trajectory: first and last warp that hold rows of it, and the first one's entry in red
  float* om;
  uint8_t* ub;
  float2* xs;
  float* g;
  float2* yy;
  int tid, lane, warp, r0, nr, np, gi, G, B, k;
  int nch, c0, c1, b0, cc0;  // chunks of 32 rows per trajectory; this warp's run of all trajectories' chunks and where it starts
  int vb0, nvb, nwe, nu;  // this CTA's blocks, the units of a block and of all of them
  double rsn;       // 1 / sqrt(n)
  uint32_t act;     // trajectories that take part in the current pass
  uint32_t touched;  // trajectories whose phases or slopes this launch has changed
  // grid barrier
  unsigned *bar, target, bar_extra;
  unsigned long long* fix;  // [3][B * 2 k] projections in fixed point, and from 3 B 16 on [3] trajectories without
  int* err;
  float* part;
  unsigned long long timeout_ns;
  int nbar, par, nfix, xpar;
  bool rec0;  // the pass over y (kind 0) records r
  uint32_t mc, ms;  // RES_IMMA: the bits of the largest |cos| and |sin| of this thread's rows in the pass

  __device__ Resident(const ResNet& net, unsigned char* smem, int gi_, int G_) : N(net), gi(gi_), G(G_) {
    const ResSplit& sp = net.split;
    int off[18];
    res_layout(sp, HL, MODE, NT, off);
    tr = (TrajG*)(smem + off[0]);
    wt = (float*)(smem + off[1]);
    red = (float*)(smem + off[3]);
    rsum = (float*)(smem + off[4]);
    ex = (float*)(smem + off[5]);
    slice = (float*)(smem + off[6]);
    tab = (float2*)(smem + off[7]);
    flag = (int*)(smem + off[8]);
    ps = flag + 16;
    wr = ps + 4 * net.B;
    ut = (uint32_t*)(smem + off[9]);
    om = (float*)(smem + off[10]);
    ub = (uint8_t*)(smem + off[11]);
    xs = (float2*)(smem + off[12]);
    g = (float*)(smem + off[13]);
    yy = (float2*)(smem + off[14]);
    te = (double*)(smem + off[2]);
    if (DEN) {
      Fr = (float2*)(smem + off[15]);
      xt = (float4*)(smem + off[16]);
      ring = (float4*)(smem + off[17]);
    }
    xpar = 0;
    tid = threadIdx.x;
    lane = tid & 31;
    warp = tid >> 5;
    B = net.B;
    k = net.k;
    target = 0;
    mc = ms = 0;
    if (DEN == RES_IMMA && tid < 2) flag[2 + tid] = 0;
    nbar = 0;
    par = 0;
    nfix = 0;
    rsn = 1.0 / sqrt((double)net.n);
    if (EX) {
      vb0 = gi * sp.vblocks / G;
      nvb = (gi + 1) * sp.vblocks / G - vb0;
      r0 = min(net.n, vb0 * sp.vrows);
      nr = min(net.n, (vb0 + nvb) * sp.vrows) - r0;
      np = B * sp.rows;
      nwe = res_units(sp);
      nu = nvb * nwe;
      for (int u = tid; u < nu; u += NT) {
        const int v = u / nwe, a = v * sp.vrows + 32 * (u - v * nwe), z = min((v + 1) * sp.vrows, nr);
        ut[u] = (uint32_t)min(a, z) | (uint32_t)z << 16;
      }
    } else {
      r0 = min(net.n, gi * sp.rows);
      nr = min(net.n, r0 + sp.rows) - r0;
      np = B * sp.rows;
      nch = (nr + 31) / 32;
      c0 = run_start(warp);
      c1 = run_start(warp + 1);
      b0 = c0 / max(nch, 1);
      cc0 = c0 - b0 * nch;
      if (tid < B) {
        // a run's first trajectory is entry 0 of its warp, a second one entry 1; only the first warp
        // of a trajectory can have started in another
        int lo = -1, hi = -1;
        for (int w = 0; w < NW; ++w) {
          const int a = run_start(w), z = run_start(w + 1);
          if (a == z || a >= (tid + 1) * nch || z <= tid * nch) continue;
          if (lo < 0) lo = w;
          hi = w;
        }
        wr[tid * 3] = lo;
        wr[tid * 3 + 1] = hi;
        wr[tid * 3 + 2] = lo >= 0 && run_start(lo) < tid * nch ? 1 : 0;
      }
      // a warp without rows never writes its sums; the trajectories' totals run over it
      if (c0 == c1)
        for (int v = lane; v < 2 * RES_RED; v += 32) red[warp * 2 * RES_RED + v] = 0.f;
    }
  }
  __device__ __forceinline__ int run_start(int w) const { return w * B * nch / NW; }
  __device__ __forceinline__ size_t gaddr(int buf, int b, int r) const {
    return (size_t)(buf * B + b) * N.ld + r0 + r;
  }
  // slots of k1 and of k2 / k7 in shared memory (they swap when a step is accepted)
  __device__ __forceinline__ int slot_a(int b) const { return tr[b].rot_g & 1; }

  // ---------------------------------------------------------------- sums
  __device__ static __forceinline__ float wsum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
  }
  // 16 values per lane -> v[0] of lane L holds the warp total of value L >> 1
  __device__ static __forceinline__ void scatter16(float (&v)[16], int lane) {
#pragma unroll
    for (int half = 8, bit = 16; half >= 1; half >>= 1, bit >>= 1) {
      const bool upper = lane & bit;
#pragma unroll
      for (int j = 0; j < half; ++j) {
        const float send = upper ? v[j] : v[j + half];
        const float keep = upper ? v[j + half] : v[j];
        v[j] = keep + __shfl_xor_sync(0xffffffffu, send, bit);
      }
    }
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
  }

  __device__ __forceinline__ unsigned long long now() const {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
  }
  // RES_IMMA: the largest |cos| and |sin| of all rows, by their bits, in the exchange of barrier `i`.
  // Three pairs: the one read after the last barrier is cleared after this one and used after the next.
  __device__ __forceinline__ uint32_t* largest(int i) const { return reinterpret_cast<uint32_t*>(fix) + 2 * (i % 3); }
  // Whether digits of 2^-30 hold the components as well as floats do: the largest is 2^-7 or more, so
  // that half a step is at most half an ulp of it, or all are zero; none is infinite or NaN.  Otherwise
  // the product is the float one.  Sums of sin, relative error at N = 40009: phases over pi 6e-8 (float
  // product 9e-7), of 1e-2 around 0 5e-8 (4e-7), of 1e-4 in digits 3e-6 (5e-7), of 1e-6 3e-4 (7e-7)
  __device__ static __forceinline__ bool digits_hold(uint32_t bits) {
    return bits == 0 || (bits >= __float_as_uint(0.0078125f) && bits < __float_as_uint(1.5f));
  }
  // grid barrier with a time limit (as the persistent kernel's); every thread gets the verdict
  __device__ bool grid_sync() {
    __syncthreads();
    target += (unsigned)G;
    if (tid == 0) {
      if (DEN == RES_IMMA) {
        uint32_t* w = largest(nbar);
        atomicMax(w, (uint32_t)flag[2]);
        atomicMax(w + 1, (uint32_t)flag[3]);
        flag[2] = flag[3] = 0;
      }
      // the release covers what the other threads wrote before the block barrier above
      asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(bar), "r"(1u) : "memory");
      const unsigned long long t0 = now();
      int abort = 0;
      unsigned spins = 0;
      while (true) {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
        if ((int)(v - (target + bar_extra)) >= 0) break;
        if (*(volatile int*)err != 0) { abort = 1; break; }
        if ((++spins & 63u) == 0 && now() - t0 > timeout_ns) {
          atomicCAS(err, 0, KURA_ERR_BARRIER_TIMEOUT);
          abort = 1;
          break;
        }
      }
      flag[0] = abort;
    }
    __syncthreads();
    nbar++;
    return flag[0] == 0;
  }

  // The warps' sums -> rsum[b * RES_RED + v] over all CTAs: values v0 .. v0 + nv - 1 of every
  // trajectory (projections, then the plain sums or the error from value 16).
  // Projections leave as f3_m = (-1)^m / N sum_n u_mn x_n (m1, kuramoto.cu:62-81).
  __device__ __forceinline__ float finish(float s, int v, bool proj) const {
    return proj && v < 2 * RES_KMAX ? (((v >> 1) & 1) ? -s : s) / (float)N.n : s;
  }
  // The units' sums -> totals of the blocks -> (to every CTA of the cluster) -> slices of at most 16
  // blocks -> rsum: the same additions in the same order as a grid of vblocks CTAs of the persistent
  // kernel, so that a run gives the same bits however many CTAs carry it.
  // npw: the values per trajectory that the persistent kernel would gather at once.
  // DEN, want_F: the couplings of the rows as well; nv may be 0 then.
  __device__ __forceinline__ bool exchange_blocks(int v0, int nv, bool proj, int npw, bool want_F = false) {
    if (!DEN || nv) __syncthreads();
    const int NV = B * nv, VB = N.split.vblocks;
    float* mine = ex + (MODE == RES_CLUSTER ? par * VB * B * RES_RED : 0);
    // thread t of a round: value q of block vb; a block's NV values fill vstep threads
    const int vstep = NV <= 16 ? 16 : NV <= 32 ? 32 : NV <= 64 ? 64 : NV <= 128 ? 128 : 256;
    const int q = tid & (vstep - 1), b = B == 1 ? 0 : q / nv, v = v0 + q - b * nv;
    for (int vb = tid / vstep; vb < nvb; vb += NT / vstep) {
      if (q >= NV) break;
      const float* e = red + (b * nu + vb * nwe) * RES_RED + v;
      float x[4];
      float s = 0.f;
      for (int w = 0; w < nwe; w += 4) {
#pragma unroll
        for (int j = 0; j < 4; ++j) x[j] = w + j < nwe ? e[(w + j) * RES_RED] : 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) s += x[j];
      }
      if (MODE == RES_ONE) {
        mine[vb * NV + q] = s;
      } else if (MODE == RES_GRIDX) {
        part[res_part(N.split, nbar & 1, gi, NV) + q] = s;
      } else {
        const uint32_t a = (uint32_t)__cvta_generic_to_shared(mine + (vb0 + vb) * NV + q);
#pragma unroll 4
        for (int r = 0; r < G; ++r) {
          uint32_t peer;
          asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(a), "r"(r));
          asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(peer), "f"(s) : "memory");
        }
      }
    }
    if (MODE == RES_CLUSTER) {
      asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
      asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
      // these slots are written again two exchanges later, after the barrier of the next one, which
      // a CTA reaches only when it has read them
      par ^= 1;
    } else if (MODE == RES_GRIDX) {
      if (DEN == RES_F32 && want_F) mv_f32().first_chunks();  // they land during the barrier
      if (!grid_sync()) {
        if (DEN) cp_async_wait<0>();
        return false;
      }
      mine = part + res_part(N.split, (nbar - 1) & 1, 0, NV);
    } else {
      __syncthreads();
    }
    const int S = res_slices(VB, npw);
    if (S > 1 && NV) {
      for (int sl = tid / vstep; sl < S; sl += NT / vstep) {
        if (q >= NV) break;
        const int g0 = sl * VB / S, g1 = (sl + 1) * VB / S;
        float s = 0.f;
        for (int x0 = g0; x0 < g1; x0 += 16) s = add16<MODE == RES_GRIDX>(s, mine + x0 * NV + q, NV, g1 - x0);
        slice[sl * NV + q] = s;
      }
      __syncthreads();
    }
    if (tid < NV) {
      float s = 0.f;
      s = S > 1 ? add16(s, slice + tid, NV, S) : add16<MODE == RES_GRIDX>(s, mine + tid, NV, VB);
      rsum[b * RES_RED + v] = finish(s, v, proj);
    }
    if (MODE != RES_GRIDX) nbar++;
    bool digits = false;
    if (DEN == RES_IMMA) {
      if (want_F) {
        const uint2 m = __ldcg(reinterpret_cast<const uint2*>(largest(nbar - 1)));
        digits = digits_hold(m.x) && digits_hold(m.y);
      }
      if (gi == 0 && tid == 0) __stcg(reinterpret_cast<uint2*>(largest(nbar + 1)), make_uint2(0u, 0u));
    }
    if (DEN && want_F) {
      const float2* x = N.x + (size_t)xpar * N.ld;
      if (DEN == RES_F32)
        mv_f32().run(x, [&](int, int row, float Fc, float Fs, float2) { Fr[row - r0] = make_float2(Fc, Fs); });
      else if (DEN == RES_IMMA && digits)
        mv_imma().run(N.xdig + (size_t)xpar * 8 * N.ld,
                      [&](int row, float Fc, float Fs) { Fr[row - r0] = make_float2(Fc, Fs); });
      else
        mv_i8().run(x, [&](int row, float Fc, float Fs, float2) { Fr[row - r0] = make_float2(Fc, Fs); });
    }
    if (DEN) xpar ^= 1;
    __syncthreads();
    return true;
  }
  __device__ __forceinline__ MatvecF32<1, RES_CTF> mv_f32() const {
    return {N.adj, N.split.ld, r0, r0 + nr, 1, reinterpret_cast<float2*>(xt), ring, tid, NT, lane, warp, NW};
  }
  __device__ __forceinline__ MatvecImma mv_imma() const {
    int8_t* t = reinterpret_cast<int8_t*>(xt);
    return {N.adj8, N.invn, N.split.ld, r0, r0 + nr, (int)N.ld, t, reinterpret_cast<int*>(t + IM_SMEM_X),
            reinterpret_cast<uint4*>(ring), tid, NT, lane, warp, NW};
  }
  __device__ __forceinline__ MatvecI8 mv_i8() const {
    return {N.adj8, N.invn, N.split.ld, r0, r0 + nr, xt, reinterpret_cast<uint4*>(ring), tid, NT, lane, warp, NW};
  }
  // s + p[0] + p[stride] + .. of n <= 16 values, in that order
  template <bool L2 = false>
  __device__ static __forceinline__ float add16(float s, const float* p, int stride, int n) {
    float x[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) x[j] = j < n ? (L2 ? __ldcg(p + j * stride) : p[j * stride]) : 0.f;
#pragma unroll
    for (int j = 0; j < 16; ++j) s += x[j];
    return s;
  }

  // fixed: the totals are sums of sines and cosines, at most 2^20 of them.
  __device__ __forceinline__ bool exchange(int v0, int nv, bool proj, int npw, bool fixed) {
    if (EX) return exchange_blocks(v0, nv, proj, npw);
    __syncthreads();
    const int NV = B * nv;
    float tot = 0.f;
    int b = 0, v = 0;
    if (tid < NV) {
      b = tid / nv;
      v = v0 + tid - b * nv;
      const int lo = wr[b * 3], hi = wr[b * 3 + 1];
      if (lo >= 0) {
        tot = red[(lo * 2 + wr[b * 3 + 2]) * RES_RED + v];
#pragma unroll 4
        for (int w = lo + 1; w <= hi; ++w) tot += red[w * 2 * RES_RED + v];
      }
    }
    if (fixed) {
      // An integer sum does not depend on its order, so the CTAs add their totals to one place in L2
      // (2^-41 of rounding each) instead of leaving them for every CTA to gather: one load after the
      // barrier in the place of a round of 16 per thread and two more block barriers.  Three
      // buffers: the one read after the last barrier is cleared after this one and used after the next.
      // A total that is not finite has no integer: the trajectory's bit in a word beside them says so.
      unsigned long long* f = fix + (size_t)(nfix % 3) * NV;
      unsigned long long* nan = fix + 3 * B * 16;
      if (tid < NV) {
        if (!isfinite(tot)) atomicOr(nan + nfix % 3, 1ull << b);
        const long long q = __float2ll_rn(tot * 1099511627776.f);
        asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(f + tid), "l"(q) : "memory");
      }
      if (!grid_sync()) return false;
      if (tid < NV) {
        const long long q = (long long)__ldcg(f + tid);
        const uint32_t lost = (uint32_t)__ldcg(nan + nfix % 3) >> b & 1u;
        // (added, so that both loads are under way together: 0.4 us an exchange as a branch)
        rsum[b * RES_RED + v] = finish(__ll2float_rn(q) * (1.f / 1099511627776.f) + __uint_as_float(lost * 0x7fc00000u), v, proj);
        if (gi == 0) __stcg(fix + (size_t)((nfix + 2) % 3) * NV + tid, 0ull);
        if (gi == 0 && tid == 0) __stcg(nan + (nfix + 2) % 3, 0ull);
      }
      nfix++;
      __syncthreads();
      return true;
    }
    const int pp = nbar & 1;
    if (tid < NV) part[((size_t)(pp * G + gi) * B + b) * PW_MAX + v] = tot;
    if (!grid_sync()) return false;
    // slices of at most 16 CTAs where the buffer allows, each one round of loads in flight
    int S = 1024 / NV;
    if (S < 1) S = 1;
    if (S > (G + 15) / 16) S = (G + 15) / 16;
    const size_t stride = (size_t)B * PW_MAX;
    for (int t = tid; t < S * NV; t += NT) {
      const int q = t % NV, sl = t / NV;
      const int bb = q / nv, vv = v0 + q - bb * nv;
      const int g0 = sl * G / S, g1 = (sl + 1) * G / S;
      const float* src = part + ((size_t)pp * G * B + bb) * PW_MAX + vv;
      float s = 0.f;
      for (int q0 = g0; q0 < g1; q0 += 16) {
        float x[16];
#pragma unroll
        for (int u = 0; u < 16; ++u) x[u] = q0 + u < g1 ? __ldcg(src + (size_t)(q0 + u) * stride) : 0.f;
#pragma unroll
        for (int u = 0; u < 16; ++u) s += x[u];
      }
      slice[sl * NV + q] = s;
    }
    __syncthreads();
    if (tid < NV) {
      float s = 0.f;
      for (int sl = 0; sl < S; ++sl) s += slice[sl * NV + tid];
      rsum[b * RES_RED + v] = finish(s, v, proj);
    }
    __syncthreads();
    return true;
  }

  // F = sum_m +-f3_m for every sign pattern of the factor bits (m2, kuramoto.cu:83-101)
  __device__ void fill_table() {
    for (int t = tid; t < (B << k); t += NT) {
      const int b = t >> k, pat = t & ((1 << k) - 1);
      if (!((act >> b) & 1)) continue;
      const float* f = rsum + b * RES_RED;
      float Fc = 0.f, Fs = 0.f;
      for (int m = 0; m < k; ++m) {
        const float fc = f[2 * m], fs = f[2 * m + 1];
        const bool pos = (pat >> m) & 1;
        Fc += pos ? fc : -fc;
        Fs += pos ? fs : -fs;
      }
      tab[t] = make_float2(Fc, Fs);
    }
    __syncthreads();
  }

  // ---------------------------------------------------------------- the pass over the pairs
  __device__ __forceinline__ float2 load_y(int b, int r, int P) const {
    if (HL) return yy[P];
    const size_t a = gaddr(ps[b * 4], b, r);
    return make_float2(N.hi[a], N.lo[a]);
  }
  __device__ __forceinline__ void store_y(int b, int r, int P, float2 y) const {
    if (HL) {
      yy[P] = y;
    } else {
      const size_t a = gaddr(ps[b * 4], b, r);
      N.hi[a] = y.x;
      N.lo[a] = y.y;
    }
  }
  // y + omega (mh + ml) + gs as a float pair
  __device__ static __forceinline__ f2 advance(float om, float2 y, float mh, float ml, float gs) {
    const f2 pr = two_prod(om, mh);
    const f2 s1 = two_sum(y.x, pr.hi);
    const f2 s2 = two_sum(s1.hi, gs);
    return {s2.hi, y.y + ((s1.lo + s2.lo) + __fmaf_rn(om, ml, pr.lo))};
  }
  // The candidate of the accepted attempt: weights row w (stage 7) on the slopes, k1 in slot s1
  __device__ __forceinline__ f2 candidate(const float* w, int s1, float omr, float2 y, int P) const {
    float gs = w[0] * g[s1 * np + P];
#pragma unroll
    for (int j = 2; j < 6; ++j) gs = __fmaf_rn(w[j], g[j * np + P], gs);
    const f2 a = advance(omr, y, w[7], w[8], gs);
    return two_sum(a.hi, a.lo);
  }

  static constexpr int U = EX ? 1 : 2;    // rows of a lane in flight
  static constexpr int NA = EX ? U : 1;  // sets of sums: one per unit, or one for the warp's rows of a trajectory

  // The rows base[u] + lane, + step, .. of trajectory b.  Kind 2..7: the slope of the stage before
  // (kind > 2), the argument of stage `kind`, its (cos, sin) and sums; 2 first makes an accepted
  // candidate the new y.  8: the slope k7 and the error.  0: (cos, sin) and sums at y.  1: the slope
  // k1 of that.  9: the dense output with the record weights.
  template <int KIND>
  __device__ __forceinline__ void rows(int b, const int (&base)[U], const int (&end)[U], int step, int todo,
                                       float (&acc)[NA][16], float (&sx)[NA], float (&sy)[NA]) {
    constexpr bool SLOPE = KIND == 1 || (KIND >= 3 && KIND <= 8), ARG = KIND != 1 && KIND != 8;
    constexpr int ROW = KIND == 0 || KIND == 1 ? RW_ZERO : KIND == 9 ? RW_REC : KIND == 8 ? RW_ERR : KIND - 2;
    const int sa = slot_a(b), sb = sa ^ 1;
    const float* w = wt + (b * RES_ROWS_WT + ROW) * RES_WT;
    const float4 wa = *reinterpret_cast<const float4*>(w), wb = *reinterpret_cast<const float4*>(w + 4);
    const float W[8] = {wa.x, wa.y, wa.z, wa.w, wb.x, wb.y, wb.z, wb.w};  // the weights, the time offset
    const float ml = w[8];
    const bool commit = KIND == 2 && ps[b * 4 + 1];
    const float* wc = wt + (b * RES_ROWS_WT + RW_COMMIT) * RES_WT;
    const float c1b = tr[b].c1;
    const float2* tb = tab + (b << k);
    // the k1 / k7 pair of a record: after the accept k1 of the step sits in sb, k7 in sa
    float* ga = g + (KIND == 9 ? sb : sa) * np;
    float* gb = g + (KIND == 9 ? sa : sb) * np;
    const int P0 = b * N.split.rows;
    // U rows at a time: all their loads, then the arithmetic, then the stores, so that the
    // chains of the U rows overlap (the compiler moves no load over a store that could alias it)
#pragma unroll 1
    for (int q = 0; q < todo; q += step) {
      bool ok[U];
      int P[U], rr[U];
      uint32_t bits[U];
      float gn[U], gs[U], omr[U];
      float2 y[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int r = base[u] + q + lane;
        ok[u] = r < end[u];
        rr[u] = ok[u] ? r : 0;  // an idle lane reads row 0 and stores nothing
        P[u] = P0 + rr[u];
        bits[u] = DEN ? 0u : ub[rr[u]];
        gn[u] = gs[u] = omr[u] = 0.f;
        y[u] = make_float2(0.f, 0.f);
        if (SLOPE) {
          const float2 F = DEN ? Fr[rr[u]] : tb[bits[u]], x = xs[P[u]];
          gn[u] = c1b * (x.y * F.x - x.x * F.y);
        }
        if (ARG) {
          y[u] = load_y(b, rr[u], P[u]);
          omr[u] = om[rr[u]];
        }
        if (KIND >= 2) gs[u] = __fmaf_rn(W[0], ga[P[u]], 0.f);
        if (KIND == 3) gs[u] = __fmaf_rn(W[1], gn[u], gs[u]);
        if (KIND >= 4 && KIND <= 6) gs[u] = __fmaf_rn(W[1], gb[P[u]], gs[u]);
        if (KIND >= 4 && KIND <= 7) {
#pragma unroll
          for (int j = 2; j < KIND - 2; ++j) gs[u] = __fmaf_rn(W[j], g[j * np + P[u]], gs[u]);
          gs[u] = __fmaf_rn(W[KIND - 2], gn[u], gs[u]);
        }
        if (KIND == 8 || KIND == 9) {
#pragma unroll
          for (int j = 2; j < 6; ++j) gs[u] = __fmaf_rn(W[j], g[j * np + P[u]], gs[u]);
          gs[u] = __fmaf_rn(W[6], KIND == 8 ? gn[u] : gb[P[u]], gs[u]);
        }
      }
      if (KIND == 2 && commit) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const f2 y7 = candidate(wc, sb, omr[u], y[u], P[u]);
          float h7 = y7.hi, l7 = y7.lo;
          long long dw = 0;
          wrap_phase(h7, l7, dw);
          y[u] = make_float2(h7, l7);
          if (ok[u]) {
            if (dw) N.w[gaddr(ps[b * 4], b, rr[u])] += dw;
            store_y(b, rr[u], P[u], y[u]);
          }
        }
      }
      float cs[U], sn[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int a = EX ? u : 0;
        if (KIND == 8) {
          float tol = (float)N.atol;
          if (N.rtol != 0.0) {
            const float2 y0 = load_y(b, rr[u], P[u]);
            const long long wn = N.w[gaddr(ps[b * 4], b, rr[u])];
            const f2 y7 = candidate(wt + (b * RES_ROWS_WT + 5) * RES_WT, sa, om[rr[u]], y0, P[u]);
            float h7 = y7.hi, l7 = y7.lo;
            long long w7 = wn;
            wrap_phase(h7, l7, w7);
            const float a0 = fabsf(__fmaf_rn((float)wn, P2_1, y0.x));
            const float a1 = fabsf(__fmaf_rn((float)w7, P2_1, h7));
            tol = (float)N.atol + (float)N.rtol * fmaxf(a0, a1);
          }
          const float ye = gs[u] / tol;
          if (ok[u]) sx[a] = __fmaf_rn(ye, ye, sx[a]);
        }
        if (ARG) {
          const f2 z = advance(omr[u], y[u], W[7], ml, gs[u]);
          sincos_pair(z.hi, z.lo, &sn[u], &cs[u]);
          if ((KIND == 9 || KIND == 0) && N.dense_level >= 1 && ps[b * 4 + 2] >= 0 && ok[u]) {
            const f2 yv = two_sum(z.hi, z.lo);
            const long long wn = N.w[gaddr(ps[b * 4], b, rr[u])];
            N.out_theta[((size_t)b * N.ring + ps[b * 4 + 2]) * N.out_ld + r0 + rr[u]] =
                (float)((double)wn * TWO_PI_D + (double)yv.hi + (double)yv.lo);
          }
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int a = EX ? u : 0;
        if (SLOPE && ok[u]) {
          if (KIND == 3 || KIND == 8) gb[P[u]] = gn[u];
          else if (KIND == 1) ga[P[u]] = gn[u];
          else g[(KIND - 2) * np + P[u]] = gn[u];  // k3..k6 in slots 2..5
        }
        if (ARG && ok[u]) {
          xs[P[u]] = make_float2(cs[u], sn[u]);
          if (DEN == RES_IMMA) {
            int8_t* xd = N.xdig + (size_t)xpar * 8 * N.ld + r0 + rr[u];
            const uint32_t dc = x_digits(cs[u]), ds = x_digits(sn[u]);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              xd[j * N.ld] = (int8_t)(dc >> (8 * j));
              xd[(4 + j) * N.ld] = (int8_t)(ds >> (8 * j));
            }
            mc = max(mc, __float_as_uint(fabsf(cs[u])));
            ms = max(ms, __float_as_uint(fabsf(sn[u])));
          }
          if (DEN) {
            N.x[(size_t)xpar * N.ld + r0 + rr[u]] = make_float2(cs[u], sn[u]);
          }
          sx[a] += cs[u];
          sy[a] += sn[u];
          if (!DEN && (KIND != 9 || N.dense_level >= 2)) {
            // sums over the rows with u_mn = +1 (the factor bits from k on are zero)
#pragma unroll
            for (int m = 0; m < 4; ++m)
              if (bits[u] & (1u << m)) {
                acc[a][2 * m] += cs[u];
                acc[a][2 * m + 1] += sn[u];
              }
            if (k > 4) {
#pragma unroll
              for (int m = 4; m < 6; ++m)
                if (bits[u] & (1u << m)) {
                  acc[a][2 * m] += cs[u];
                  acc[a][2 * m + 1] += sn[u];
                }
            }
            if (k > 6) {
#pragma unroll
              for (int m = 6; m < 8; ++m)
                if (bits[u] & (1u << m)) {
                  acc[a][2 * m] += cs[u];
                  acc[a][2 * m + 1] += sn[u];
                }
            }
          }
        }
      }
    }
  }

  // One pass of all rows.  The row bodies are specialised by kind, everything around them is not:
  // with the flush and the exchange in every kind the kernel had 180-370 KB of code, which the
  // instruction caches do not hold (a stage of a small network took twice as long); with one body
  // for all kinds its loads no longer run ahead of the arithmetic (1.4 times as long at 5 x 200000).
  __device__ __forceinline__ void pass(const int kind) {
    const bool full = !DEN && kind != 1 && kind != 8 && (kind != 9 || N.dense_level >= 2);  // with projections
    const bool flush = kind != 1 && (!DEN || kind >= 8 || (kind == 0 && rec0));
    const int pairs = EX ? (nu + U - 1) / U : 0;  // EX: a warp takes U units at a time
    int e = 0;
#pragma unroll 1
    for (int c = EX ? warp : c0, b = b0 - 1, cc = cc0, run = 0; EX ? c < B * pairs : c < c1; c += EX ? NW : run, cc = 0) {
      int base[U], end[U], q0 = 0;
      if (EX) {
        b = B == 1 ? 0 : c / max(pairs, 1);
        q0 = U * (c - b * pairs);
        run = 0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const uint32_t t = q0 + u < nu ? ut[q0 + u] : 0u;
          base[u] = (int)(t & 0xffffu);
          end[u] = (int)(t >> 16);
          run = max(run, end[u] - base[u]);
        }
      } else {
        ++b;
        run = min(c1 - c, nch - cc);
#pragma unroll
        for (int u = 0; u < U; ++u) {
          base[u] = (cc + u) * 32;
          end[u] = min((cc + run) * 32, nr);
        }
      }
      if (!((act >> b) & 1)) {
        e = 1;
        continue;
      }
      const int step = EX ? 32 * res_vwarps(B) : 32 * U, todo = EX ? run : run * 32;
      float acc[NA][16], sx[NA], sy[NA];
#pragma unroll
      for (int a = 0; a < NA; ++a) {
        sx[a] = sy[a] = 0.f;
#pragma unroll
        for (int j = 0; j < 16; ++j) acc[a][j] = 0.f;
      }
      switch (kind) {
        case 0: rows<0>(b, base, end, step, todo, acc, sx, sy); break;
        case 1: rows<1>(b, base, end, step, todo, acc, sx, sy); break;
        case 2: rows<2>(b, base, end, step, todo, acc, sx, sy); break;
        case 3: rows<3>(b, base, end, step, todo, acc, sx, sy); break;
        case 4: rows<4>(b, base, end, step, todo, acc, sx, sy); break;
        case 5: rows<5>(b, base, end, step, todo, acc, sx, sy); break;
        case 6: rows<6>(b, base, end, step, todo, acc, sx, sy); break;
        case 7: rows<7>(b, base, end, step, todo, acc, sx, sy); break;
        case 8: rows<8>(b, base, end, step, todo, acc, sx, sy); break;
        default: rows<9>(b, base, end, step, todo, acc, sx, sy); break;
      }
      if (DEN == RES_IMMA) {
        const uint32_t c = __reduce_max_sync(0xffffffffu, mc), s = __reduce_max_sync(0xffffffffu, ms);
        if (lane == 0) {
          atomicMax((uint32_t*)flag + 2, c);
          atomicMax((uint32_t*)flag + 3, s);
        }
        mc = ms = 0;
      }
      if (!flush) continue;
      float* dst = red + (EX ? b * nu + q0 : warp * 2 + e) * RES_RED;
      e = 1;
      __syncwarp();
      // sum_n u_mn x_n = 2 (sum over u_mn = +1) - sum_n x_n on every lane, where it costs no digits
      // (of a CTA's totals it did: the error norm of a small step came out three times too large)
      if (full) {
#pragma unroll
        for (int a = 0; a < NA; ++a)
#pragma unroll
          for (int j = 0; j < 16; ++j) acc[a][j] = 2.f * acc[a][j] - ((j & 1) ? sy[a] : sx[a]);
      }
      if (!full || k == 8) {  // the plain sums, or the error, alone
#pragma unroll
        for (int a = 0; a < NA; ++a) {
          const float tx = wsum(sx[a]), ty = kind == 8 ? 0.f : wsum(sy[a]);
          if (lane == 0 && (!EX || q0 + a < nu)) {
            dst[a * RES_RED + 16] = tx;
            dst[a * RES_RED + 17] = ty;
          }
        }
        if (!full) continue;
      } else {  // the two plain sums ride in the unused last pair
#pragma unroll
        for (int a = 0; a < NA; ++a) {
          acc[a][14] = sx[a];
          acc[a][15] = sy[a];
        }
      }
      const int v = lane >> 1, vd = k < 8 && v >= 14 ? v + 2 : v;
#pragma unroll
      for (int a = 0; a < NA; ++a) {
        scatter16(acc[a], lane);
        if (!(lane & 1) && (!EX || q0 + a < nu)) dst[a * RES_RED + vd] = acc[a][0];
      }
    }
  }

  // ---------------------------------------------------------------- controller
  // weights of the next attempt (dp45.cu:90-106) and, for a trajectory whose last attempt was
  // accepted, its stage-7 row moved to the commit row; 16 threads per (stage, trajectory)
  __device__ void setup_attempt() {
    for (int t = tid; t < 6 * B * 16; t += NT) {
      const int j = t & 15, b = (t >> 4) % B, s = 2 + (t >> 4) / B;
      if (!((act >> b) & 1)) continue;
      float* w = wt + (b * RES_ROWS_WT + s - 2) * RES_WT;
      float* wc = wt + (b * RES_ROWS_WT + RW_COMMIT) * RES_WT;
      const double h = tr[b].h;
      if (j < 7) {
        if (s == 7 && ps[b * 4 + 1]) wc[j] = w[j];
        w[j] = (j < s - 1) ? (float)(h * A_TAB[s - 1][j]) : 0.f;
      } else if (j < 14) {
        if (s == 7) wt[(b * RES_ROWS_WT + RW_ERR) * RES_WT + j - 7] = (float)(h * E_TAB[j - 7]);
      } else if (j == 14) {
        if (s == 7 && ps[b * 4 + 1]) {
          wc[7] = w[7];
          wc[8] = w[8];
        }
        const double mh = C_TAB[s - 1] * h;
        const float hi = (float)mh;
        w[7] = hi;
        w[8] = (float)(mh - (double)hi);
      }
    }
    __syncthreads();
  }
  // (read from L2: an acquire at every barrier empties L1, so the controller compares with te first)
  __device__ __forceinline__ double eval_time(int i) const {
    return (double)N.t_eval[i];
  }
  // dense output at te from the last accepted step (interpolate, dp45.cu:70-76)
  __device__ void fill_record(int b, int j) {
    float* w = wt + (b * RES_ROWS_WT + RW_REC) * RES_WT;
    const TrajG& T = tr[b];
    const double hs = T.t - T.t_last, dl = eval_time(T.eval_i) - T.t_last;
    if (j < 7) {
      const double x = dl / hs;
      const double c = ((P_TAB[j][3] * x + P_TAB[j][2]) * x + P_TAB[j][1]) * x * x + P_TAB[j][0] * x;
      w[j] = (float)(hs * c);
    } else if (j == 14) {
      const float hi = (float)dl;
      w[7] = hi;
      w[8] = (float)(dl - (double)hi);
    }
  }
  // controller of one trajectory after the error norm (dp45.cu:109-139)
  __device__ void decide(int b) {
    TrajG& T = tr[b];
    const double h = T.h;
    bool accept = true;
    double factor = 1.0;
    if (!N.fixed) {
      const double sum = (double)rsum[b * RES_RED + 2 * RES_KMAX];
      const double norm = sqrt(sum) * rsn;
      if (isnan(norm)) {
        T.status = KURA_ERR_NONFINITE;
        return;
      }
      factor = (double)(0.9f * exp2f(-0.2f * log2f((float)norm)));
      accept = sum < (double)N.n;  // norm < 1
    }
    if (accept) {
      T.t_last = T.t;
      T.t = T.t + h;
      T.rot_y ^= 1;
      T.rot_g ^= 1;
      ps[b * 4 + 1] = 1;  // y still has to be advanced
      T.accepted++;
      if (!N.fixed) T.h = h * fmin(factor, 10.0);
      int e = T.eval_i;
      if (T.t >= te[b])
        while (e < N.n_eval && T.t >= eval_time(e)) e++;
      T.eval_end = e;
      if (N.log_cap > 0 && gi == 0) {
        N.log_t[(size_t)b * N.log_cap + T.log_count] = T.t;
        N.log_h[(size_t)b * N.log_cap + T.log_count] = T.h;
      }
      T.log_count++;
    } else {
      T.rejected++;
      if (factor < 1.0) T.h = h * fmax(factor, 0.2);
      if (!(T.h >= 1e-14 * fmax(1.0, fabs(T.t)))) T.status = KURA_ERR_STEP_UNDERFLOW;
    }
  }
  // r of the trajectories that record, from the totals
  __device__ void record_r() {
    if (gi != 0 || tid >= B || !((act >> tid) & 1) || ps[tid * 4 + 2] < 0) return;
    const float* s = rsum + tid * RES_RED;
    const float xn = s[2 * RES_KMAX] / (float)N.n, yn = s[2 * RES_KMAX + 1] / (float)N.n;
    N.out_r[(size_t)tid * N.ring + ps[tid * 4 + 2]] = sqrtf(xn * xn + yn * yn);
    N.out_idx[(size_t)tid * N.ring + ps[tid * 4 + 2]] = ps[tid * 4 + 3];
  }
  // couplings of the recorded rows (dense level 2), from the table
  __device__ void record_couplings() {
    for (int b = 0; b < B; ++b) {
      if (!((act >> b) & 1) || ps[b * 4 + 2] < 0) continue;
      float2* dst = reinterpret_cast<float2*>(N.out_coup + ((size_t)b * N.ring + ps[b * 4 + 2]) * 2 * N.out_ld) + r0;
      for (int r = tid; r < nr; r += NT) dst[r] = DEN ? Fr[r] : tab[(b << k) + ub[r]];
    }
  }

  // ---------------------------------------------------------------- the whole run
  // tr[] holds the controllers (loaded by the caller, all threads synchronised).  Of a trajectory b,
  // ps[4 b] is the phase buffer of y and its windings, ps[4 b + 1] the state of its candidate (0: y
  // is current, 1: the accepted step is still to be taken, 2: see load_phases), ps[4 b + 2] and
  // ps[4 b + 3] the record slot (-1: none) and index of the current pass.  Returns false when a
  // barrier gave up.
  __device__ bool run() {
    for (int r = tid; r < nr; r += NT) {
      const int i = r0 + r;
      if (!DEN) {
        uint32_t w = 0;
        for (int m = 0; m < k; ++m)
          w |= (stream_word(N.seed, (unsigned long long)m * (unsigned long long)N.n + (unsigned long long)i) & 1u) << m;
        ub[r] = (uint8_t)w;
      }
      om[r] = N.omega[i];
    }
    if (tid < B) {
      const TrajG& T = tr[tid];
      const bool owes = T.status == 0 && T.eval_i < T.eval_end;
      ps[tid * 4] = owes ? T.rot_y ^ 1 : T.rot_y;
      ps[tid * 4 + 1] = owes ? 2 : 0;
      ps[tid * 4 + 2] = -1;
    }
    if (tid < B * RES_WT) wt[(tid / RES_WT * RES_ROWS_WT + RW_ZERO) * RES_WT + tid % RES_WT] = 0.f;
    touched = 0;
    __syncthreads();
    for (int b = 0; b < B; ++b) {
      const int sa = slot_a(b), k1 = tr[b].rot_g ? 6 : 0, k7 = 6 - k1;
      for (int r = tid; r < nr; r += NT) {
        const int P = b * N.split.rows + r;
        // a launch that resumes the records of a step reads all its slopes
        g[sa * np + P] = N.g[gaddr(k1, b, r)];
        g[(sa ^ 1) * np + P] = N.g[gaddr(k7, b, r)];
#pragma unroll
        for (int j = 2; j < 6; ++j) g[j * np + P] = N.g[gaddr(j, b, r)];
      }
      load_phases(b, ps[b * 4]);
    }
    __syncthreads();

    if (tid < B) te[tid] = tr[tid].eval_i < N.n_eval ? eval_time(tr[tid].eval_i) : INFINITY;
    // first slope (dp45.cu:151) and the record at t0 (kuramoto.cu:587-626)
    act = 0;
    bool want_r = false;
    for (int b = 0; b < B; ++b) {
      const TrajG& T = tr[b];
      if (T.status == 0 && T.need_k1) {
        act |= 1u << b;
        want_r |= T.need_init && T.out_count < N.ring;
      }
    }
    rec0 = want_r;
    const bool coup = N.dense_level >= 2;
    long long attempts = 0;
    int kind = 0;
    if (act) {
      if (tid < B && ((act >> tid) & 1) && tr[tid].need_init && tr[tid].out_count < N.ring) {
        ps[tid * 4 + 2] = tr[tid].out_count;
        ps[tid * 4 + 3] = -1;
      }
      touched |= act;
      __syncthreads();
    } else if ((kind = next(attempts)) < 0) {
      return true;
    }
    // one pass, one exchange and one table per turn
#pragma unroll 1
    while (true) {
      pass(kind);
      if (kind == 1 || (kind == 8 && N.fixed)) {
        __syncthreads();
      } else {
        const ResSums q = res_sums(kind, k, DEN, want_r, coup);
        if (DEN) {
          if (!exchange_blocks(q.v0, q.nv, q.proj, q.npw, kind < 8 || (kind == 9 && coup))) return false;
        } else {
          if (!exchange(q.v0, q.nv, q.proj, q.npw, kind >= 2 && kind <= 7)) return false;
          if (q.proj) fill_table();
        }
      }
      const bool mine = tid < B && ((act >> tid) & 1);
      if (kind >= 2 && kind <= 7) {
        if (kind == 2 && mine) ps[tid * 4 + 1] = 0;  // the candidate has been taken
        ++kind;
        continue;
      }
      if (kind == 0) {
        if (want_r) record_r();
        kind = 1;
        continue;
      }
      if (kind == 8) {
        if (mine) decide(tid);
        attempts++;
      } else if (kind == 9) {
        record_r();
        if (coup) record_couplings();
        __syncthreads();
        if (mine) {
          const int i = ++tr[tid].eval_i;
          te[tid] = i < N.n_eval ? eval_time(i) : INFINITY;
          tr[tid].out_count++;
          ps[tid * 4 + 2] = -1;
        }
      } else {
        if (want_r && coup) record_couplings();
        __syncthreads();
        if (mine) {
          TrajG& T = tr[tid];
          T.need_k1 = 0;
          if (ps[tid * 4 + 2] >= 0) {
            T.need_init = 0;
            T.out_count++;
            ps[tid * 4 + 2] = -1;
          }
        }
      }
      __syncthreads();
      if ((kind = next(attempts)) < 0) break;
    }
    store_state();
    return true;
  }

  // What comes next: 9 a pending record, 2 an attempt (both made ready), -1 the end of the launch.
  __device__ __forceinline__ int next(long long attempts) {
    uint32_t owe = 0, step = 0;
    bool full = false;
    for (int b = 0; b < B; ++b) {
      const TrajG& T = tr[b];
      if (T.status != 0) continue;
      if (T.eval_i < T.eval_end) {
        if (T.out_count < N.ring) owe |= 1u << b; else full = true;
      } else if (T.t < T.t1) {
        if (N.log_cap > 0 && T.log_count >= N.log_cap) full = true; else step |= 1u << b;
      }
    }
    __syncthreads();  // every thread has read the controllers
    if (tid < B && tr[tid].status == 0 && tr[tid].eval_i >= tr[tid].eval_end && !(tr[tid].t < tr[tid].t1))
      tr[tid].status = 1;
    if (owe) {
      act = owe;
      if (tid < B * 16 && ((owe >> (tid >> 4)) & 1)) {
        const int b = tid >> 4, j = tid & 15;
        fill_record(b, j);
        if (j == 15) {
          ps[b * 4 + 2] = tr[b].out_count;
          ps[b * 4 + 3] = tr[b].eval_i;
        }
      }
      __syncthreads();
      return 9;
    }
    if (full || (N.max_attempts >= 0 && attempts >= N.max_attempts) || !step) {
      __syncthreads();
      return -1;
    }
    act = step;
    touched |= act;
    leave_records();
    setup_attempt();
    return 2;
  }

  // A trajectory that a former launch stopped between an accepted step and its records holds y one
  // step ahead in buffer rot_y and the old y in the other.  Its records read the old one (candidate
  // state 2); afterwards y comes back from rot_y.
  __device__ void load_phases(int b, int buf) {
    if (HL)
      for (int r = tid; r < nr; r += NT) {
        const size_t a = gaddr(buf, b, r);
        yy[b * N.split.rows + r] = make_float2(N.hi[a], N.lo[a]);
      }
  }
  __device__ void leave_records() {
    bool any = false;
    for (int b = 0; b < B; ++b)
      if (ps[b * 4 + 1] == 2) {
        any = true;
        load_phases(b, tr[b].rot_y);
      }
    if (!any) return;
    __syncthreads();
    if (tid < B && ps[tid * 4 + 1] == 2) {
      ps[tid * 4] = tr[tid].rot_y;
      ps[tid * 4 + 1] = 0;
    }
    __syncthreads();
  }

  // phases and slopes back to where other launches look for them
  __device__ void store_state() {
    __syncthreads();
    for (int b = 0; b < B; ++b) {
      if (!((touched >> b) & 1)) continue;
      const TrajG& T = tr[b];
      const int src = ps[b * 4], dst = T.rot_y, sa = slot_a(b), sb = sa ^ 1, k1 = T.rot_g ? 6 : 0, k7 = 6 - k1;
      const float* w = wt + (b * RES_ROWS_WT + 5) * RES_WT;  // the accepted attempt's stage 7
      for (int r = tid; r < nr; r += NT) {
        const int P = b * N.split.rows + r;
        const float2 y = load_y(b, r, P);
        const long long wn = N.w[gaddr(src, b, r)];
        if (ps[b * 4 + 1]) {
          const f2 y7 = candidate(w, sb, om[r], y, P);
          float h7 = y7.hi, l7 = y7.lo;
          long long w7 = wn;
          wrap_phase(h7, l7, w7);
          const size_t o = gaddr(dst ^ 1, b, r), a = gaddr(dst, b, r);
          N.hi[o] = y.x;
          N.lo[o] = y.y;
          N.w[o] = wn;
          N.hi[a] = h7;
          N.lo[a] = l7;
          N.w[a] = w7;
        } else if (HL || src != dst) {
          const size_t a = gaddr(dst, b, r);
          N.hi[a] = y.x;
          N.lo[a] = y.y;
          N.w[a] = wn;
        }
        N.g[gaddr(k1, b, r)] = g[sa * np + P];
        N.g[gaddr(k7, b, r)] = g[sb * np + P];
#pragma unroll
        for (int j = 2; j < 6; ++j) N.g[gaddr(j, b, r)] = g[j * np + P];
      }
    }
    __syncthreads();
  }
};

}  // namespace kura
