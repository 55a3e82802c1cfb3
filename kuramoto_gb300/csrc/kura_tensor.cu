// kura_tensor.cu -- the shared-adjacency ensemble on tcgen05 tensor cores.
//
// B trajectories (up to 128) share one dense adjacency A and the frequencies, with
// their own phases, coupling constants and adaptive steps.  Each RHS of the batch is
// one GEMM over A:
//   F[i][(cos|sin), b] = sum_j A_ij (cos, sin)(theta_jb)
// computed as (N A) x [X_hi | X_lo] with X = [cos | sin] split into F16 hi + lo and FP32
// accumulation in TMEM; the GEMM epilogue forms g = c_b (sin F_c - cos F_s) / N directly.
// For the reference's volcano rule N*A_ij is an integer in [-K, K], exact in F16 up to 2048, so
// the product carries the precision of the hi+lo split of X: 2^-21 of 1 and 2^-18 or better of itself,
// where BF16 parts of the same size and rate hold 2^-18 of x.  A general adjacency is split as 2^p_i N A_ij = A_hi + A_lo
// with a power of two per row, which puts a row's largest entry below 2^15: 11 significant bits in A_hi
// and 11 more in A_lo.  The term A_lo X_hi is added by further K steps.  F16 has five bits of exponent:
// an adjacency with a row whose entries span more than 2^21 (or lie below 2^-70, or are not finite) is
// held in BF16 parts instead, as are its X: each entry to 2^-18 of itself, at the same size and rate.
//
// The DP45 attempt (dp45_step, dp45.cu:87-141) is a fixed sequence of launches --
// coefficients, 6 x (stage, GEMM), error norm, controller, outputs -- captured once in a
// CUDA graph and replayed; every per-trajectory decision (accept/reject, step size, t,
// output crossings) stays on the device.  The host only polls a completion flag.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <algorithm>
#include <cstring>
#include <string>
#include <vector>
#include "kura.h"
#include "kura_device.cuh"
#include "kura_kernels.cuh"
#include "kura_tensor.h"
#include "kura_tensor_gemm.cuh"
#include "kura_tensor_split.cuh"

namespace kura {

namespace {

constexpr int T_MAXC = 32;  // output times recorded per launch; a step that crosses more waits for the next one
// K per pipeline stage of the coupling GEMM, in 128-byte swizzle rows: 64 (three 64 KB stages, eight MMAs
// per stage handshake) measured 7 % faster per launch at N=65536, B=128 than 32 in 64-byte rows (seven
// 32 KB stages, four MMAs per handshake).  The split GEMM reads through the same tensor maps.
constexpr int TE_BK = 64;
static_assert(TE_BK == TS_BK, "one tensor map for both GEMMs");
// The parts of a component x of (cos, sin): X_hi is a multiple of a step, X_lo the rest to 11 bits.
// From |x| = 2^-3 on the step is 2^-8: the tensor core cuts each product off at the accumulator's last
// bit, always toward zero, and coarse steps leave it nothing to cut from A_hi X_hi.  Below, X_hi has
// X_BITS significant bits: where all phases lie near 0 or pi, a step of 2^-8 leaves all of sin to X_lo.
// n = 6007 positive weights, rms error of the sums of sin against 64 bits: phases over [0, pi) 3.0e-7
// of the absolute row sum (2.4e-7 with steps of 2^-8 throughout, 1.1e-6 with BF16 parts), phases of
// 1e-2 around 0 1.0e-6 of the sums themselves (3.1e-5 and 4.4e-6).  9 bits in X_hi: 3.2e-7 and 5e-7.
// Both parts carry a factor 2^15, which keeps X_lo clear of F16's smallest steps down to x = 2^-22
// and comes off again with the scale of the row (rinv).
constexpr int X_BITS = 7;
constexpr float X_SCALE = 32768.f;
constexpr int T_RBLK = 256; // rows per block of the reduction kernels

struct TCoef {
  float W[7];
  float E[7];
  float m_hi, m_lo;
  int slot[7];
  int base, gout, active, store_y7, rec, nW;
  float c1;
  int pad;
};

struct TView {
  int n, np, bp, B, mode;
  const float* omega;
  float* ph_hi;
  float* ph_lo;
  long long* ph_w;
  float* g;
  __half* X;
  float2* x32;
  float* fin_theta;
  float* fin_coup;
  float* Flo;  // [2][bp][np] partial couplings of the A_lo pass (general adjacency)
  const float* rinv;  // [np] 1 / (N 2^p_i X_SCALE): the scale of a row's couplings
  int bf16;           // the parts are BF16 (rinv is 1 / N)
};

// row of X holding column q (0 hi cos, 1 hi sin, 2 lo cos, 3 lo sin) of trajectory b: the
// trajectories are grouped by 64 so that each group's 4 x 64 columns are one contiguous
// block, the column block of one GEMM work unit
__host__ __device__ __forceinline__ int x_bph(int bp) { return bp > 64 ? 64 : bp; }
__device__ __forceinline__ size_t xrow(int q, int b, int bp) {
  const int g = x_bph(bp);
  return (size_t)(b / g) * 4 * g + (size_t)q * g + (b % g);
}
__device__ __forceinline__ int slot_k1(int rot_g) { return rot_g ? 6 : 0; }
__device__ __forceinline__ int slot_k7(int rot_g) { return rot_g ? 0 : 6; }

// ---------------------------------------------------------------- coefficients
// Per-trajectory sources: src[0] = phases y (first slope, RHS), src[1..6] = stages 2..7
// of the next attempt (dp45.cu:90-106), src[7] = dense output (set by the output kernels).
// src[0] of the trajectories that still need their first slope; flags[0]: there is one
__global__ void k_t_first(const TrajG* traj, TCoef* src, int* flags) {
  const int b = blockIdx.x, j = threadIdx.x;
  TCoef& S = src[b];
  const TrajG& T = traj[b];
  if (j < 7) {
    S.W[j] = 0.f;
    S.slot[j] = j;
  } else if (j == 7) {
    S.m_hi = S.m_lo = 0.f;
    S.nW = 0;
    S.base = T.rot_y;
    S.gout = slot_k1(T.rot_g);
    S.active = (T.status == 0 && T.need_k1);
    S.store_y7 = 0;
    S.rec = 0;
    S.c1 = T.c1;
    if (S.active) flags[0] = 1;
  }
}
// the six stages of trajectory b's next attempt, by 16 threads per stage; flags[1]: some
// trajectory steps in it, or sits it out because it still owes records of its last step (how many
// output times a step crosses depends on the step control, and that on rounding: no limit on it)
__device__ __forceinline__ void fill_attempt(const TrajG& T, TCoef* src, int bp, int b, int t, int* flags) {
  const bool act = (T.status == 0 && T.eval_i >= T.eval_end && T.t < T.t1);
  if (t == 0 && (act || (T.status == 0 && T.eval_i < T.eval_end))) flags[1] = 1;
  if (t >= 6 * 16) return;
  const int j = t & 15, s = 2 + (t >> 4);
  TCoef& S = src[(s - 1) * bp + b];
  const double h = T.h;
  if (j < 7) {
    S.W[j] = (j < s - 1) ? (float)(h * A_TAB[s - 1][j]) : 0.f;
  } else if (j < 14) {
    if (s == 7) S.E[j - 7] = (float)(h * E_TAB[j - 7]);
  } else if (j == 14) {
    double mh = C_TAB[s - 1] * h;
    float hi = (float)mh;
    S.m_hi = hi;
    S.m_lo = (float)(mh - (double)hi);
  } else {
    S.nW = s - 1;
    S.slot[0] = slot_k1(T.rot_g);
    for (int q = 1; q < 6; ++q) S.slot[q] = q;
    S.slot[6] = slot_k7(T.rot_g);
    S.base = T.rot_y;
    S.gout = (s < 7) ? s - 1 : slot_k7(T.rot_g);
    S.store_y7 = (s == 7);
    S.rec = 0;
    S.active = act;
    S.c1 = T.c1;
  }
}

// source for the end-of-run record (interpolation with k1 replaced by k7, as after the
// reference's FSAL copy, kuramoto.cu:632) or the current phases (RHS, no step taken)
__global__ void k_t_coef_final(TrajG* traj, TCoef* src, int B, const float* t_eval, int n_eval, int use_eval) {
  const int b = threadIdx.x;
  if (b >= B) return;
  TCoef& S = src[b];
  const TrajG& T = traj[b];
  for (int q = 0; q < 7; ++q) { S.W[q] = 0.f; S.slot[q] = q; }
  S.m_hi = S.m_lo = 0.f;
  S.nW = 0;
  S.base = T.rot_y;
  if (use_eval && n_eval > 0 && T.accepted > 0) {
    const double hs = T.t - T.t_last, dl = (double)t_eval[n_eval - 1] - T.t_last, x = dl / hs;
    for (int j = 0; j < 7; ++j) {
      const double c = ((P_TAB[j][3] * x + P_TAB[j][2]) * x + P_TAB[j][1]) * x * x + P_TAB[j][0] * x;
      S.W[j] = (float)(hs * c);
    }
    S.nW = 7;
    S.m_hi = (float)dl;
    S.m_lo = (float)(dl - (double)S.m_hi);
    const int ks = slot_k1(T.rot_g);
    S.slot[0] = ks;
    S.slot[6] = ks;
    S.base = T.rot_y ^ 1;
  }
  S.gout = -1;
  S.active = 1;
  S.store_y7 = 0;
  S.rec = 1;
  S.c1 = T.c1;
}

// ---------------------------------------------------------------- stage (elementwise)
// theta = phase[base] + omega*(m_hi+m_lo) + sum_j W_j g_j for trajectory b and four oscillators
// i .. i + 3; writes the F16 hi/lo operand columns (cos, sin) and the FP32 (cos, sin) for the
// epilogue.  A thread takes four oscillators because the kernel is bound by the bytes it has in
// flight: one at a time moved 336 MB at N = 65536, B = 128 in 99 us, four in about 62.  The last
// group may reach into the padding (np is a multiple of 256), whose state stays finite and meets
// zero columns of A.
// the 16-bit parts of x, hi in the lower half
__device__ __forceinline__ uint32_t x_parts(float x, bool bf16) {
  if (bf16) {
    const __nv_bfloat16 hi = __float2bfloat16_rn(x);
    const __nv_bfloat162 h = __halves2bfloat162(hi, __float2bfloat16_rn(x - __bfloat162float(hi)));
    return *reinterpret_cast<const uint32_t*>(&h);
  }
  // adding and taking away 1.5 * 2^23 steps rounds to a multiple of the step
  const uint32_t small = (__float_as_uint(x) & 0x7f800000u) + ((uint32_t)(24 - X_BITS) << 23);
  const uint32_t large = __float_as_uint(32768.f);  // 2^23 * 2^-8
  const float m = __uint_as_float(((__float_as_uint(x) & 0x7fffffffu) < __float_as_uint(0.125f) ? small : large) | 0x400000u);
  const float hi = __fsub_rn(__fadd_rn(x, m), m);
  const __half2 h = __floats2half2_rn(hi * X_SCALE, (x - hi) * X_SCALE);
  return *reinterpret_cast<const uint32_t*>(&h);
}
constexpr int ST_THREADS = 128;
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float a, float b, float c, float d) {
  *reinterpret_cast<float4*>(p) = make_float4(a, b, c, d);
}

// `last`: the newest slope where the caller has it in registers, else null; X: the operand buffer
__device__ __forceinline__ void stage4(const TView& v, const TCoef& s, int b, int i, __half* X, const float4* last) {
  const size_t boff = ((size_t)s.base * v.bp + b) * v.np + i;
  const float4 om4 = ld4(v.omega + i), hi4 = ld4(v.ph_hi + boff), lo4 = ld4(v.ph_lo + boff);
  float4 gk[6];
#pragma unroll
  for (int j = 0; j < 6; ++j) {
    gk[j] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (j < s.nW) gk[j] = last && j == s.nW - 1 ? *last : ld4(v.g + ((size_t)s.slot[j] * v.bp + b) * v.np + i);
  }
  float gs[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int j = 0; j < 6; ++j)
    if (j < s.nW) {
      gs[0] = __fmaf_rn(s.W[j], gk[j].x, gs[0]);
      gs[1] = __fmaf_rn(s.W[j], gk[j].y, gs[1]);
      gs[2] = __fmaf_rn(s.W[j], gk[j].z, gs[2]);
      gs[3] = __fmaf_rn(s.W[j], gk[j].w, gs[3]);
    }
  if (s.nW > 6) {  // the end-of-run record uses all seven
    const float4 g6 = ld4(v.g + ((size_t)s.slot[6] * v.bp + b) * v.np + i);
    gs[0] = __fmaf_rn(s.W[6], g6.x, gs[0]);
    gs[1] = __fmaf_rn(s.W[6], g6.y, gs[1]);
    gs[2] = __fmaf_rn(s.W[6], g6.z, gs[2]);
    gs[3] = __fmaf_rn(s.W[6], g6.w, gs[3]);
  }
  const float om[4] = {om4.x, om4.y, om4.z, om4.w}, yh[4] = {hi4.x, hi4.y, hi4.z, hi4.w}, yl[4] = {lo4.x, lo4.y, lo4.z, lo4.w};
  float cs[4], sn[4], zh[4], zl[4];
  uint32_t cp[4], sp[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const f2 pr = two_prod(om[q], s.m_hi);
    const f2 s1 = two_sum(yh[q], pr.hi);
    const f2 s2 = two_sum(s1.hi, gs[q]);
    zh[q] = s2.hi;
    zl[q] = yl[q] + ((s1.lo + s2.lo) + __fmaf_rn(om[q], s.m_lo, pr.lo));
    sincos_pair(zh[q], zl[q], &sn[q], &cs[q]);
    cp[q] = x_parts(cs[q], v.bf16);
    sp[q] = x_parts(sn[q], v.bf16);
  }
  float* x = reinterpret_cast<float*>(v.x32 + (size_t)b * v.np + i);
  st4(x, cs[0], sn[0], cs[1], sn[1]);
  st4(x + 4, cs[2], sn[2], cs[3], sn[3]);
  auto put = [&](int q, const uint32_t (&h)[4], uint32_t half) {  // half: 0x5410 the hi parts, 0x7632 the lo parts
    *reinterpret_cast<uint2*>(X + xrow(q, b, v.bp) * v.np + i) =
        make_uint2(__byte_perm(h[0], h[1], half), __byte_perm(h[2], h[3], half));
  };
  put(0, cp, 0x5410u);
  put(1, sp, 0x5410u);
  put(2, cp, 0x7632u);
  put(3, sp, 0x7632u);
  if (s.store_y7 || s.rec) {
    const size_t o = ((size_t)(s.base ^ 1) * v.bp + b) * v.np + i;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      f2 y = two_sum(zh[q], zl[q]);
      long long w = v.ph_w[boff + q];
      if (s.store_y7) {
        float hi7 = y.hi, lo7 = y.lo;
        long long w7 = w;
        wrap_phase(hi7, lo7, w7);
        v.ph_hi[o + q] = hi7;
        v.ph_lo[o + q] = lo7;
        v.ph_w[o + q] = w7;
      } else if (v.fin_theta) {
        v.fin_theta[(size_t)b * v.np + i + q] = (float)((double)w * TWO_PI_D + (double)y.hi + (double)y.lo);
      }
    }
  }
}
__global__ void __launch_bounds__(ST_THREADS) k_t_stage(TView v, const TCoef* src) {
  pdl_launch();
  pdl_wait();
  const int b = blockIdx.y;
  const int i = (blockIdx.x * ST_THREADS + threadIdx.x) * 4;
  if (src[b].active && i < v.n) stage4(v, src[b], b, i, v.X, nullptr);
}

// ---------------------------------------------------------------- GEMM epilogues
// accumulator columns of work unit sp: [hi cos | hi sin | lo cos | lo sin] of trajectories
// sp*BP .. sp*BP + BP - 1, BP columns each
template <int BP> struct KuraEpi {
  TView v;
  const TCoef* src;
  int has_lo;
  __device__ bool f16() const { return !v.bf16; }
  __device__ void row(uint32_t taddr, int row, int m0, int sp) {
    const int i = m0 + row;
    const float rinv = v.rinv[i];
#pragma unroll 1
    for (int b0 = 0; b0 < BP; b0 += 16) {
      float hc[16], hs[16], lc[16], ls[16];
      umma::tmem_ld16(taddr + 0 * BP + b0, hc);
      umma::tmem_ld16(taddr + 1 * BP + b0, hs);
      umma::tmem_ld16(taddr + 2 * BP + b0, lc);
      umma::tmem_ld16(taddr + 3 * BP + b0, ls);
      umma::tmem_ld_wait();
      if (i >= v.n) continue;
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const int b = sp * BP + b0 + j;
        if (b >= v.B) break;
        const TCoef& s = src[b];
        if (!s.active) continue;
        float Fc = hc[j] + lc[j], Fs = hs[j] + ls[j];
        if (has_lo) {
          Fc += v.Flo[((size_t)0 * v.bp + b) * v.np + i];
          Fs += v.Flo[((size_t)1 * v.bp + b) * v.np + i];
        }
        Fc *= rinv;
        Fs *= rinv;
        const float2 x = v.x32[(size_t)b * v.np + i];
        const float gv = s.c1 * (x.y * Fc - x.x * Fs);
        if (s.gout >= 0) v.g[((size_t)s.gout * v.bp + b) * v.np + i] = gv;
        if (v.mode != 0 && s.rec) {
          v.fin_coup[((size_t)b * v.np + i) * 2] = Fc;
          v.fin_coup[((size_t)b * v.np + i) * 2 + 1] = Fs;
          if (v.mode == 2) v.fin_theta[(size_t)b * v.np + i] = v.omega[i] + gv;
        }
      }
    }
  }
};
// The same for the split GEMM: the couplings (times N) of rows i..i+3 of trajectory b.  Within an
// attempt it goes on to the operands of the next stage (`next`), which need no other row, into the
// operand buffer that this launch does not read, which saves the launch and the pass of a stage
// kernel between two GEMMs (Impl::one_group() says when).
struct SplitEpi {
  TView v;
  const TCoef* src;
  const TCoef* next;  // or null
  __half* Xn;
  __device__ bool f16() const { return !v.bf16; }
  __device__ bool wants(int b) const { return b < v.B && src[b].active; }
  __device__ void rows4(int i, int b, const float4& c4, const float4& s4) const {
    if (i >= v.n) return;
    const TCoef& s = src[b];
    const size_t o = (size_t)b * v.np + i;
    // np is a multiple of 4: the last group's loads and stores past n stay in the padding
    const float4 x01 = *reinterpret_cast<const float4*>(v.x32 + o), x23 = *reinterpret_cast<const float4*>(v.x32 + o + 2);
    const float4 ri = *reinterpret_cast<const float4*>(v.rinv + i);
    const float Fc[4] = {c4.x * ri.x, c4.y * ri.y, c4.z * ri.z, c4.w * ri.w};
    const float Fs[4] = {s4.x * ri.x, s4.y * ri.y, s4.z * ri.z, s4.w * ri.w};
    const float gv[4] = {s.c1 * (x01.y * Fc[0] - x01.x * Fs[0]), s.c1 * (x01.w * Fc[1] - x01.z * Fs[1]),
                         s.c1 * (x23.y * Fc[2] - x23.x * Fs[2]), s.c1 * (x23.w * Fc[3] - x23.z * Fs[3])};
    if (s.gout >= 0)
      *reinterpret_cast<float4*>(v.g + ((size_t)s.gout * v.bp + b) * v.np + i) = make_float4(gv[0], gv[1], gv[2], gv[3]);
    if (v.mode != 0 && s.rec) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (i + q >= v.n) break;
        v.fin_coup[(o + q) * 2] = Fc[q];
        v.fin_coup[(o + q) * 2 + 1] = Fs[q];
        if (v.mode == 2) v.fin_theta[o + q] = v.omega[i + q] + gv[q];
      }
    }
    if (next) {
      const float4 last = make_float4(gv[0], gv[1], gv[2], gv[3]);
      stage4(v, next[b], b, i, Xn, &last);
    }
  }
};
// the A_lo pass: columns [hi cos | hi sin]; stores the partial couplings
template <int BP> struct LoEpi {
  TView v;
  const TCoef* src;
  __device__ bool f16() const { return !v.bf16; }
  __device__ void row(uint32_t taddr, int row, int m0, int sp) {
    const int i = m0 + row;
#pragma unroll 1
    for (int b0 = 0; b0 < BP; b0 += 16) {
      float hc[16], hs[16];
      umma::tmem_ld16(taddr + 0 * BP + b0, hc);
      umma::tmem_ld16(taddr + 1 * BP + b0, hs);
      umma::tmem_ld_wait();
      if (i >= v.n) continue;
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const int b = sp * BP + b0 + j;
        if (b >= v.B) break;
        v.Flo[((size_t)0 * v.bp + b) * v.np + i] = hc[j];
        v.Flo[((size_t)1 * v.bp + b) * v.np + i] = hs[j];
      }
    }
  }
};

// ---------------------------------------------------------------- reductions
__device__ __forceinline__ float block_sum(float v, float* sh) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) sh[w] = v;
  __syncthreads();
  float t = 0.f;
  if (threadIdx.x == 0)
    for (int q = 0; q < (int)(blockDim.x >> 5); ++q) t += sh[q];
  return t;  // valid on thread 0
}

// whether this block is the last of the gridDim.x blocks of trajectory b to get here; the counter
// is left at zero for the next kernel
__device__ __forceinline__ bool last_of(unsigned* cnt, int b) {
  __shared__ int last;
  if (threadIdx.x == 0) {
    __threadfence();  // this block's partial sums before its arrival
    last = atomicAdd(cnt + b, 1u) == gridDim.x - 1;
    if (last) {
      cnt[b] = 0;
      __threadfence();
    }
  }
  __syncthreads();
  return last;
}
// the nblk values p[q * stride], added in the order of q; every thread of the block calls it
__device__ __forceinline__ float sum_in_order(const float* p, int nblk, int stride, float* buf) {
  __syncthreads();
  for (int q = threadIdx.x; q < nblk; q += blockDim.x) buf[q] = __ldcg(p + (size_t)q * stride);
  __syncthreads();
  float s = 0.f;
  if (threadIdx.x == 0) {
#pragma unroll 8
    for (int q = 0; q < nblk; ++q) s += buf[q];
  }
  return s;  // valid on thread 0
}
constexpr int T_MAXBLK = 1024;  // blocks per trajectory of the two kernels below

// The error norm of stage 7 (dp45.cu:79-84) and the controller (dp45.cu:109-139) of each
// trajectory, which the last block of the trajectory runs: a launch of its own for the controller
// and one thread per trajectory over its partial sums cost 6 us of latency per attempt.  flags[1]
// is cleared for the output kernel, which sets it anew.
__global__ void k_t_error(TView v, const TCoef* src7, double atol, double rtol, float* part, int nblk, TrajG* traj,
                          int fixed, const float* t_eval, int n_eval, unsigned* cnt, int* flags) {
  __shared__ float sh[32];
  __shared__ float buf[T_MAXBLK];
  pdl_launch();
  pdl_wait();
  const int b = blockIdx.y;
  const TCoef& s = src7[b];
  if (b == 0 && blockIdx.x == 0 && threadIdx.x == 0) flags[1] = 0;
  if (!s.active) return;
  float acc = 0.f;
  if (!fixed) {
    const size_t yb = ((size_t)s.base * v.bp + b) * v.np, y7b = ((size_t)(s.base ^ 1) * v.bp + b) * v.np;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < v.n; i += gridDim.x * blockDim.x) {
      float e = 0.f;
#pragma unroll
      for (int j = 0; j < 7; ++j) e = __fmaf_rn(s.E[j], v.g[((size_t)s.slot[j] * v.bp + b) * v.np + i], e);
      float tol = (float)atol;
      if (rtol != 0.0) {
        float a0 = fabsf(__fmaf_rn((float)v.ph_w[yb + i], P2_1, v.ph_hi[yb + i]));
        float a1 = fabsf(__fmaf_rn((float)v.ph_w[y7b + i], P2_1, v.ph_hi[y7b + i]));
        tol = (float)atol + (float)rtol * fmaxf(a0, a1);
      }
      const float ye = e / tol;
      acc = __fmaf_rn(ye, ye, acc);
    }
    const float t = block_sum(acc, sh);
    if (threadIdx.x == 0) part[(size_t)b * nblk + blockIdx.x] = t;
    if (!last_of(cnt, b)) return;
  } else if (blockIdx.x > 0) {
    return;
  }
  const float ss = fixed ? 0.f : sum_in_order(part + (size_t)b * nblk, nblk, 1, buf);
  if (threadIdx.x != 0) return;
  TrajG& T = traj[b];
  const double h = T.h;
  bool accept = true;
  double factor = 1.0;
  if (!fixed) {
    const double norm = sqrt((double)ss) / sqrt((double)v.n);
    if (isnan(norm)) {
      T.status = KURA_ERR_NONFINITE;
      return;
    }
    factor = (double)(0.9f * exp2f(-0.2f * log2f((float)norm)));
    accept = norm < 1.0;
  }
  if (accept) {
    T.t_last = T.t;
    T.t = T.t + h;
    T.rot_y ^= 1;
    T.rot_g ^= 1;
    T.accepted++;
    if (!fixed) T.h = h * fmin(factor, 10.0);
    int e = T.eval_i;
    while (e < n_eval && T.t >= (double)t_eval[e]) e++;
    T.eval_end = e;
  } else {
    T.rejected++;
    if (factor < 1.0) T.h = h * fmax(factor, 0.2);
    if (!(T.h >= 1e-14 * fmax(1.0, fabs(T.t)))) T.status = KURA_ERR_STEP_UNDERFLOW;
  }
}

// The order parameter at the pending output times of each trajectory (dense output, dp45.cu:70-76,
// kuramoto.cu:212-220); the last block of the trajectory writes the records, ends the trajectory
// when it has reached t1 and fills the coefficients of its next attempt (on their own, over all
// trajectories in one block, these took 4 and 15 us per attempt).  first: the call after the
// first slopes.
__global__ void k_t_output(TView v, TrajG* traj, const float* t_eval, float* part, int nblk, float* out_r, int* out_idx,
                           int ring, TCoef* src, unsigned* cnt, int* flags, int first) {
  __shared__ float sh[32];
  __shared__ float buf[T_MAXBLK];
  pdl_launch();
  pdl_wait();
  const int b = blockIdx.y;
  TrajG& T = traj[b];
  const int ncross = min(T.eval_end - T.eval_i, T_MAXC);
  const bool initial = T.need_init != 0;
  const int nrec = initial ? 1 : max(ncross, 0);
  if (nrec == 0 && blockIdx.x > 0) return;
  if (nrec > 0) {
    const size_t bl = initial ? ((size_t)T.rot_y * v.bp + b) * v.np : ((size_t)(T.rot_y ^ 1) * v.bp + b) * v.np;
    // after the accept, k1 of the step sits in the k7 slot and vice versa
    const int k1s = slot_k7(T.rot_g), k7s = slot_k1(T.rot_g);
    __shared__ float sw[9];  // the record's weights: W[0..6], then the time offset hi and lo
    for (int c = 0; c < nrec; ++c) {
      // the weights in double, once per block (FP64 is a small fraction of this GPU's FP32 rate:
      // computed by every thread they cost more than the record's memory traffic)
      if (threadIdx.x == 0) {
        for (int j = 0; j < 9; ++j) sw[j] = 0.f;
        if (!initial) {
          const double hs = T.t - T.t_last, dl = (double)t_eval[T.eval_i + c] - T.t_last, x = dl / hs;
          for (int j = 0; j < 7; ++j) {
            const double cc = ((P_TAB[j][3] * x + P_TAB[j][2]) * x + P_TAB[j][1]) * x * x + P_TAB[j][0] * x;
            sw[j] = (float)(hs * cc);
          }
          const float mh0 = (float)dl;
          sw[7] = mh0;
          sw[8] = (float)(dl - (double)mh0);
        }
      }
      __syncthreads();
      float W[7];
#pragma unroll
      for (int j = 0; j < 7; ++j) W[j] = sw[j];
      const float mh = sw[7], ml = sw[8];
      float ax = 0.f, ay = 0.f;
      for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < v.n; i += gridDim.x * blockDim.x) {
        float gsum = 0.f;
        if (!initial) {
          gsum = __fmaf_rn(W[0], v.g[((size_t)k1s * v.bp + b) * v.np + i], gsum);
          for (int j = 1; j < 6; ++j) gsum = __fmaf_rn(W[j], v.g[((size_t)j * v.bp + b) * v.np + i], gsum);
          gsum = __fmaf_rn(W[6], v.g[((size_t)k7s * v.bp + b) * v.np + i], gsum);
        }
        const float om = v.omega[i];
        const f2 pr = two_prod(om, mh);
        const f2 s1 = two_sum(v.ph_hi[bl + i], pr.hi);
        const f2 s2 = two_sum(s1.hi, gsum);
        const float lo = v.ph_lo[bl + i] + ((s1.lo + s2.lo) + __fmaf_rn(om, ml, pr.lo));
        float sn, cs;
        sincos_pair(s2.hi, lo, &sn, &cs);
        ax += cs;
        ay += sn;
      }
      const float tx = block_sum(ax, sh);
      const float ty = block_sum(ay, sh);
      if (threadIdx.x == 0) {
        part[(((size_t)b * T_MAXC + c) * nblk + blockIdx.x) * 2] = tx;
        part[(((size_t)b * T_MAXC + c) * nblk + blockIdx.x) * 2 + 1] = ty;
      }
    }
    if (!last_of(cnt, b)) return;
    for (int c = 0; c < nrec; ++c) {
      const float* pc = part + ((size_t)b * T_MAXC + c) * nblk * 2;
      const float X = sum_in_order(pc, nblk, 2, buf), Y = sum_in_order(pc + 1, nblk, 2, buf);
      if (threadIdx.x == 0 && T.out_count < ring) {
        const float xn = X / (float)v.n, yn = Y / (float)v.n;
        out_r[(size_t)b * ring + T.out_count] = sqrtf(xn * xn + yn * yn);
        out_idx[(size_t)b * ring + T.out_count] = initial ? -1 : T.eval_i;
        T.out_count++;
        if (!initial) T.eval_i++;
      }
    }
    if (threadIdx.x == 0) {
      if (initial) T.need_init = 0;
      else if (T.eval_i < T.eval_end && T.out_count >= ring) T.status = KURA_ERR_UNSUPPORTED;  // no room for the rest
    }
  }
  if (threadIdx.x == 0) {
    if (first) T.need_k1 = 0;
    if (T.status == 0 && !(T.t < T.t1) && T.eval_i >= T.eval_end) T.status = 1;
  }
  __syncthreads();
  fill_attempt(T, src, v.bp, b, threadIdx.x, flags);
}

// N*A for the volcano rule, exact in F16 (integers in [-K, K], K <= 2048; hi + lo above)
__global__ void k_t_volcano_f16(const uint32_t* __restrict__ bits, int n, int k, int words, int np,
                                __half* __restrict__ A, __half* __restrict__ Alo) {
  for (int i = blockIdx.y; i < np; i += gridDim.y)
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < np; j += gridDim.x * blockDim.x) {
      int kk = 0;
      if (i < n && j < n) {
        for (int wd = 0; wd < words; ++wd) {
          const int m0 = 32 * wd, cnt = min(32, k - m0);
          const uint32_t valid = cnt >= 32 ? 0xffffffffu : ((1u << cnt) - 1u);
          const uint32_t even = 0x55555555u & valid, odd = 0xAAAAAAAAu & valid;
          const uint32_t dis = bits[(size_t)wd * n + i] ^ bits[(size_t)wd * n + j];
          kk += __popc(even) - __popc(odd) - 2 * __popc(dis & even) + 2 * __popc(dis & odd);
        }
      }
      const __half hi = __float2half_rn((float)kk);
      A[(size_t)i * np + j] = hi;
      if (Alo) Alo[(size_t)i * np + j] = __float2half_rn((float)kk - __half2float(hi));
    }
}
__global__ void k_t_fill(float* p, int n, float v) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) p[i] = v;
}
// general adjacency, one block per row: 2^p N A = hi + lo in F16, 11 bits each, with 2^p so that the
// row's largest entry lies in [2^14, 2^15) (1 for a row of zeros).  *wide is set where F16 holds an
// entry less well than BF16 would: one below 2^-7, whose lo part meets F16's smallest step, one that is
// not finite, or a row below what 2^-p / N / X_SCALE can undo.
__global__ void k_t_split(const float* __restrict__ adj, int n, int np, float scale, __half* hi, __half* lo,
                          float* rinv, int* wide) {
  __shared__ float sh[32];
  __shared__ float smax;
  for (int i = blockIdx.x; i < np; i += gridDim.x) {
    float m = 0.f;
    if (i < n)
      for (int j = threadIdx.x; j < n; j += blockDim.x) m = fmaxf(m, fabsf(adj[(size_t)i * n + j] * scale));
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    __syncthreads();
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 1; w < (int)(blockDim.x >> 5); ++w) m = fmaxf(m, sh[w]);
      int e = 15;  // frexp's exponent: m in [2^(e-1), 2^e)
      if (m > 0.f && isfinite(m)) frexpf(m, &e);
      if (e < -70) {
        e = 15;
        *wide = 1;
      }
      smax = ldexpf(1.f, 15 - e);
      rinv[i] = (1.f / scale) * ldexpf(1.f, e - 15) * (1.f / X_SCALE);
    }
    __syncthreads();
    const float p = smax;
    bool out = false;
    for (int j = threadIdx.x; j < np; j += blockDim.x) {
      const float a0 = (i < n && j < n) ? adj[(size_t)i * n + j] * scale : 0.f, a = a0 * p;
      out |= !isfinite(a) || (a0 != 0.f && fabsf(a) < 0.0078125f);
      const __half h = __float2half_rn(a);
      hi[(size_t)i * np + j] = h;
      lo[(size_t)i * np + j] = __float2half_rn(a - __half2float(h));
    }
    if (out) *wide = 1;
  }
}
// the same in BF16: N A = hi + lo, 8 bits each
__global__ void k_t_split_bf16(const float* __restrict__ adj, int n, int np, float scale, __nv_bfloat16* hi,
                               __nv_bfloat16* lo, float* rinv) {
  for (int i = blockIdx.x; i < np; i += gridDim.x) {
    if (threadIdx.x == 0) rinv[i] = 1.f / scale;
    for (int j = threadIdx.x; j < np; j += blockDim.x) {
      const float a = (i < n && j < n) ? adj[(size_t)i * n + j] * scale : 0.f;
      const __nv_bfloat16 h = __float2bfloat16_rn(a);
      hi[(size_t)i * np + j] = h;
      lo[(size_t)i * np + j] = __float2bfloat16_rn(a - __bfloat162float(h));
    }
  }
}
__global__ void k_t_adj_out(const uint16_t* hi, const uint16_t* lo, int n, int np, const float* rinv, int bf16, float* adj) {
  auto part = [&](uint16_t h) {
    return bf16 ? __bfloat162float(__ushort_as_bfloat16(h)) : __half2float(__ushort_as_half(h));
  };
  for (int i = blockIdx.y; i < n; i += gridDim.y)
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
      float a = part(hi[(size_t)i * np + j]);
      if (lo) a += part(lo[(size_t)i * np + j]);
      adj[(size_t)i * n + j] = __fmul_rn(a, bf16 ? rinv[i] : rinv[i] * X_SCALE);
    }
}

}  // namespace

// ====================================================================== host engine
struct TensorEngine::Impl {
  int n = 0, np = 0, bp = 0, B = 0, K = 0, seed = 1, fixed = 0, dense_level = 0, device = 0;
  double atol = 1e-6, rtol = 0.0;
  cudaStream_t st = nullptr;
  float* omega = nullptr;
  float* ph_hi = nullptr;
  float* ph_lo = nullptr;
  long long* ph_w = nullptr;
  float* g = nullptr;
  __half* X = nullptr;
  float2* x32 = nullptr;
  __half* Ahi = nullptr;  // (the 16-bit buffers hold BF16 where bf16 is set)
  __half* Alo = nullptr;
  float* Flo = nullptr;
  float* rinv = nullptr;  // [np] scale of each row's couplings
  float* fin_theta = nullptr;
  float* fin_coup = nullptr;
  TrajG* traj = nullptr;
  TCoef* src = nullptr;       // [8][bp]
  float* part = nullptr;      // reductions
  float* t_eval = nullptr;
  float* out_r = nullptr;
  int* out_idx = nullptr;
  int* ctl = nullptr;       // flags, err, a word for k_t_split and cnt in one piece, cleared and read at once
  int* err = nullptr;
  int* flags = nullptr;     // [0]: a trajectory needs its first slope, [1]: one steps in the next attempt; the GEMMs skip on 0
  unsigned* cnt = nullptr;  // [bp] arrivals of a trajectory's blocks
  int* h_run = nullptr;     // pinned: the flags and the error code
  // pinned copies of a small ensemble's uploads, and whether one is still on its way
  float* h_theta = nullptr;
  TrajG* h_traj = nullptr;
  std::vector<char> on_its_way;
  size_t t_eval_cap = 0, ring_cap = 0;
  int graph_ring = 0, graph_n_eval = 0;  // what the attempt graph was captured with
  void drop_graph() {
    if (graph) cudaGraphExecDestroy(graph);
    graph = nullptr;
  }
  // the product's form (parts of A, their map, the split) goes into the attempt graph
  void new_adjacency(bool lo, bool bf) {
    has_lo = lo;
    bf16 = bf;
    adj_set = true;
    shaped = false;
    drop_graph();
  }
  int ring = 0, n_eval = 0, nblk = 1;
  CUtensorMap tmA, tmAlo, tmX, tmXhi, tmX2, tmX2hi;
  // the second operand buffer: the split GEMM reads one and makes the next stage's operands in the other
  __half* X2 = nullptr;
  // The rule: a thread of the split GEMM then has one group of four rows, so that nothing in its
  // epilogue waits for a second pass over the slopes.  Whole runs, with the stage kernel / in the
  // epilogue: 3000 x 24 (one group) 8.41 / 8.07 ms; 6007 x 64 (3.2 groups a thread) 5.55 / 5.71 ms.
  bool one_group() const { return shaped && shape.mt != 0 && shape.mt * x_bph(bp) * (TG_BM / 4) <= shape.s * TS_THREADS; }
  bool fused() const { return X2 && one_group(); }
  bool has_lo = false, adj_set = false, bf16 = false;
  SplitShape shape;  // how the coupling GEMM runs, chosen at its first launch
  bool shaped = false;
  cudaGraphExec_t graph = nullptr;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  // KURA_TIME_COUPLING=1: event nodes around the six coupling GEMMs of the attempt graph; the
  // durations of the last replay of each batch of replays are summed into the stats
  bool time_gemm = false;
  cudaEvent_t gev[12] = {};
};

static std::string g_terr;
#define TCU(x)                                                               \
  do {                                                                       \
    cudaError_t e_ = (x);                                                    \
    if (e_ != cudaSuccess) {                                                 \
      g_terr = std::string(#x) + ": " + cudaGetErrorString(e_);              \
      return e_ == cudaErrorMemoryAllocation ? KURA_ERR_NOMEM : KURA_ERR_CUDA; \
    }                                                                        \
  } while (0)

const char* TensorEngine::last_error() { return g_terr.c_str(); }

template <typename T> static cudaError_t zalloc(T** p, size_t count) {
  cudaError_t e = cudaMalloc((void**)p, std::max<size_t>(count, 1) * sizeof(T));
  if (e == cudaSuccess) e = cudaMemset(*p, 0, std::max<size_t>(count, 1) * sizeof(T));
  // the memset runs on the legacy default stream, which does not order with the non-blocking
  // stream a handle may own: wait for it, so that no later copy on that stream lands first
  if (e == cudaSuccess) e = cudaStreamSynchronize(0);
  return e;
}

TensorEngine::TensorEngine() : d(new Impl) {}
TensorEngine::~TensorEngine() {
  void* ptrs[] = {d->omega, d->ph_hi, d->ph_lo, d->ph_w, d->g, d->X, d->X2, d->x32, d->Ahi, d->Alo, d->Flo, d->rinv, d->fin_theta,
                  d->fin_coup, d->traj, d->src, d->part, d->t_eval, d->out_r, d->out_idx, d->ctl};
  for (void* p : ptrs)
    if (p) cudaFree(p);
  if (d->h_run) cudaFreeHost(d->h_run);
  if (d->h_theta) cudaFreeHost(d->h_theta);
  if (d->h_traj) cudaFreeHost(d->h_traj);
  if (d->graph) cudaGraphExecDestroy(d->graph);
  if (d->ev0) cudaEventDestroy(d->ev0);
  if (d->ev1) cudaEventDestroy(d->ev1);
  for (cudaEvent_t e : d->gev)
    if (e) cudaEventDestroy(e);
  delete d;
}

int TensorEngine::init(int64_t n, int k, int batch, int seed, double atol, double rtol, int fixed, int dense_level,
                       int device, cudaStream_t st) {
  if (batch < 1 || batch > 128) { g_terr = "tensor engine: batch must be 1..128"; return KURA_ERR_UNSUPPORTED; }
  if (dense_level >= 1) { g_terr = "tensor engine keeps the order parameter only (dense level 0)"; return KURA_ERR_UNSUPPORTED; }
  if (n < 1 || n > (1LL << 20)) { g_terr = "tensor engine: n must be in [1, 2^20]"; return KURA_ERR_UNSUPPORTED; }
  Impl& I = *d;
  I.n = (int)n; I.K = k; I.B = batch; I.seed = seed; I.atol = atol; I.rtol = rtol; I.fixed = fixed;
  I.dense_level = dense_level; I.device = device; I.st = st;
  I.np = (I.n + 255) / 256 * 256;  // work units of two 128-row tiles
  I.bp = 16;
  while (I.bp < batch) I.bp *= 2;
  const size_t np = I.np, bp = I.bp;
  I.nblk = std::min(T_MAXBLK, (I.n + T_RBLK - 1) / T_RBLK);
  TCU(zalloc(&I.omega, np));
  TCU(zalloc(&I.ph_hi, 2 * bp * np));
  TCU(zalloc(&I.ph_lo, 2 * bp * np));
  TCU(zalloc(&I.ph_w, 2 * bp * np));
  TCU(zalloc(&I.g, 7 * bp * np));
  TCU(zalloc(&I.X, 4 * bp * np));
  TCU(zalloc(&I.x32, bp * np));
  TCU(zalloc(&I.Ahi, np * np));
  TCU(zalloc(&I.rinv, np));
  TCU(zalloc(&I.fin_theta, bp * np));
  TCU(zalloc(&I.fin_coup, 2 * bp * np));
  TCU(zalloc(&I.traj, bp));
  TCU(zalloc(&I.src, 8 * bp));
  TCU(zalloc(&I.part, (size_t)bp * T_MAXC * I.nblk * 2));
  TCU(zalloc(&I.ctl, 4 + bp));
  I.flags = I.ctl;
  I.err = I.ctl + 2;
  I.cnt = reinterpret_cast<unsigned*>(I.ctl + 4);
  TCU(cudaHostAlloc((void**)&I.h_run, 3 * sizeof(int), cudaHostAllocDefault));
  // from 4 MB of phases on the copies themselves outweigh the waits
  if ((size_t)I.B * I.n * sizeof(float) <= (4u << 20)) {
    TCU(cudaHostAlloc((void**)&I.h_theta, (size_t)I.B * I.n * sizeof(float), cudaHostAllocDefault));
    TCU(cudaHostAlloc((void**)&I.h_traj, sizeof(TrajG) * I.B, cudaHostAllocDefault));
    I.on_its_way.assign(I.B, 0);
  }
  TCU(cudaEventCreate(&I.ev0));
  TCU(cudaEventCreate(&I.ev1));
  const char* tg = getenv("KURA_TIME_COUPLING");
  I.time_gemm = tg && atoi(tg) != 0;
  if (I.time_gemm)
    for (cudaEvent_t& e : I.gev) TCU(cudaEventCreate(&e));
  // X is [4 bp][np]: a work unit's column block is 4 * x_bph(bp) rows (its hi + lo columns),
  // of which the A_lo pass reads the first half
  if (make_tmap_16(&I.tmA, true, I.Ahi, np, np, TG_BM, TE_BK) ||
      make_tmap_16(&I.tmX, true, I.X, np, 4 * bp, 4 * x_bph(I.bp), TE_BK) ||
      make_tmap_16(&I.tmXhi, true, I.X, np, 4 * bp, 2 * x_bph(I.bp), TE_BK)) {
    g_terr = "cuTensorMapEncodeTiled failed";
    return KURA_ERR_CUDA;
  }
  return KURA_OK;
}

size_t TensorEngine::memory_required(int64_t n, int batch) {
  size_t np = ((size_t)n + 255) / 256 * 256, bp = 16;
  while ((int)bp < batch) bp *= 2;
  return np * np * 2 + np * bp * (2 * 16 + 7 * 4 + 4 * 2 + 8 + 4 + 8) + np * 8;
}

int TensorEngine::set_frequencies(const float* omega) {
  TCU(cudaMemcpyAsync(d->omega, omega, sizeof(float) * d->n, cudaMemcpyHostToDevice, d->st));
  TCU(cudaStreamSynchronize(d->st));
  return KURA_OK;
}

int TensorEngine::generate_adjacency() {
  Impl& I = *d;
  const int words = (I.K + 31) / 32;
  uint32_t* bits = nullptr;
  if (words > 0) {
    TCU(cudaMalloc((void**)&bits, sizeof(uint32_t) * (size_t)words * I.n));
    TCU(launch_volcano_words(I.seed, I.n, I.K, words, bits, I.st));
  }
  // N*A_ij is an integer in [-K, K]: exact in F16 for K <= 2048, else as hi + lo
  const bool need_lo = I.K > 2048;
  if (need_lo && !I.Alo) TCU(zalloc(&I.Alo, (size_t)I.np * I.np));
  if (need_lo && !I.Flo) TCU(zalloc(&I.Flo, (size_t)2 * I.bp * I.np));
  dim3 grid((unsigned)std::min((I.np + 255) / 256, 64), (unsigned)std::min(I.np, 65535));
  k_t_volcano_f16<<<grid, 256, 0, I.st>>>(bits, I.n, I.K, words, I.np, I.Ahi, need_lo ? I.Alo : nullptr);
  k_t_fill<<<(I.np + 255) / 256, 256, 0, I.st>>>(I.rinv, I.np, (1.0f / (float)I.n) * (1.f / X_SCALE));
  TCU(cudaGetLastError());
  TCU(cudaStreamSynchronize(I.st));
  if (bits) cudaFree(bits);
  if (need_lo && make_tmap_16(&I.tmAlo, true, I.Alo, I.np, I.np, TG_BM, TE_BK)) {
    g_terr = "cuTensorMapEncodeTiled failed";
    return KURA_ERR_CUDA;
  }
  I.new_adjacency(need_lo, false);
  return KURA_OK;
}

int TensorEngine::set_adjacency(const float* adj_host) {
  Impl& I = *d;
  float* dadj = nullptr;
  TCU(cudaMalloc((void**)&dadj, sizeof(float) * (size_t)I.n * I.n));
  TCU(cudaMemcpyAsync(dadj, adj_host, sizeof(float) * (size_t)I.n * I.n, cudaMemcpyHostToDevice, I.st));
  if (!I.Alo) TCU(zalloc(&I.Alo, (size_t)I.np * I.np));
  if (!I.Flo) TCU(zalloc(&I.Flo, (size_t)2 * I.bp * I.np));
  int wide = 0;
  TCU(cudaMemsetAsync(I.ctl + 3, 0, sizeof(int), I.st));
  k_t_split<<<(unsigned)std::min(I.np, 65535), 256, 0, I.st>>>(dadj, I.n, I.np, (float)I.n, I.Ahi, I.Alo, I.rinv, I.ctl + 3);
  TCU(cudaGetLastError());
  TCU(cudaMemcpyAsync(&wide, I.ctl + 3, sizeof(int), cudaMemcpyDeviceToHost, I.st));
  TCU(cudaStreamSynchronize(I.st));
  if (wide) {
    k_t_split_bf16<<<(unsigned)std::min(I.np, 65535), 256, 0, I.st>>>(dadj, I.n, I.np, (float)I.n, (__nv_bfloat16*)I.Ahi,
                                                                      (__nv_bfloat16*)I.Alo, I.rinv);
    TCU(cudaGetLastError());
    TCU(cudaStreamSynchronize(I.st));
  }
  cudaFree(dadj);
  if (make_tmap_16(&I.tmAlo, true, I.Alo, I.np, I.np, TG_BM, TE_BK)) {
    g_terr = "cuTensorMapEncodeTiled failed";
    return KURA_ERR_CUDA;
  }
  I.new_adjacency(true, wide != 0);
  return KURA_OK;
}

int TensorEngine::get_adjacency(float* adj_host) {
  Impl& I = *d;
  float* dadj = nullptr;
  TCU(cudaMalloc((void**)&dadj, sizeof(float) * (size_t)I.n * I.n));
  dim3 grid((unsigned)std::min((I.n + 255) / 256, 64), (unsigned)std::min(I.n, 65535));
  k_t_adj_out<<<grid, 256, 0, I.st>>>((const uint16_t*)I.Ahi, I.has_lo ? (const uint16_t*)I.Alo : nullptr, I.n, I.np, I.rinv,
                                      I.bf16 ? 1 : 0, dadj);
  TCU(cudaGetLastError());
  TCU(cudaMemcpyAsync(adj_host, dadj, sizeof(float) * (size_t)I.n * I.n, cudaMemcpyDeviceToHost, I.st));
  TCU(cudaStreamSynchronize(I.st));
  cudaFree(dadj);
  return KURA_OK;
}

int TensorEngine::set_state(int b, const float* theta_dev, const TrajG& T) {
  Impl& I = *d;
  const size_t off = (size_t)b * I.np;  // phase buffer 0
  TCU(launch_init_state(theta_dev, I.n, I.np, I.ph_hi + off, I.ph_lo + off, I.ph_w + off, I.st));
  TCU(cudaMemcpyAsync(I.traj + b, &T, sizeof(TrajG), cudaMemcpyHostToDevice, I.st));
  TCU(cudaStreamSynchronize(I.st));
  return KURA_OK;
}
int TensorEngine::upload_state(int b, const float* theta, const TrajG& T) {
  Impl& I = *d;
  float* dev = staging(b);
  if (!I.h_theta) {
    TCU(cudaMemcpyAsync(dev, theta, sizeof(float) * I.n, cudaMemcpyHostToDevice, I.st));
    return set_state(b, dev, T);
  }
  if (I.on_its_way[b]) {  // its pinned copy may still be read
    TCU(cudaStreamSynchronize(I.st));
    I.on_its_way.assign(I.B, 0);
  }
  float* pin = I.h_theta + (size_t)b * I.n;
  std::memcpy(pin, theta, sizeof(float) * I.n);
  I.h_traj[b] = T;
  I.on_its_way[b] = 1;
  const size_t off = (size_t)b * I.np;  // phase buffer 0
  TCU(cudaMemcpyAsync(dev, pin, sizeof(float) * I.n, cudaMemcpyHostToDevice, I.st));
  TCU(launch_init_state(dev, I.n, I.np, I.ph_hi + off, I.ph_lo + off, I.ph_w + off, I.st));
  TCU(cudaMemcpyAsync(I.traj + b, I.h_traj + b, sizeof(TrajG), cudaMemcpyHostToDevice, I.st));
  return KURA_OK;
}
float* TensorEngine::staging(int b) { return d->fin_theta + (size_t)b * d->np; }

int TensorEngine::set_horizon(const std::vector<float>& t_eval, int ring, std::vector<TrajG>& traj) {
  Impl& I = *d;
  I.n_eval = (int)t_eval.size();
  // the buffers of an earlier horizon serve as long as they are large enough, and the attempt graph
  // as long as nothing that it was captured with has changed
  const bool grow_t = !I.t_eval || t_eval.size() > I.t_eval_cap;
  const bool grow_r = !I.out_r || (size_t)ring > I.ring_cap;
  if (grow_t || grow_r || I.graph_ring != ring || I.graph_n_eval != I.n_eval) I.drop_graph();
  if (grow_t) {
    if (I.t_eval) cudaFree(I.t_eval);
    I.t_eval = nullptr;
    TCU(zalloc(&I.t_eval, t_eval.size()));
    I.t_eval_cap = t_eval.size();
  }
  if (grow_r) {
    I.ring_cap = 0;  // until both are there
    if (I.out_r) cudaFree(I.out_r);
    if (I.out_idx) cudaFree(I.out_idx);
    I.out_r = nullptr; I.out_idx = nullptr;
    TCU(zalloc(&I.out_r, (size_t)I.bp * ring));
    TCU(zalloc(&I.out_idx, (size_t)I.bp * ring));
    I.ring_cap = ring;
  }
  I.ring = ring;
  if (!t_eval.empty())
    TCU(cudaMemcpyAsync(I.t_eval, t_eval.data(), sizeof(float) * t_eval.size(), cudaMemcpyHostToDevice, I.st));
  TCU(cudaMemcpyAsync(I.traj, traj.data(), sizeof(TrajG) * I.B, cudaMemcpyHostToDevice, I.st));
  TCU(cudaStreamSynchronize(I.st));
  if (!I.on_its_way.empty()) I.on_its_way.assign(I.B, 0);
  return KURA_OK;
}

template <int NCOL, int MT>
static int clusters_at_once(int s) {
  auto k = k_split_gemm<NCOL, MT, SplitEpi>;
  if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, TSCfg<NCOL, MT>::SMEM) != cudaSuccess) return 0;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = s;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)s);
  cfg.blockDim = dim3(TS_THREADS);
  cfg.dynamicSmemBytes = TSCfg<NCOL, MT>::SMEM;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, (void*)k, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

template <int NCOL, int MT>
static cudaError_t launch_split(TensorEngine::Impl& I, const TView& v, const TCoef* src, int s, int ktiles, int nsplit,
                                int xstride, const int* run_flag, int xbuf, const TCoef* next) {
  using C = TSCfg<NCOL, MT>;
  auto k = k_split_gemm<NCOL, MT, SplitEpi>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
  if (e != cudaSuccess) return e;
  const int tiles = (I.n + TG_BM - 1) / TG_BM;
  return launch_pdl(k, dim3((unsigned)((tiles + MT - 1) / MT * nsplit * s)), TS_THREADS, C::SMEM, I.st, s, I.tmA,
                    I.has_lo ? I.tmAlo : I.tmA, xbuf ? I.tmX2 : I.tmX, xbuf ? I.tmX2hi : I.tmXhi, ktiles, s, nsplit, xstride, I.has_lo ? 1 : 0,
                    SplitEpi{v, src, next, xbuf ? I.X : I.X2}, I.err, 20000000000ull, run_flag);
}

template <int NCOL>
static cudaError_t launch_gemm(TensorEngine::Impl& I, const TCoef* src, int mode, const int* run_flag, int xbuf,
                               const TCoef* next) {
  TView v{I.n, I.np, I.bp, I.B, mode, I.omega, I.ph_hi, I.ph_lo, I.ph_w, I.g, I.X, I.x32, I.fin_theta, I.fin_coup,
          I.Flo, I.rinv, I.bf16};
  constexpr int BP = NCOL / 4;  // trajectories per work unit
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, I.device);
  const int mtiles = I.np / (2 * TG_BM), ktiles = I.np / TE_BK;  // groups of two row tiles
  const int nsplit = I.bp / BP, xstride = 4 * BP;
  const int grid = std::min(mtiles * nsplit, sms);
  // Units of two row tiles fill whole waves of the grid; the rest run as one-tile units, when
  // that shortens the last wave (in unit times: a one-tile unit is half of a two-tile one)
  int big = mtiles;
  double waves = 0;
  {
    const int full = (mtiles * nsplit) / grid;
    const int b = full * grid / nsplit;
    const int tail = (mtiles - b) * 2 * nsplit;
    const double t_split = full + 0.5 * ((tail + grid - 1) / grid);
    const double t_big = (mtiles * nsplit + grid - 1) / grid;
    if (b < mtiles && t_split < t_big) big = b;
    waves = std::min(t_split, t_big);
  }
  if (!I.shaped) {
    I.shape = split_shape((I.n + TG_BM - 1) / TG_BM, nsplit, NCOL, ktiles, waves,
                          [&](int mt, int s) { return mt == 1 ? clusters_at_once<NCOL, 1>(s) : clusters_at_once<NCOL, 2>(s); });
    I.shaped = true;
  }
  const SplitShape sh = I.shape;
  if (sh.mt == 1) return launch_split<NCOL, 1>(I, v, src, sh.s, ktiles, nsplit, xstride, run_flag, xbuf, next);
  if (sh.mt == 2) return launch_split<NCOL, 2>(I, v, src, sh.s, ktiles, nsplit, xstride, run_flag, xbuf, next);
  const unsigned long long limit = 20000000000ull;
  if (I.has_lo) {
    auto kl = k_tensor_gemm<NCOL / 2, LoEpi<BP>, 2, TE_BK>;
    cudaFuncSetAttribute(kl, cudaFuncAttributeMaxDynamicSharedMemorySize, TGCfg<NCOL / 2, 2, TE_BK>::SMEM);
    LoEpi<BP> le{v, src};
    kl<<<grid, TG_THREADS, TGCfg<NCOL / 2, 2, TE_BK>::SMEM, I.st>>>(I.tmAlo, I.tmXhi, mtiles, big, ktiles, nsplit, xstride, le,
                                                             I.err, limit, run_flag);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  auto k = k_tensor_gemm<NCOL, KuraEpi<BP>, 2, TE_BK>;
  cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, TGCfg<NCOL, 2, TE_BK>::SMEM);
  KuraEpi<BP> ep{v, src, I.has_lo ? 1 : 0};
  k<<<grid, TG_THREADS, TGCfg<NCOL, 2, TE_BK>::SMEM, I.st>>>(I.tmA, I.tmX, mtiles, big, ktiles, nsplit, xstride, ep, I.err, limit,
                                                   run_flag);
  return cudaGetLastError();
}

// one unit holds up to 64 trajectories (NCOL = 256: two accumulators fit in TMEM); a batch
// of 128 is two column blocks per row tile
static cudaError_t gemm(TensorEngine::Impl& I, const TCoef* src, int mode, const int* run_flag, int xbuf,
                        const TCoef* next) {
  switch (I.bp) {
    case 16: return launch_gemm<64>(I, src, mode, run_flag, xbuf, next);
    case 32: return launch_gemm<128>(I, src, mode, run_flag, xbuf, next);
    default: return launch_gemm<256>(I, src, mode, run_flag, xbuf, next);
  }
}

// xbuf: the operand buffer; made: its operands are there already; next: the coefficients of the stage
// whose operands the GEMM makes
static cudaError_t coupling(TensorEngine::Impl& I, const TCoef* src, int mode, float* fin_theta, const int* run_flag,
                            int timed = -1, int xbuf = 0, bool made = false, const TCoef* next = nullptr) {
  TView v{I.n, I.np, I.bp, I.B, mode, I.omega, I.ph_hi, I.ph_lo, I.ph_w, I.g, I.X, I.x32, fin_theta, I.fin_coup,
          I.Flo, I.rinv, I.bf16};
  cudaError_t e = cudaSuccess;
  if (!made)
    e = launch_pdl(k_t_stage, dim3((unsigned)((I.n + 4 * ST_THREADS - 1) / (4 * ST_THREADS)), (unsigned)I.B), ST_THREADS, 0,
                   I.st, 1, v, src);
  if (e != cudaSuccess) return e;
  const bool tm = I.time_gemm && timed >= 0;
  if (tm && (e = cudaEventRecordWithFlags(I.gev[2 * timed], I.st, cudaEventRecordExternal)) != cudaSuccess) return e;
  if ((e = gemm(I, src, mode, run_flag, xbuf, next)) != cudaSuccess) return e;
  if (tm) e = cudaEventRecordWithFlags(I.gev[2 * timed + 1], I.st, cudaEventRecordExternal);
  return e;
}

static cudaError_t output(TensorEngine::Impl& I, int first) {
  TView v{I.n, I.np, I.bp, I.B, 0, I.omega, I.ph_hi, I.ph_lo, I.ph_w, I.g, I.X, I.x32, nullptr, I.fin_coup, I.Flo, I.rinv, I.bf16};
  return launch_pdl(k_t_output, dim3((unsigned)I.nblk, (unsigned)I.B), T_RBLK, 0, I.st, 1, v, I.traj, I.t_eval, I.part,
                    I.nblk, I.out_r, I.out_idx, I.ring, I.src, I.cnt, I.flags, first);
}

// one attempt of every trajectory, its outputs, and the coefficients of the next
static cudaError_t attempt(TensorEngine::Impl& I) {
  TView v{I.n, I.np, I.bp, I.B, 0, I.omega, I.ph_hi, I.ph_lo, I.ph_w, I.g, I.X, I.x32, nullptr, I.fin_coup, I.Flo, I.rinv, I.bf16};
  cudaError_t e = cudaSuccess;
  for (int s = 2; s <= 7; ++s) {
    const TCoef* src = I.src + (size_t)(s - 1) * I.bp;
    if (I.fused())
      e = coupling(I, src, 0, nullptr, I.flags + 1, s - 2, s & 1, s > 2, s < 7 ? src + I.bp : nullptr);
    else
      e = coupling(I, src, 0, nullptr, I.flags + 1, s - 2);
    if (e != cudaSuccess) return e;
  }
  e = launch_pdl(k_t_error, dim3((unsigned)(I.fixed ? 1 : I.nblk), (unsigned)I.B), T_RBLK, 0, I.st, 1, v,
                 I.src + 6 * (size_t)I.bp, I.atol, I.rtol, I.part, I.nblk, I.traj, I.fixed, I.t_eval, I.n_eval, I.cnt, I.flags);
  if (e != cudaSuccess) return e;
  return output(I, 0);
}

int TensorEngine::run(std::vector<TrajG>& traj, kura_stats& stats, long long max_replays) {
  Impl& I = *d;
  if (!I.adj_set) { g_terr = "adjacency not set"; return KURA_ERR_INVALID; }
  TCU(cudaMemsetAsync(I.ctl, 0, sizeof(int) * (4 + I.bp), I.st));
  TCU(cudaEventRecord(I.ev0, I.st));
  // first slope of the run, the record at t0 and the coefficients of the first attempt
  k_t_first<<<I.B, 32, 0, I.st>>>(I.traj, I.src, I.flags);
  TCU(cudaGetLastError());
  TCU(coupling(I, I.src, 0, nullptr, I.flags));
  TCU(output(I, 1));
  if (!I.graph) {
    if (I.one_group() && !I.X2) {
      // without room for it the stage kernel goes on making all operands
      if (zalloc(&I.X2, 4 * (size_t)I.bp * I.np) != cudaSuccess ||
          make_tmap_16(&I.tmX2, true, I.X2, I.np, 4 * I.bp, 4 * x_bph(I.bp), TE_BK) ||
          make_tmap_16(&I.tmX2hi, true, I.X2, I.np, 4 * I.bp, 2 * x_bph(I.bp), TE_BK)) {
        cudaGetLastError();
        if (I.X2) cudaFree(I.X2);
        I.X2 = nullptr;
      }
    }
    cudaGraph_t gr;
    TCU(cudaStreamBeginCapture(I.st, cudaStreamCaptureModeThreadLocal));
    cudaError_t e = attempt(I);
    cudaError_t e2 = cudaStreamEndCapture(I.st, &gr);
    if (e != cudaSuccess || e2 != cudaSuccess) {
      g_terr = std::string("graph capture: ") + cudaGetErrorString(e != cudaSuccess ? e : e2);
      return KURA_ERR_CUDA;
    }
    TCU(cudaGraphInstantiate(&I.graph, gr, 0));
    cudaGraphDestroy(gr);
    I.graph_ring = I.ring;
    I.graph_n_eval = I.n_eval;
  }
  long long launches = 0;
  while (true) {
    for (int r = 0; r < 4; ++r) {
      TCU(cudaGraphLaunch(I.graph, I.st));
      launches++;
    }
    TCU(cudaMemcpyAsync(I.h_run, I.ctl, 3 * sizeof(int), cudaMemcpyDeviceToHost, I.st));
    TCU(cudaStreamSynchronize(I.st));
    if (I.h_run[2]) { g_terr = "tensor GEMM aborted (wait time limit)"; return KURA_ERR_BARRIER_TIMEOUT; }
    if (!I.h_run[1]) break;
    if (I.time_gemm) {  // every replay of this batch stepped some trajectory: sample the last one
      for (int q = 0; q < 6; ++q) {
        float gm = 0.f;
        if (cudaEventElapsedTime(&gm, I.gev[2 * q], I.gev[2 * q + 1]) == cudaSuccess) {
          stats.coupling_ms += gm;
          stats.coupling_launches++;
        }
      }
    }
    if (max_replays > 0 && launches >= max_replays) break;
  }
  TCU(cudaEventRecord(I.ev1, I.st));
  TCU(cudaMemcpyAsync(traj.data(), I.traj, sizeof(TrajG) * I.B, cudaMemcpyDeviceToHost, I.st));
  TCU(cudaStreamSynchronize(I.st));
  float ms = 0;
  TCU(cudaEventElapsedTime(&ms, I.ev0, I.ev1));
  stats.kernel_ms += ms;
  stats.launches += launches;
  return KURA_OK;
}

int TensorEngine::read_orders(int count, std::vector<float>& r, std::vector<int>& idx) {
  const size_t w = sizeof(float) * count, pitch = sizeof(float) * d->ring;
  r.resize((size_t)d->B * count);
  idx.resize((size_t)d->B * count);
  if (count <= 0) return KURA_OK;
  TCU(cudaMemcpy2DAsync(r.data(), w, d->out_r, pitch, w, d->B, cudaMemcpyDeviceToHost, d->st));
  TCU(cudaMemcpy2DAsync(idx.data(), w, d->out_idx, pitch, w, d->B, cudaMemcpyDeviceToHost, d->st));
  TCU(cudaStreamSynchronize(d->st));
  return KURA_OK;
}

int TensorEngine::get_state(int b, int rot_y, float* theta) {
  Impl& I = *d;
  const size_t off = ((size_t)rot_y * I.bp + b) * I.np;
  float* tmp = I.fin_theta + (size_t)b * I.np;
  TCU(launch_unwrap(I.ph_hi + off, I.ph_lo + off, I.ph_w + off, I.n, tmp, I.st));
  TCU(cudaMemcpyAsync(theta, tmp, sizeof(float) * I.n, cudaMemcpyDeviceToHost, I.st));
  TCU(cudaStreamSynchronize(I.st));
  return KURA_OK;
}

// mode 1: end-of-run record (theta at the last output time, couplings); mode 2: RHS
int TensorEngine::evaluate(int mode, int b, float* theta_out, float* coup_out) {
  Impl& I = *d;
  k_t_coef_final<<<1, 128, 0, I.st>>>(I.traj, I.src + 7 * (size_t)I.bp, I.B, I.t_eval, I.n_eval, mode == 1);
  TCU(cudaGetLastError());
  TCU(coupling(I, I.src + 7 * (size_t)I.bp, mode, I.fin_theta, nullptr));
  TCU(cudaStreamSynchronize(I.st));
  std::vector<float> tmp(2 * (size_t)I.n);
  if (theta_out)
    TCU(cudaMemcpy(theta_out, I.fin_theta + (size_t)b * I.np, sizeof(float) * I.n, cudaMemcpyDeviceToHost));
  if (coup_out)
    TCU(cudaMemcpy(coup_out, I.fin_coup + (size_t)b * I.np * 2, sizeof(float) * 2 * I.n, cudaMemcpyDeviceToHost));
  int errv = 0;
  TCU(cudaMemcpy(&errv, I.err, sizeof(int), cudaMemcpyDeviceToHost));
  if (errv) { g_terr = "tensor GEMM aborted (wait time limit)"; return KURA_ERR_BARRIER_TIMEOUT; }
  return KURA_OK;
}

int TensorEngine::sync_traj(std::vector<TrajG>& traj, bool to_device) {
  Impl& I = *d;
  // on the engine's stream: the legacy-stream cudaMemcpy does not order with it
  if (to_device)
    TCU(cudaMemcpyAsync(I.traj, traj.data(), sizeof(TrajG) * I.B, cudaMemcpyHostToDevice, I.st));
  else
    TCU(cudaMemcpyAsync(traj.data(), I.traj, sizeof(TrajG) * I.B, cudaMemcpyDeviceToHost, I.st));
  TCU(cudaStreamSynchronize(I.st));
  return KURA_OK;
}

}  // namespace kura
