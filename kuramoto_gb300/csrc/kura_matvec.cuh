// kura_matvec.cuh -- the stored-adjacency products of the integrator kernels: rows r0..r1 of A (float32,
// or N*A as int8) times the (cos, sin) of the stage phases, one pass over A for both sums (the
// reference reads A twice, with two GEMV calls, kuramoto.cu:110-115).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include "kura_kernels.cuh"

namespace kura {

// 16 bytes global -> shared without a register round trip (L2 only); src_bytes 0 zero-fills
__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gsrc, int src_bytes) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(gsrc), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ float mv_warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// ---------------------------------------------------------------- float32
// x is staged in shared memory one column tile at a time; each warp works on up to RG rows, each lane
// on 16-byte chunks of them.  A lane's 4 columns of x are 32 bytes from the next lane's, so back to
// back they would fall on four of the eight 16-byte bank groups; a stride of F_CHUNK = 6 (cos, sin)
// pairs (48 bytes) per 4 columns uses all eight.
//
// A streams through the warp's ring of A_STAGES * RG chunk slots with cp.async: every lane copies its
// own 16 bytes of each row, ST = A_STAGES * RG / NR column steps ahead, and reads back only what it
// copied, so the ring needs no barrier and holds no registers per byte in flight.  A warp with fewer
// rows (small N, the last pass) keeps as many bytes in flight with more steps.  The first chunks of a
// CTA's first tile are copied before the grid barrier that the other CTAs' x waits for
// (first_chunks); those of other tiles before the x tile has landed.  No part holds a barrier of its
// own, so warps with different NR run side by side between the block barriers of run().
template <int BMAX, int CTF>
struct MatvecF32 {
  static constexpr int RG = A_ROWS;
  static constexpr int CTFP = CTF / 4 * F_CHUNK;
  const float* adj;
  int ld, r0, r1, B;
  float2* xt;
  float4* ring;
  int tid, nt, lane, warp, mw;  // mw warps take part

  // the rows of this warp in the pass that starts at pr0: warp w takes rows pr0 + w + mw*q, so small
  // row blocks keep every warp busy; its nr rows in the CTA's block are q < nr
  __device__ __forceinline__ int pass_rows(int pr0, const float* (&src)[RG]) const {
    const int row0 = pr0 + warp;
#pragma unroll
    for (int q = 0; q < RG; ++q) {
      const int row = row0 + mw * q;
      src[q] = adj + (size_t)(row < r1 ? row : r0) * ld + lane * 4;
    }
    return r1 > row0 ? min(RG, (r1 - row0 + mw - 1) / mw) : 0;
  }
  // column steps of this lane in a tile of cw columns: cc = lane*4 + 128*it < cw
  __device__ __forceinline__ int lane_steps(int cw) const { return (cw - lane * 4 + 127) >> 7; }
  __device__ __forceinline__ float4* my_ring() const { return ring + (size_t)warp * (A_STAGES * RG * 32) + lane; }

  template <int NR>
  __device__ __forceinline__ void prologue(float4* my, const float* const (&src)[RG], int c0, int nit) const {
    constexpr int ST = A_STAGES * RG / NR;
    static_assert(ST * NR <= A_STAGES * RG, "ring slots");
#pragma unroll
    for (int s = 0; s < ST - 1; ++s) {
      if (s < nit)
#pragma unroll
        for (int q = 0; q < NR; ++q) cp_async16(my + (s * NR + q) * 32, src[q] + c0 + 128 * s, 16);
      cp_async_commit();
    }
  }
  __device__ __forceinline__ void prologue_of(int nr, float4* my, const float* const (&src)[RG], int c0, int nit) const {
    if (nr == 4) prologue<4>(my, src, c0, nit);
    else if (nr == 3) prologue<3>(my, src, c0, nit);
    else if (nr == 2) prologue<2>(my, src, c0, nit);
    else if (nr == 1) prologue<1>(my, src, c0, nit);
  }
  __device__ __forceinline__ void first_chunks() const {
    const float* src[RG];
    const int nr = pass_rows(r0, src);
    prologue_of(nr, my_ring(), src, 0, lane_steps(min(CTF, ld)));
  }
  // one x tile for the NR rows this warp holds
  template <int NR>
  __device__ __forceinline__ void steps(float4* my, const float* const (&src)[RG], int c0, int nit,
                                        float (&acc)[RG][BMAX][2]) const {
    constexpr int ST = A_STAGES * RG / NR;
    for (int it = 0; it < nit; ++it) {
      const int ahead = it + ST - 1;
      if (ahead < nit) {
        const int sl = ahead % ST;
#pragma unroll
        for (int q = 0; q < NR; ++q) cp_async16(my + (sl * NR + q) * 32, src[q] + c0 + 128 * ahead, 16);
      }
      cp_async_commit();
      cp_async_wait<ST - 1>();  // the chunks of step it have landed
      const int sl = it % ST;
      float4 a[NR];
#pragma unroll
      for (int q = 0; q < NR; ++q) a[q] = my[(sl * NR + q) * 32];
      const int cc = lane * 4 + 128 * it;
#pragma unroll
      for (int b = 0; b < BMAX; ++b) {
        if (b < B) {
          const float4* xp = reinterpret_cast<const float4*>(xt + b * CTFP + (cc >> 2) * F_CHUNK);
          float4 x01 = xp[0], x23 = xp[1];  // (c0,s0,c1,s1), (c2,s2,c3,s3)
#pragma unroll
          for (int q = 0; q < NR; ++q) {
            acc[q][b][0] += a[q].x * x01.x + a[q].y * x01.z + a[q].z * x23.x + a[q].w * x23.z;
            acc[q][b][1] += a[q].x * x01.y + a[q].y * x01.w + a[q].z * x23.y + a[q].w * x23.w;
          }
        }
      }
    }
    cp_async_wait<0>();
  }
  // The same where the prologue has brought the whole of the rows (N up to 1408 with one row per warp):
  // no copies and no waits, so that the reads of several steps overlap (340 clocks a step otherwise,
  // most of it latency: 1.4 of the 5 us of a RHS at N = 997)
  template <int NR>
  __device__ __forceinline__ void landed(const float4* my, int nit, float (&acc)[RG][BMAX][2]) const {
#pragma unroll 4
    for (int it = 0; it < nit; ++it) {
      const float4* xp = reinterpret_cast<const float4*>(xt + (lane + 32 * it) * F_CHUNK);
      const float4 x01 = xp[0], x23 = xp[1];
#pragma unroll
      for (int q = 0; q < NR; ++q) {
        const float4 a = my[(it * NR + q) * 32];
        acc[q][0][0] += a.x * x01.x + a.y * x01.z + a.z * x23.x + a.w * x23.z;
        acc[q][0][1] += a.x * x01.y + a.y * x01.w + a.z * x23.y + a.w * x23.w;
      }
    }
  }
  // The product with x (the CTAs' (cos, sin) of trajectory b at x + b*ld), after first_chunks() and the
  // barrier.  done(b, row, Fc, Fs, own (cos, sin)) is called by one lane for each row and trajectory.
  template <class Done>
  __device__ __forceinline__ void run(const float2* x, Done done) const {
    float4* my = my_ring();
    for (int pr0 = r0; pr0 < r1; pr0 += mw * RG) {
      float acc[RG][BMAX][2];
#pragma unroll
      for (int q = 0; q < RG; ++q)
#pragma unroll
        for (int b = 0; b < BMAX; ++b) acc[q][b][0] = acc[q][b][1] = 0.f;
      const float* src[RG];
      const int row0 = pr0 + warp, nr = pass_rows(pr0, src);
      int c0 = 0;
      for (; c0 < ld; c0 += CTF) {
        const bool first = pr0 == r0 && c0 == 0;  // its prologue has run
        if (!first) __syncthreads();              // the previous tile's readers are done
        const int cw = min(CTF, ld - c0);         // a multiple of 32
        // the x tile, 16 bytes (two columns) per copy
        for (int b = 0; b < B; ++b)
          for (int c = 2 * tid; c < cw; c += 2 * nt)
            cp_async16(xt + b * CTFP + (c >> 2) * F_CHUNK + (c & 3), x + (size_t)b * ld + c0 + c, 16);
        cp_async_commit();
        const int nit = lane_steps(cw);
        if (!first) prologue_of(nr, my, src, c0, nit);
        // this thread's copies of the x tile have landed (a first tile's ring was issued before it)
        if (first || nr == 0) cp_async_wait<0>();
        else if (nr == 4) cp_async_wait<A_STAGES - 1>();
        else if (nr == 3) cp_async_wait<A_STAGES * RG / 3 - 1>();
        else if (nr == 2) cp_async_wait<A_STAGES * RG / 2 - 1>();
        else cp_async_wait<A_STAGES * RG - 1>();
        __syncthreads();  // every thread's part has
        constexpr int ALL = A_STAGES * RG;  // ring slots: ALL / nr - 1 steps are on their way before a first tile
        if (BMAX == 1 && first && nr == 1 && cw <= 128 * (ALL - 1)) landed<1>(my, nit, acc);
        else if (BMAX == 1 && first && nr == 2 && cw <= 128 * (ALL / 2 - 1)) landed<2>(my, nit, acc);
        else if (nr == 4) steps<4>(my, src, c0, nit, acc);
        else if (nr == 3) steps<3>(my, src, c0, nit, acc);
        else if (nr == 2) steps<2>(my, src, c0, nit, acc);
        else if (nr == 1) steps<1>(my, src, c0, nit, acc);
      }
      const int xt_c0 = c0 - CTF;  // first column of the tile still staged
#pragma unroll
      for (int q = 0; q < RG; ++q)
        if (q < nr)
#pragma unroll
          for (int b = 0; b < BMAX; ++b) {
            acc[q][b][0] = mv_warp_sum(acc[q][b][0]);
            acc[q][b][1] = mv_warp_sum(acc[q][b][1]);
          }
      // lane q*BMAX+b finishes row row0+q of trajectory b; its own (cos, sin) come from the
      // staged tile when the last tile holds the row
#pragma unroll
      for (int q = 0; q < RG; ++q)
#pragma unroll
        for (int b = 0; b < BMAX; ++b) {
          const int row = row0 + mw * q;
          if (lane == q * BMAX + b && b < B && row < r1) {
            const int c = row - xt_c0;
            const float2 own = c >= 0 ? xt[b * CTFP + (c >> 2) * F_CHUNK + (c & 3)] : __ldcg(x + (size_t)b * ld + row);
            done(b, row, acc[q][b][0], acc[q][b][1], own);
          }
        }
    }
  }
};

// ---------------------------------------------------------------- int8, one trajectory
// Packed FP32 pairs (sm_100 and later): one instruction, each half rounded as the scalar
// operation.  (a.lo*b.lo + c.lo, a.hi*b.hi + c.hi):
__device__ __forceinline__ unsigned long long ffma2(unsigned long long a, unsigned long long b,
                                                    unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ float2 unpack_f2(unsigned long long v) {
  float2 r;
  asm("mov.b64 {%0,%1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
// byte j of w0 and of w1 (biased by 0x80) as the exact float pair (lo: w0, hi: w1): both placed under
// the exponent of 2^23 (0x4B000000), then 2^23 + 128 subtracted from the pair in one packed add
__device__ __forceinline__ unsigned long long i8_pair_to_f2(uint32_t w0, uint32_t w1, int j) {
  const uint32_t lo = __byte_perm(w0, 0x4B000000u, 0x7540u + (unsigned)j);
  const uint32_t hi = __byte_perm(w1, 0x4B000000u, 0x7540u + (unsigned)j);
  const unsigned long long bias = 0xCB000080CB000080ull;  // (-8388736.0f, -8388736.0f)
  unsigned long long d;
  asm("{\n\t.reg .b64 t;\n\tmov.b64 t, {%1,%2};\n\tadd.rn.f32x2 %0, t, %3;\n\t}"
      : "=l"(d) : "r"(lo), "r"(hi), "l"(bias));
  return d;
}

// The same product with A stored as the integers N*A (int8, exact for the reference's volcano rule,
// K <= 127): a quarter of the bytes.  Each lane streams 16 columns of 8 rows per load; the bytes of
// two rows at a time become a packed float pair that one packed FMA multiplies by a column's
// (cos, cos) and another by (sin, sin): 2.5 instructions per byte instead of 4.  (16 rows of 8
// columns halves the shared-memory reads of x but measured 2x slower at N=65536: half the bytes in
// flight per load.)  The x tile holds per column the float4 (cos, cos, sin, sin); a lane's 16 columns
// start I8_CHUNK4 = 17 float4 (272 bytes) after the previous lane's, which puts the 8 lanes of each
// phase of a 16-byte shared-memory read on distinct banks.
struct MatvecI8 {
  static constexpr int CTX = CT_I8;  // columns per x tile
  static constexpr int RG = 8;
  const int8_t* adj8;
  float invn;
  int ld8, r0, r1;
  float4* xt4;
  uint4* ring;
  int tid, nt, lane, warp, mw;

  // The columns [c0, c0 + cw) of the staged tile for the first RGT of the pass's RG rows of this warp
  // (rows row0 + mw*q), 16 int8 columns per lane and step; rows 2qp and 2qp+1 share the packed
  // accumulators acc[qp].  A streams through the warp's ring of I8_SLOTS chunk slots (16 bytes per
  // lane) with cp.async, I8_SLOTS / RGT steps deep, so the loads of the next step are in flight during
  // this step's conversion and FMAs.  No barrier inside: warps with different RGT run side by side
  // between the tile barriers of run().
  template <int RGT>
  __device__ __forceinline__ void tile(unsigned long long (&acc)[RG / 2][2], int row0, int c0, int cw) const {
    static_assert(RGT % 2 == 0 && RGT <= RG && I8_SLOTS % RGT == 0, "rows are taken in pairs");
    constexpr int ST = I8_SLOTS / RGT;
    uint4* my = ring + (size_t)warp * (I8_SLOTS * 32) + lane;
    const int8_t* src[RGT];
    int nb[RGT];
#pragma unroll
    for (int q = 0; q < RGT; ++q) {
      const int row = row0 + mw * q;
      nb[q] = row < r1 ? 16 : 0;  // rows past the CTA's block are zero-filled
      src[q] = adj8 + (size_t)(row < r1 ? row : r0) * ld8 + c0 + lane * 16;
    }
    // steps of this lane: columns cc = lane*16 + 512*it < cw (cw is a multiple of 16)
    const int nit = cw > lane * 16 ? (cw - lane * 16 + 511) >> 9 : 0;
#pragma unroll
    for (int s = 0; s < ST - 1; ++s) {
      if (s < nit)
#pragma unroll
        for (int q = 0; q < RGT; ++q) cp_async16(my + (s * RGT + q) * 32, src[q] + 512 * s, nb[q]);
      cp_async_commit();
    }
    for (int it = 0; it < nit; ++it) {
      const int ahead = it + ST - 1;
      if (ahead < nit) {
        const int sl = ahead % ST;
#pragma unroll
        for (int q = 0; q < RGT; ++q) cp_async16(my + (sl * RGT + q) * 32, src[q] + 512 * ahead, nb[q]);
      }
      cp_async_commit();
      cp_async_wait<ST - 1>();  // the chunks of step it have landed
      const int sl = it % ST;
      uint32_t a[RGT][4];
#pragma unroll
      for (int q = 0; q < RGT; ++q) {
        const uint4 v = my[(sl * RGT + q) * 32];
        a[q][0] = v.x ^ 0x80808080u;
        a[q][1] = v.y ^ 0x80808080u;
        a[q][2] = v.z ^ 0x80808080u;
        a[q][3] = v.w ^ 0x80808080u;
      }
      const int cc = lane * 16 + 512 * it;
#pragma unroll
      for (int wd = 0; wd < 4; ++wd) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          // ((cos, cos), (sin, sin)) of column cc + 4*wd + j
          const ulonglong2 xj = *reinterpret_cast<const ulonglong2*>(xt4 + (cc >> 4) * I8_CHUNK4 + 4 * wd + j);
#pragma unroll
          for (int qp = 0; qp < RGT / 2; ++qp) {
            const unsigned long long kp = i8_pair_to_f2(a[2 * qp][wd], a[2 * qp + 1][wd], j);
            acc[qp][0] = ffma2(kp, xj.x, acc[qp][0]);
            acc[qp][1] = ffma2(kp, xj.y, acc[qp][1]);
          }
        }
      }
    }
    cp_async_wait<0>();
  }
  // done(row, Fc, Fs, own (cos, sin)) is called by one lane for each row
  template <class Done>
  __device__ __forceinline__ void run(const float2* x, Done done) const {
    for (int pr0 = r0; pr0 < r1; pr0 += mw * RG) {
      // [qp][0]: (sum k cos) of rows (2qp, 2qp+1); [qp][1]: the same for sin
      unsigned long long acc[RG / 2][2];
#pragma unroll
      for (int q = 0; q < RG / 2; ++q) acc[q][0] = acc[q][1] = 0ull;
      const int row0 = pr0 + warp;
      const int nr = r1 > row0 ? min(RG, (r1 - row0 + mw - 1) / mw) : 0;
      int c0 = 0;
      for (; c0 < ld8; c0 += CTX) {
        __syncthreads();
        const int cw = min(CTX, ld8 - c0);  // a multiple of 16
        for (int c = tid; c < cw; c += nt) {
          const float2 v = __ldcg(x + c0 + c);
          xt4[(c >> 4) * I8_CHUNK4 + (c & 15)] = make_float4(v.x, v.x, v.y, v.y);
        }
        __syncthreads();
        // a warp with at most 4 rows in the pass (small N, the last pass) converts no bytes of
        // the absent ones
        if (nr <= 4) tile<4>(acc, row0, c0, cw);
        else tile<RG>(acc, row0, c0, cw);
      }
      float accf[RG][2];
#pragma unroll
      for (int qp = 0; qp < RG / 2; ++qp)
#pragma unroll
        for (int v = 0; v < 2; ++v) {
          const float2 u = unpack_f2(acc[qp][v]);
          accf[2 * qp][v] = mv_warp_sum(u.x);
          accf[2 * qp + 1][v] = mv_warp_sum(u.y);
        }
      // the row's own (cos, sin) from the staged tile when the last tile holds it
      const int xt_c0 = c0 - CTX;
#pragma unroll
      for (int q = 0; q < RG; ++q) {
        const int row = row0 + mw * q;
        if (lane == q && row < r1) {
          const int c = row - xt_c0;
          float2 own;
          if (c >= 0) {
            const float4 v = xt4[(c >> 4) * I8_CHUNK4 + (c & 15)];
            own = make_float2(v.x, v.z);
          } else {
            own = __ldcg(x + row);
          }
          done(row, accf[q][0] * invn, accf[q][1] * invn, own);
        }
      }
    }
  }
};

// ---------------------------------------------------------------- int8 on the integer tensor pipe
// The int8 product of a large network as integers: x = X 2^-30 with X = round(x 2^30) in four signed
// base-256 digits, so the 8 digits of (cos, sin) are the 8 columns of mma.m16n8k32.s8 and one
// instruction multiplies 512 bytes of A.  The sums are exact (|sum| <= 127 128 n < 2^31 for
// n <= 132000); the product's only errors are the 2^-31 of X and the final rounding.  The byte
// conversions and packed FMAs of MatvecI8 cost 20 issue slots per 8 bytes and lane and held A at 4.1
// to 5.1 TB/s (N = 40009, 65536); here 512 bytes take 16 clocks of an SM's integer pipe (measured) of
// the 23 that HBM needs to deliver them, and A arrives at 5.6 / 6.0 / 6.8 TB/s at N = 16384 / 40009 /
// 65536.
//
// Work: a pass holds up to 8 tiles of 16 rows; the warps split the columns, warp w takes the 64-column
// chunks w, w + 16, .. and all rows of the pass, so that any number of rows keeps all warps busy and a
// chunk of x is read once per pass.  K order: in a chunk, lane (g, t) = (lane / 4, lane % 4) holds
// columns 16 t .. 16 t + 15 of rows g and g + 8 and of digit plane g, 16 bytes each; the words 0, 1 and
// 2, 3 of A and x meet in one MMA each.  A streams through the warp's ring of IM_SLOTS units (one row
// tile of a chunk, 32 bytes per lane), across chunks and x tiles; x arrives in two tiles of IM_TC
// columns, one ahead.  The warps' sums meet in shared memory by integer atomics.
constexpr int IM_TC = 4096;           // columns per x tile
constexpr int IM_XS = IM_TC + 64;     // bytes per digit plane of a tile: a phase's two planes on distinct banks
constexpr int IM_SLOTS = 8;           // units in a warp's ring
constexpr int IM_MT = 8;              // row tiles per pass
constexpr int IM_SMEM_X = 2 * 8 * IM_XS;
constexpr int IM_SMEM_ACC = IM_MT * 16 * 8 * 4;

// the four signed base-256 digits of round(x 2^30), lowest first, |x| <= 1
__device__ __forceinline__ uint32_t x_digits(float x) {
  const int X = __float2int_rn(x * 1073741824.f);
  return ((uint32_t)X + 0x00808080u) ^ 0x00808080u;
}

struct MatvecImma {
  const int8_t* adj8;
  float invn;
  int ld8, r0, r1;
  int xld;     // bytes per digit plane of x
  int8_t* xt;  // [2][8][IM_XS]
  int* sums;   // [IM_MT * 16][8]
  uint4* ring;
  int tid, nt, lane, warp, nw;

  // the digits of tile `t` of x into buffer t & 1
  __device__ __forceinline__ void load_x(const int8_t* x, int t) const {
    int8_t* dst = xt + (t & 1) * 8 * IM_XS;
    const int c0 = t * IM_TC;
    for (int i = tid; i < 8 * IM_TC / 16; i += nt) {
      const int pl = i / (IM_TC / 16), c = i % (IM_TC / 16) * 16;
      const bool in = c0 + c < xld;
      cp_async16(dst + pl * IM_XS + c, x + (size_t)pl * xld + (in ? c0 + c : 0), in ? 16 : 0);
    }
  }
  // rows row0 .. row0 + 16 MT: sums[row][digit]
  template <int MT>
  __device__ __forceinline__ void pass(const int8_t* x, int row0) const {
    const int g = lane >> 2, t = lane & 3;
    int acc[MT][4];
#pragma unroll
    for (int m = 0; m < MT; ++m) acc[m][0] = acc[m][1] = acc[m][2] = acc[m][3] = 0;
    uint4* my = ring + (size_t)warp * (IM_SLOTS * 64) + lane;
    const int nch = (ld8 + 63) / 64;  // chunks
    const int mine = warp < nch ? (nch - warp + nw - 1) / nw : 0, units = mine * MT;
    // unit u: chunk u / MT of this warp, row tile u % MT
    int lc = 64 * warp + 16 * t, lm = 0, lu = 0;  // the next unit to load
    auto load = [&]() {
      if (lu < units) {
        const int ra = row0 + 16 * lm + g, rb = ra + 8;
        const bool in = lc < ld8;
        uint4* s = my + (lu % IM_SLOTS) * 64;
        cp_async16(s, adj8 + (size_t)(ra < r1 ? ra : r0) * ld8 + (in ? lc : 0), in && ra < r1 ? 16 : 0);
        cp_async16(s + 32, adj8 + (size_t)(rb < r1 ? rb : r0) * ld8 + (in ? lc : 0), in && rb < r1 ? 16 : 0);
        if (++lm == MT) {
          lm = 0;
          lc += 64 * nw;
        }
        ++lu;
      }
      cp_async_commit();
    };
    const int tiles = (ld8 + IM_TC - 1) / IM_TC;
    load_x(x, 0);
    cp_async_commit();
#pragma unroll 1
    for (int s = 0; s < IM_SLOTS - 1; ++s) load();
    int u = 0;
#pragma unroll 1
    for (int tl = 0; tl < tiles; ++tl) {
      // this tile of x has landed: the first was committed before the ring's units, a later one with
      // the first unit of the tile before, IM_SLOTS units or more ago where that had so many
      if (tl > 0 && MT * (IM_TC / 64 / 16) < IM_SLOTS) cp_async_wait<0>();
      else cp_async_wait<IM_SLOTS - 1>();
      __syncthreads();  // every thread's part of it, and the tile before is no longer read
      if (tl + 1 < tiles) load_x(x, tl + 1);
      const int8_t* xb = xt + (tl & 1) * 8 * IM_XS + g * IM_XS + 16 * t;
      const int cend = min(nch, (tl + 1) * (IM_TC / 64));
#pragma unroll 1
      for (int c = warp + (u / MT) * nw; c < cend; c += nw) {
        const uint4 b = *reinterpret_cast<const uint4*>(xb + (c * 64 - tl * IM_TC));
#pragma unroll
        for (int m = 0; m < MT; ++m, ++u) {
          load();
          cp_async_wait<IM_SLOTS - 1>();  // unit u has landed
          const uint4* s = my + (u % IM_SLOTS) * 64;
          const uint4 a = s[0], h = s[32];
          asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                       : "+r"(acc[m][0]), "+r"(acc[m][1]), "+r"(acc[m][2]), "+r"(acc[m][3])
                       : "r"(a.x), "r"(h.x), "r"(a.y), "r"(h.y), "r"(b.x), "r"(b.y));
          asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                       : "+r"(acc[m][0]), "+r"(acc[m][1]), "+r"(acc[m][2]), "+r"(acc[m][3])
                       : "r"(a.z), "r"(h.z), "r"(a.w), "r"(h.w), "r"(b.z), "r"(b.w));
        }
      }
    }
    cp_async_wait<0>();
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      int* d = sums + (16 * m + g) * 8 + 2 * t;
      atomicAdd(d, acc[m][0]);
      atomicAdd(d + 1, acc[m][1]);
      atomicAdd(d + 64, acc[m][2]);
      atomicAdd(d + 65, acc[m][3]);
    }
  }
  // x: [8][xld] digit planes.  done(row, Fc, Fs) is called by one thread for each row.
  template <class Done>
  __device__ __forceinline__ void run(const int8_t* x, Done done) const {
    int left = (r1 - r0 + 15) / 16;
    for (int row0 = r0; left > 0;) {
      const int passes = (left + IM_MT - 1) / IM_MT, mt = (left + passes - 1) / passes;  // passes of even height
      for (int i = tid; i < mt * 16 * 8; i += nt) sums[i] = 0;
      __syncthreads();
      switch (mt) {
        case 1: pass<1>(x, row0); break;
        case 2: pass<2>(x, row0); break;
        case 3: pass<3>(x, row0); break;
        case 4: pass<4>(x, row0); break;
        case 5: pass<5>(x, row0); break;
        case 6: pass<6>(x, row0); break;
        case 7: pass<7>(x, row0); break;
        default: pass<8>(x, row0); break;
      }
      __syncthreads();
      for (int r = tid; r < mt * 16 && row0 + r < r1; r += nt) {
        const int* d = sums + r * 8;
        const long long c = 16777216ll * d[3] + 65536ll * d[2] + 256ll * d[1] + d[0];
        const long long s = 16777216ll * d[7] + 65536ll * d[6] + 256ll * d[5] + d[4];
        constexpr float S = 1.f / 1073741824.f;
        done(row0 + r, __ll2float_rn(c) * S * invn, __ll2float_rn(s) * S * invn);
      }
      __syncthreads();  // before the sums and the x tiles are written again
      row0 += 16 * mt;
      left -= mt;
    }
  }
};

}  // namespace kura
