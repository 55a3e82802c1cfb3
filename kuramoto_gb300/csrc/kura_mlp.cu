// kura_mlp.cu -- the order-parameter surrogate: a 4-layer MLP (SiLU, BF16 weights, FP32
// accumulation) trained and evaluated on the GPU by this library's own kernels.
//
// The reference has no learned component.  This network maps features of a Kuramoto run
// (coupling, rank, frequency scale and family, the first samples of r(t)) to the steady
// mean and spread of r, and places coupling-sweep points near the volcano transition.
//
// Every GEMM of the forward and the backward pass runs on tcgen05 through k_tensor_gemm
// (TMA-fed shared memory, FP32 accumulation in TMEM) with its own fused epilogue:
//   forward  Z_l = H_l W_l^T + b_l       A = H_l [B][in], X = W_l [out][in]
//            H_{l+1} = silu(Z_l) (BF16, plus its transpose) and silu'(Z_l) kept for backward
//   weights  dW_l = dZ_l^T H_l            A = dZ_l^T [out][B], X = H_l^T [in][B]
//   inputs   dZ_{l-1} = (dZ_l W_l) * silu'(Z_{l-1})   A = dZ_l [B][out], X = W_l^T [in][out]
// Widths are padded to multiples of 64 (the K tile) with zero weights, which stay zero:
// their gradients vanish.  Adam updates FP32 master weights and rewrites the BF16 copies;
// one whole training step (forward, loss, backward, Adam, gathering the next rows) is a CUDA graph
// replayed once per step, with the step counter on the device.  A step is a chain of nine kernels,
// each of some microseconds of latency: what can leave the chain (loss, weight gradients, the next
// rows) runs beside it, and a GEMM's setup overlaps the end of the kernel before it.  For 512 rows
// and 256 hidden units a step takes 49 us (313 us with one kernel for each piece, one after another).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>
#include "kura.h"
#include "kura_kernels.cuh"
#include "kura_tensor_gemm.cuh"

namespace kura {
namespace {

constexpr int NL = 4;    // linear layers
constexpr int PADW = 64;  // widths padded to the K tile
typedef __nv_bfloat16 bf16;

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&v);
}

// Every GEMM of the network is cut into column blocks of MLP_NC columns beside the 128-row tiles,
// one CTA each.  What bounds these GEMMs (512 x 256 x 256) is the epilogue's chain of TMEM reads,
// expf and stores, 16 columns at a time, not the 0.07 us of tensor work: with one block of 256
// columns a hidden layer took 33 us on 4 of the 152 SMs, with 32-column blocks on 32 SMs 9 us.
// 16 is the narrowest that the MMA takes: a training step went from 65 to 59 us, a forward pass of
// 64 rows from 55 to 48.  The K loop of a column is the same in every form, and so are the results,
// bit for bit.
constexpr int MLP_NC = 16;  // the epilogues below read that many columns at once

// ---------------------------------------------------------------- GEMM epilogues
// forward: z = acc + b; hidden layers store silu(z) (row-major and transposed, BF16) and
// silu'(z); the last layer stores the real outputs of z, packed [Bt][out_dim], and for training the
// gradient of the mean squared error, 2 (y - t) / (n out_dim), in both layouts (rows from nvalid on
// are zero; the padding columns of dZ and dZT were zeroed with the buffers and stay zero)
struct FwdEpi {
  static constexpr __device__ bool f16() { return false; }
  const float* bias;
  int last, Bt, ld, out_dim;
  bf16* H;   // [Bt][ld]
  bf16* HT;  // [ld][Bt]
  float* S;  // [Bt][ld]
  float* Y;  // [Bt][out_dim]
  const float* T;  // [Bt][out_dim], or null: no gradient
  int nvalid;
  float scale;  // 2 / (nvalid out_dim)
  bf16* dZ;     // [Bt][ld]
  bf16* dZT;    // [ld][Bt]
  __device__ void row(uint32_t taddr, int row, int m0, int sp) {
    const int r = m0 + row;
    const int c0 = sp * MLP_NC;
    float a[16];
    umma::tmem_ld16(taddr, a);
    umma::tmem_ld_wait();
    float z[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) z[j] = a[j] + bias[c0 + j];
    if (last) {
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        if (c0 + j >= out_dim) break;
        Y[(size_t)r * out_dim + c0 + j] = z[j];
        if (T) {
          const float e = z[j] - T[(size_t)r * out_dim + c0 + j];
          const bf16 b = __float2bfloat16_rn(r < nvalid ? scale * e : 0.f);
          dZ[(size_t)r * ld + c0 + j] = b;
          dZT[(size_t)(c0 + j) * Bt + r] = b;
        }
      }
      return;
    }
    float h[16], d[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const float s = 1.f / (1.f + expf(-z[j]));
      h[j] = z[j] * s;
      d[j] = s * (1.f + z[j] * (1.f - s));
    }
    uint4* hp = reinterpret_cast<uint4*>(H + (size_t)r * ld + c0);
    hp[0] = make_uint4(pack_bf16(h[0], h[1]), pack_bf16(h[2], h[3]), pack_bf16(h[4], h[5]), pack_bf16(h[6], h[7]));
    hp[1] = make_uint4(pack_bf16(h[8], h[9]), pack_bf16(h[10], h[11]), pack_bf16(h[12], h[13]),
                       pack_bf16(h[14], h[15]));
#pragma unroll
    for (int j = 0; j < 16; ++j) HT[(size_t)(c0 + j) * Bt + r] = __float2bfloat16_rn(h[j]);
    float4* dp = reinterpret_cast<float4*>(S + (size_t)r * ld + c0);
#pragma unroll
    for (int q = 0; q < 4; ++q) dp[q] = make_float4(d[4 * q], d[4 * q + 1], d[4 * q + 2], d[4 * q + 3]);
  }
};

// weight gradient: rows are output units; rows beyond the padded width are not stored
struct DwEpi {
  static constexpr __device__ bool f16() { return false; }
  float* G;  // [out_p][ld]
  int out_p, ld;
  __device__ void row(uint32_t taddr, int row, int m0, int sp) {
    const int r = m0 + row;
    float a[16];
    umma::tmem_ld16(taddr, a);
    umma::tmem_ld_wait();
    if (r >= out_p) return;
    float4* g = reinterpret_cast<float4*>(G + (size_t)r * ld + sp * MLP_NC);
#pragma unroll
    for (int q = 0; q < 4; ++q) g[q] = make_float4(a[4 * q], a[4 * q + 1], a[4 * q + 2], a[4 * q + 3]);
  }
};

// input gradient of a hidden layer: dZ_{l-1} = (dZ_l W_l) * silu'(Z_{l-1}), BF16, both layouts
struct DhEpi {
  static constexpr __device__ bool f16() { return false; }
  const float* S;  // [Bt][ld]
  bf16* dZ;        // [Bt][ld]
  bf16* dZT;       // [ld][Bt]
  int Bt, ld;
  __device__ void row(uint32_t taddr, int row, int m0, int sp) {
    const int r = m0 + row;
    const int c0 = sp * MLP_NC;
    float a[16];
    umma::tmem_ld16(taddr, a);
    umma::tmem_ld_wait();
    const float4* sp4 = reinterpret_cast<const float4*>(S + (size_t)r * ld + c0);
    float d[16];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float4 s = sp4[q];
      d[4 * q] = a[4 * q] * s.x;
      d[4 * q + 1] = a[4 * q + 1] * s.y;
      d[4 * q + 2] = a[4 * q + 2] * s.z;
      d[4 * q + 3] = a[4 * q + 3] * s.w;
    }
    uint4* dp = reinterpret_cast<uint4*>(dZ + (size_t)r * ld + c0);
    dp[0] = make_uint4(pack_bf16(d[0], d[1]), pack_bf16(d[2], d[3]), pack_bf16(d[4], d[5]), pack_bf16(d[6], d[7]));
    dp[1] = make_uint4(pack_bf16(d[8], d[9]), pack_bf16(d[10], d[11]), pack_bf16(d[12], d[13]),
                       pack_bf16(d[14], d[15]));
#pragma unroll
    for (int j = 0; j < 16; ++j) dZT[(size_t)(c0 + j) * Bt + r] = __float2bfloat16_rn(d[j]);
  }
};

// ---------------------------------------------------------------- small kernels
// minibatch rows of the dataset (training) or of a caller's chunk (idx == null): BF16 input
// rows and their transpose, FP32 targets; rows >= nvalid are zero.  The padding columns past
// in_dim were zeroed with the buffers and are never written
struct GatherArgs {
  const float *X, *T;
  const int *idx, *counter;
  long long steps;  // with a counter: steps of the run, past which there is nothing to gather
  int in_dim, out_dim, Bt, nvalid;
  bf16 *H0, *HT0;
  float* Tb;
};
__device__ __forceinline__ void gather_rows(const GatherArgs& a, int block, int blocks) {
  const int step = a.counter ? *a.counter : 0;
  if (a.counter && step >= a.steps) return;
  const int total = a.Bt * max(a.in_dim, a.out_dim);
  for (int t = block * blockDim.x + threadIdx.x; t < total; t += blocks * blockDim.x) {
    const int c = t / a.Bt, r = t % a.Bt;  // c-major: the transposed store is coalesced
    long long src = -1;
    if (r < a.nvalid) src = a.idx ? (long long)a.idx[(long long)step * a.Bt + r] : (long long)r;
    if (c < a.in_dim) {
      const bf16 b = __float2bfloat16_rn(src >= 0 ? a.X[src * a.in_dim + c] : 0.f);
      a.HT0[(size_t)c * a.Bt + r] = b;
      a.H0[(size_t)r * PADW + c] = b;
    }
    if (a.T && c < a.out_dim) a.Tb[(size_t)r * a.out_dim + c] = src >= 0 ? a.T[src * a.out_dim + c] : 0.f;
  }
}
constexpr int GATHER_BLOCKS = 64;
__global__ void k_mlp_gather(const __grid_constant__ GatherArgs a) {
  pdl_launch();
  gather_rows(a, blockIdx.x, gridDim.x);
}

// mean squared error over the valid rows and the first out_dim outputs (its gradient is the last
// layer's epilogue's); beside the backward pass, on a stream of its own
__global__ void k_mlp_loss(const float* __restrict__ Y, const float* __restrict__ Tb, int nvalid, int out_dim, int Bt,
                           float* loss, int* counter) {
  __shared__ float red[32];
  float acc = 0.f;
  for (int t = threadIdx.x; t < Bt * out_dim; t += blockDim.x) {
    const int j = t / Bt, r = t % Bt;
    if (r < nvalid) {
      const float e = Y[(size_t)r * out_dim + j] - Tb[(size_t)r * out_dim + j];
      acc = fmaf(e, e, acc);
    }
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    float s = 0.f;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[w];
    const int step = counter ? *counter : 0;
    loss[step] = s / ((float)nvalid * (float)out_dim);
    if (counter) *counter = step + 1;  // the update that follows is step *counter - 1
  }
}

struct UpdLayer {
  long long w_off, b_off;
  int in_p, out_p, tiles, tiles_i;  // 32 x 32 weight tiles of the layer, and per row of tiles
  bf16* W;
  bf16* WT;
  const bf16* dZ;  // [Bt][out]
};
struct UpdArgs {
  UpdLayer l[NL];
};
struct AdamArgs {
  float *M, *V;
  const int* counter;
  float lr0, lr1;
  long long total_steps;
  float b1, b2, eps;
};
// the parameter after its step, from its gradient and its own state
struct AdamVal {
  float p, m, v;
  __device__ __forceinline__ void load(const float* P, const AdamArgs& a, long long i) {
    p = P[i];
    m = a.M[i];
    v = a.V[i];
  }
  __device__ __forceinline__ float step(float* P, const AdamArgs& a, long long i, float g, float lr, float c1, float c2) {
    // which product is rounded by itself is written out: training amplifies the last bit
    m = __fmaf_rn(1.f - a.b1, g, __fmul_rn(a.b1, m));
    v = __fmaf_rn(__fmul_rn(1.f - a.b2, g), g, __fmul_rn(a.b2, v));
    a.M[i] = m;
    a.V[i] = v;
    p = p - lr * (m / c1) / (sqrtf(v / c2) + a.eps);
    P[i] = p;
    return p;
  }
};
constexpr int UPD_THREADS = 256;
constexpr int UPD_BIAS = 32;    // output units per bias block
constexpr int UPD_ROWS = 128;   // rows of dZ staged per round of a bias block (the batch is a multiple)
// What follows a backward pass, in one launch: blocks of 32 x 32 weights and blocks of UPD_BIAS
// output units.  UPD_ADAM: the Adam step (Kingma & Ba; learning rate interpolated linearly from
// lr0 to lr1 over the run, the step number from the device counter).  UPD_PACK: the BF16 copies of
// the weights, [out][in] and, through a shared-memory tile, [in][out].  UPD_BIAS_GRAD: the bias
// gradients, summed in the order of the rows by one thread per unit, over a tile of rows that the
// whole block has brought into shared memory (the additions of a tile take 0.3 us; a thread that
// loads its own rows waits for memory between them).  UPD_GATHER: further blocks bring the rows of
// the next step, whose launch would be 4.5 us more of the step's chain.  These are 1.3 MB of reads
// and writes, bound by launch latency and the depth of each chain: as an Adam launch, a pack launch
// and a sum by one thread per unit and layer they took 9 + 6.5 + 4 x 30 us per training step,
// together 9.7 us, and 7.8 us since a thread's loads all precede its stores.
enum { UPD_ADAM = 1, UPD_PACK = 2, UPD_BIAS_GRAD = 4, UPD_GATHER = 8 };
__global__ void __launch_bounds__(UPD_THREADS)
    k_mlp_update(float* P, float* G, const __grid_constant__ UpdArgs u, AdamArgs a,
                 const __grid_constant__ GatherArgs ga, int Bt, int what) {
  __shared__ bf16 tile[32][33];
  __shared__ bf16 stage[UPD_ROWS][32];
  int blk = blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  float lr = 0.f, c1 = 1.f, c2 = 1.f;
  if (what & UPD_ADAM) {
    const int step = *a.counter - 1;  // advanced by the loss kernel
    const float frac = a.total_steps > 1 ? (float)step / (float)(a.total_steps - 1) : 0.f;
    lr = a.lr0 + (a.lr1 - a.lr0) * frac;
    c1 = 1.f - powf(a.b1, (float)(step + 1));
    c2 = 1.f - powf(a.b2, (float)(step + 1));
  }
#pragma unroll 1
  for (int l = 0; l < NL; ++l) {
    const UpdLayer& L = u.l[l];
    if (blk < L.tiles) {
      const int o0 = blk / L.tiles_i * 32, i0 = blk % L.tiles_i * 32;
      // every load before the first store, which the compiler must take for one to the same place
      AdamVal val[4];
      float g[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const long long e = L.w_off + (long long)(o0 + warp + 8 * q) * L.in_p + i0 + lane;
        if (what & UPD_ADAM) {
          val[q].load(P, a, e);
          g[q] = G[e];
        } else {
          val[q].p = P[e];
        }
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int o = warp + 8 * q;
        const long long e = L.w_off + (long long)(o0 + o) * L.in_p + i0 + lane;
        const float p = (what & UPD_ADAM) ? val[q].step(P, a, e, g[q], lr, c1, c2) : val[q].p;
        if (what & UPD_PACK) {
          const bf16 b = __float2bfloat16_rn(p);
          L.W[(size_t)(o0 + o) * L.in_p + i0 + lane] = b;
          tile[o][lane] = b;
        }
      }
      if (what & UPD_PACK) {
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int i = warp + 8 * q;
          L.WT[(size_t)(i0 + i) * L.out_p + o0 + lane] = tile[lane][i];
        }
      }
      return;
    }
    blk -= L.tiles;
    const int nb = L.out_p / UPD_BIAS;
    if (blk < nb) {
      if (!(what & UPD_BIAS_GRAD)) return;
      const int o = blk * UPD_BIAS + lane;
      float s = 0.f;
      AdamVal val{};
      if ((what & UPD_ADAM) && warp == 0) val.load(P, a, L.b_off + o);
      const bf16* src = L.dZ + (size_t)warp * L.out_p + o;
      bf16 v[UPD_ROWS / 8];
      auto load = [&](int r0) {
#pragma unroll
        for (int q = 0; q < UPD_ROWS / 8; ++q) v[q] = src[(size_t)(r0 + 8 * q) * L.out_p];
      };
      load(0);
      for (int r0 = 0; r0 < Bt; r0 += UPD_ROWS) {
        __syncthreads();  // the previous tile has been summed
#pragma unroll
        for (int q = 0; q < UPD_ROWS / 8; ++q) stage[warp + 8 * q][lane] = v[q];
        __syncthreads();
        if (r0 + UPD_ROWS < Bt) load(r0 + UPD_ROWS);  // lands while this tile is summed
        if (warp == 0) {
#pragma unroll 32
          for (int q = 0; q < UPD_ROWS; ++q) s += __bfloat162float(stage[q][lane]);
        }
      }
      if (warp == 0) {
        G[L.b_off + o] = s;
        if (what & UPD_ADAM) val.step(P, a, L.b_off + o, s, lr, c1, c2);
      }
      return;
    }
    blk -= nb;
  }
  if (what & UPD_GATHER) gather_rows(ga, blk, GATHER_BLOCKS);
}
struct Layer {
  int in, out, in_p, out_p, out_m;  // out_m: rows of dZ^T (at least one 128-row M tile)
  long long w_off, b_off;
};

int round_up(int x, int m) { return (x + m - 1) / m * m; }

uint64_t splitmix64(uint64_t& s) {
  uint64_t z = (s += 0x9E3779B97F4A7C15ull);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
double uniform01(uint64_t& s) { return (double)(splitmix64(s) >> 11) * (1.0 / 9007199254740992.0); }

}  // namespace
}  // namespace kura

using kura::bf16;
using kura::Layer;
using kura::NL;
using kura::PADW;

struct kura_mlp {
  int device = 0, in_dim = 0, hidden = 0, out_dim = 0, Bt = 0, sms = 0;
  Layer L[NL];
  long long nparam = 0;  // padded flat size
  float *P = nullptr, *G = nullptr, *Mo = nullptr, *Vo = nullptr;
  bf16 *W[NL] = {}, *WT[NL] = {};
  bf16 *H[NL] = {}, *HT[NL] = {};  // input of layer l
  float* S[NL] = {};               // silu'(Z_{l-1}), the derivative at the input of layer l (l >= 1)
  float* Y = nullptr;
  bf16 *dZ[NL] = {}, *dZT[NL] = {};  // gradient at the output of layer l
  float *Tb = nullptr, *loss = nullptr, *Xin = nullptr, *Tin = nullptr;
  int *counter = nullptr, *err = nullptr;
  float* y_pin = nullptr;  // pinned: one chunk's outputs, then the error flag
  CUtensorMap fA[NL], fX[NL], wA[NL], wX[NL], hA[NL], hX[NL];
  // side: the loss and the weight gradients, beside the input gradients
  cudaStream_t st = nullptr, side[2] = {nullptr, nullptr};
  cudaEvent_t ev[2] = {nullptr, nullptr};
  cudaEvent_t evz[NL] = {}, evw[2] = {nullptr, nullptr};  // dZ of a layer is ready; a side stream is done
  std::vector<void*> allocs;
};

namespace {

int mlp_fail(int code, const std::string& msg) {
  kura::set_last_error(msg.c_str());
  return code;
}
#define MLPCU(x)                                                                                  \
  do {                                                                                            \
    cudaError_t e_ = (x);                                                                         \
    if (e_ != cudaSuccess)                                                                        \
      return mlp_fail(e_ == cudaErrorMemoryAllocation ? KURA_ERR_NOMEM : KURA_ERR_CUDA,           \
                      std::string(#x) + ": " + cudaGetErrorString(e_));                          \
  } while (0)

template <class T>
cudaError_t dalloc(kura_mlp* m, T** p, size_t count) {
  cudaError_t e = cudaMalloc((void**)p, sizeof(T) * std::max<size_t>(count, 1));
  if (e == cudaSuccess) {
    m->allocs.push_back(*p);
    e = cudaMemset(*p, 0, sizeof(T) * std::max<size_t>(count, 1));
    // the zero-fill runs on the legacy default stream, unordered with a non-blocking stream
    if (e == cudaSuccess) e = cudaStreamSynchronize(0);
  }
  return e;
}

constexpr unsigned long long GEMM_LIMIT_NS = 20000000000ull;

template <class Epi>
cudaError_t gemm(kura_mlp* m, cudaStream_t st, const CUtensorMap& a, const CUtensorMap& x, int mtiles, int width,
                 int ktiles, const Epi& e, bool overlap) {
  constexpr int NC = kura::MLP_NC;
  const int nsplit = width / NC;
  const dim3 grid((unsigned)std::min(mtiles * nsplit, m->sms));
  const auto k = kura::k_tensor_gemm<NC, Epi>;
  if (overlap)
    return kura::launch_pdl(k, grid, kura::TG_THREADS, kura::TGCfg<NC>::SMEM, st, 1, a, x, mtiles, mtiles, ktiles,
                            nsplit, NC, e, m->err, GEMM_LIMIT_NS, nullptr);
  k<<<grid, kura::TG_THREADS, kura::TGCfg<NC>::SMEM, st>>>(a, x, mtiles, mtiles, ktiles, nsplit, NC, e, m->err,
                                                           GEMM_LIMIT_NS, nullptr);
  return cudaGetLastError();
}
template <class Epi>
cudaError_t set_attr() {
  return cudaFuncSetAttribute(kura::k_tensor_gemm<kura::MLP_NC, Epi>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              kura::TGCfg<kura::MLP_NC>::SMEM);
}

// the first `rows` rows of the batch (rounded up to row tiles); `nvalid` > 0: with the gradient of
// the error over so many rows.  `overlap`: the kernel before the first layer lets it start early
cudaError_t forward(kura_mlp* m, int rows, int nvalid, bool overlap) {
  for (int l = 0; l < NL; ++l) {
    const Layer& L = m->L[l];
    const bool last = (l == NL - 1);
    kura::FwdEpi ep{m->P + L.b_off, last ? 1 : 0, m->Bt, L.out_p, L.out, last ? nullptr : m->H[l + 1],
                    last ? nullptr : m->HT[l + 1], last ? nullptr : m->S[l + 1], last ? m->Y : nullptr,
                    last && nvalid > 0 ? m->Tb : nullptr, nvalid, 2.f / ((float)nvalid * (float)L.out),
                    last ? m->dZ[l] : nullptr, last ? m->dZT[l] : nullptr};
    // of the last layer only the column blocks that hold real outputs
    const int width = last ? kura::round_up(L.out, kura::MLP_NC) : L.out_p;
    cudaError_t e = gemm(m, m->st, m->fA[l], m->fX[l], kura::round_up(rows, kura::TG_BM) / kura::TG_BM, width,
                         L.in_p / kura::TG_BK, ep, l > 0 || overlap);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// The input gradients follow one another; each layer's weight gradient needs only that layer's dZ
// and runs beside them, on the side streams in turn.  The loss needs only the outputs.
cudaError_t backward(kura_mlp* m, int nvalid, float* loss, int* counter) {
  cudaError_t e = cudaSuccess;
  for (int l = NL - 1; l >= 0 && e == cudaSuccess; --l) {
    const Layer& L = m->L[l];
    e = cudaEventRecord(m->evz[l], m->st);
    if (l == NL - 1) {
      cudaStream_t so = m->side[(l + 1) & 1];  // not the one that the first weight gradient takes
      if (e == cudaSuccess) e = cudaStreamWaitEvent(so, m->evz[l], 0);
      if (e == cudaSuccess) {
        kura::k_mlp_loss<<<1, 1024, 0, so>>>(m->Y, m->Tb, nvalid, m->out_dim, m->Bt, loss, counter);
        e = cudaGetLastError();
      }
    }
    cudaStream_t sw = m->side[l & 1];
    if (e == cudaSuccess) e = cudaStreamWaitEvent(sw, m->evz[l], 0);
    kura::DwEpi dw{m->G + L.w_off, L.out_p, L.in_p};
    if (e == cudaSuccess)
      e = gemm(m, sw, m->wA[l], m->wX[l], L.out_m / kura::TG_BM, L.in_p, m->Bt / kura::TG_BK, dw, false);
    if (l == 0 || e != cudaSuccess) break;
    kura::DhEpi dh{m->S[l], m->dZ[l - 1], m->dZT[l - 1], m->Bt, L.in_p};
    e = gemm(m, m->st, m->hA[l], m->hX[l], m->Bt / kura::TG_BM, L.in_p, L.out_p / kura::TG_BK, dh, true);
  }
  for (int q = 0; q < 2; ++q) {
    if (e == cudaSuccess) e = cudaEventRecord(m->evw[q], m->side[q]);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(m->st, m->evw[q], 0);
  }
  return e;
}

cudaError_t update(kura_mlp* m, const kura::AdamArgs& a, int what, const kura::GatherArgs& ga = kura::GatherArgs{}) {
  kura::UpdArgs u;
  int blocks = what & kura::UPD_GATHER ? kura::GATHER_BLOCKS : 0;
  for (int l = 0; l < NL; ++l) {
    const Layer& L = m->L[l];
    u.l[l] = {L.w_off, L.b_off, L.in_p, L.out_p, (L.in_p / 32) * (L.out_p / 32), L.in_p / 32, m->W[l], m->WT[l], m->dZ[l]};
    blocks += u.l[l].tiles + L.out_p / kura::UPD_BIAS;
  }
  kura::k_mlp_update<<<blocks, kura::UPD_THREADS, 0, m->st>>>(m->P, m->G, u, a, ga, m->Bt, what);
  return cudaGetLastError();
}
cudaError_t gather(kura_mlp* m, const kura::GatherArgs& a) {
  kura::k_mlp_gather<<<kura::GATHER_BLOCKS, 256, 0, m->st>>>(a);
  return cudaGetLastError();
}
cudaError_t pack(kura_mlp* m) { return update(m, kura::AdamArgs{}, kura::UPD_PACK); }

int check_err(kura_mlp* m) {
  int e = 0;
  MLPCU(cudaMemcpy(&e, m->err, sizeof(int), cudaMemcpyDeviceToHost));
  if (e != 0) {
    cudaMemset(m->err, 0, sizeof(int));
    cudaStreamSynchronize(0);
    return mlp_fail(KURA_ERR_BARRIER_TIMEOUT, "a tensor-core GEMM of the MLP timed out waiting for its operands");
  }
  return KURA_OK;
}

// unpadded parameter order: per layer W [out][in] row-major, then b [out]
long long public_count(const kura_mlp* m) {
  long long c = 0;
  for (const Layer& L : m->L) c += (long long)L.out * L.in + L.out;
  return c;
}
void to_public(const kura_mlp* m, const std::vector<float>& pad, float* out) {
  long long k = 0;
  for (const Layer& L : m->L) {
    for (int o = 0; o < L.out; ++o)
      for (int i = 0; i < L.in; ++i) out[k++] = pad[L.w_off + (long long)o * L.in_p + i];
    for (int o = 0; o < L.out; ++o) out[k++] = pad[L.b_off + o];
  }
}

}  // namespace

extern "C" int kura_mlp_create(int32_t in_dim, int32_t hidden, int32_t out_dim, int32_t batch, uint64_t seed,
                               int32_t device, kura_mlp** out) {
  if (!out) return mlp_fail(KURA_ERR_INVALID, "out is NULL");
  *out = nullptr;
  if (in_dim < 1 || in_dim > PADW) return mlp_fail(KURA_ERR_UNSUPPORTED, "in_dim must be 1..64");
  if (out_dim < 1 || out_dim > PADW) return mlp_fail(KURA_ERR_UNSUPPORTED, "out_dim must be 1..64");
  if (hidden != 64 && hidden != 128 && hidden != 256) return mlp_fail(KURA_ERR_UNSUPPORTED, "hidden must be 64, 128 or 256");
  if (batch < 128 || batch > 4096 || batch % 128) return mlp_fail(KURA_ERR_UNSUPPORTED, "batch must be a multiple of 128 in 128..4096");
  kura_mlp* m = new kura_mlp();
  m->device = device;
  m->in_dim = in_dim;
  m->hidden = hidden;
  m->out_dim = out_dim;
  m->Bt = batch;
  const int dims[NL + 1] = {in_dim, hidden, hidden, hidden, out_dim};
  long long off = 0;
  for (int l = 0; l < NL; ++l) {
    Layer& L = m->L[l];
    L.in = dims[l];
    L.out = dims[l + 1];
    L.in_p = kura::round_up(L.in, PADW);
    L.out_p = kura::round_up(L.out, PADW);
    L.out_m = std::max(L.out_p, kura::TG_BM);
    L.w_off = off;
    off += (long long)L.out_p * L.in_p;
    L.b_off = off;
    off += L.out_p;
  }
  m->nparam = off;
  auto bail = [&](int rc) {
    kura_mlp_destroy(m);
    return rc;
  };
  cudaError_t e = cudaSetDevice(device);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&m->sms, cudaDevAttrMultiProcessorCount, device);
  const int Bt = batch;
  if (e == cudaSuccess) e = dalloc(m, &m->P, off);
  if (e == cudaSuccess) e = dalloc(m, &m->G, off);
  if (e == cudaSuccess) e = dalloc(m, &m->Mo, off);
  if (e == cudaSuccess) e = dalloc(m, &m->Vo, off);
  for (int l = 0; l < NL && e == cudaSuccess; ++l) {
    const Layer& L = m->L[l];
    e = dalloc(m, &m->W[l], (size_t)L.out_p * L.in_p);
    if (e == cudaSuccess) e = dalloc(m, &m->WT[l], (size_t)L.out_p * L.in_p);
    if (e == cudaSuccess) e = dalloc(m, &m->H[l], (size_t)Bt * L.in_p);
    if (e == cudaSuccess) e = dalloc(m, &m->HT[l], (size_t)Bt * L.in_p);
    if (e == cudaSuccess && l > 0) e = dalloc(m, &m->S[l], (size_t)Bt * L.in_p);
    if (e == cudaSuccess) e = dalloc(m, &m->dZ[l], (size_t)Bt * L.out_p);
    if (e == cudaSuccess) e = dalloc(m, &m->dZT[l], (size_t)Bt * L.out_m);
  }
  if (e == cudaSuccess) e = dalloc(m, &m->Y, (size_t)Bt * out_dim);
  if (e == cudaSuccess) e = dalloc(m, &m->Tb, (size_t)Bt * out_dim);
  if (e == cudaSuccess) e = dalloc(m, &m->Xin, (size_t)Bt * in_dim);
  if (e == cudaSuccess) e = dalloc(m, &m->Tin, (size_t)Bt * out_dim);
  if (e == cudaSuccess) e = dalloc(m, &m->loss, 1);
  if (e == cudaSuccess) e = dalloc(m, &m->counter, 1);
  if (e == cudaSuccess) e = dalloc(m, &m->err, 1);
  if (e == cudaSuccess) e = cudaMallocHost((void**)&m->y_pin, sizeof(float) * ((size_t)Bt * out_dim + 1));
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&m->st, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaEventCreate(&m->ev[0]);
  if (e == cudaSuccess) e = cudaEventCreate(&m->ev[1]);
  for (cudaStream_t& sd : m->side)
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&sd, cudaStreamNonBlocking);
  for (cudaEvent_t* v : {&m->evz[0], &m->evz[1], &m->evz[2], &m->evz[3], &m->evw[0], &m->evw[1]})
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(v, cudaEventDisableTiming);
  if (e == cudaSuccess) e = set_attr<kura::FwdEpi>();
  if (e == cudaSuccess) e = set_attr<kura::DwEpi>();
  if (e == cudaSuccess) e = set_attr<kura::DhEpi>();
  if (e != cudaSuccess)
    return bail(mlp_fail(e == cudaErrorMemoryAllocation ? KURA_ERR_NOMEM : KURA_ERR_CUDA, cudaGetErrorString(e)));
  // tensor maps of every GEMM operand (the buffers never move)
  for (int l = 0; l < NL; ++l) {
    const Layer& L = m->L[l];
    int bad = kura::make_tmap_16(&m->fA[l], false, m->H[l], L.in_p, Bt, kura::TG_BM);
    bad |= kura::make_tmap_16(&m->fX[l], false, m->W[l], L.in_p, L.out_p, kura::MLP_NC);
    bad |= kura::make_tmap_16(&m->wA[l], false, m->dZT[l], Bt, L.out_m, kura::TG_BM);
    bad |= kura::make_tmap_16(&m->wX[l], false, m->HT[l], Bt, L.in_p, kura::MLP_NC);
    if (l > 0) {
      bad |= kura::make_tmap_16(&m->hA[l], false, m->dZ[l], L.out_p, Bt, kura::TG_BM);
      bad |= kura::make_tmap_16(&m->hX[l], false, m->WT[l], L.out_p, L.in_p, kura::MLP_NC);
    }
    if (bad) return bail(mlp_fail(KURA_ERR_CUDA, "cuTensorMapEncodeTiled failed for an MLP operand"));
  }
  // Glorot-uniform weights from a seeded splitmix64 stream, zero biases and padding
  std::vector<float> p(off, 0.f);
  uint64_t s = seed;
  for (const Layer& L : m->L) {
    const double a = std::sqrt(6.0 / (double)(L.in + L.out));
    for (int o = 0; o < L.out; ++o)
      for (int i = 0; i < L.in; ++i) p[L.w_off + (long long)o * L.in_p + i] = (float)((2 * kura::uniform01(s) - 1) * a);
  }
  e = cudaMemcpy(m->P, p.data(), sizeof(float) * off, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = pack(m);
  if (e == cudaSuccess) e = cudaStreamSynchronize(m->st);
  if (e != cudaSuccess) return bail(mlp_fail(KURA_ERR_CUDA, cudaGetErrorString(e)));
  *out = m;
  return KURA_OK;
}

extern "C" void kura_mlp_destroy(kura_mlp* m) {
  if (!m) return;
  cudaSetDevice(m->device);
  for (cudaStream_t st : {m->st, m->side[0], m->side[1]})
    if (st) cudaStreamSynchronize(st);
  for (void* p : m->allocs) cudaFree(p);
  if (m->y_pin) cudaFreeHost(m->y_pin);
  for (cudaEvent_t v : m->ev)
    if (v) cudaEventDestroy(v);
  for (cudaEvent_t v : m->evz)
    if (v) cudaEventDestroy(v);
  for (cudaEvent_t v : m->evw)
    if (v) cudaEventDestroy(v);
  for (cudaStream_t st : {m->st, m->side[0], m->side[1]})
    if (st) cudaStreamDestroy(st);
  delete m;
}

extern "C" int kura_mlp_param_count(const kura_mlp* m, int64_t* count) {
  if (!m || !count) return mlp_fail(KURA_ERR_INVALID, "NULL argument");
  *count = public_count(m);
  return KURA_OK;
}

extern "C" int kura_mlp_get_params(kura_mlp* m, float* params, int64_t count) {
  if (!m || !params) return mlp_fail(KURA_ERR_INVALID, "NULL argument");
  if (count != public_count(m)) return mlp_fail(KURA_ERR_INVALID, "count must equal kura_mlp_param_count");
  MLPCU(cudaSetDevice(m->device));
  std::vector<float> pad(m->nparam);
  MLPCU(cudaStreamSynchronize(m->st));
  MLPCU(cudaMemcpy(pad.data(), m->P, sizeof(float) * m->nparam, cudaMemcpyDeviceToHost));
  to_public(m, pad, params);
  return KURA_OK;
}

extern "C" int kura_mlp_set_params(kura_mlp* m, const float* params, int64_t count) {
  if (!m || !params) return mlp_fail(KURA_ERR_INVALID, "NULL argument");
  if (count != public_count(m)) return mlp_fail(KURA_ERR_INVALID, "count must equal kura_mlp_param_count");
  MLPCU(cudaSetDevice(m->device));
  std::vector<float> pad(m->nparam, 0.f);
  long long k = 0;
  for (const Layer& L : m->L) {
    for (int o = 0; o < L.out; ++o)
      for (int i = 0; i < L.in; ++i) pad[L.w_off + (long long)o * L.in_p + i] = params[k++];
    for (int o = 0; o < L.out; ++o) pad[L.b_off + o] = params[k++];
  }
  MLPCU(cudaStreamSynchronize(m->st));
  MLPCU(cudaMemcpy(m->P, pad.data(), sizeof(float) * m->nparam, cudaMemcpyHostToDevice));
  MLPCU(pack(m));
  MLPCU(cudaStreamSynchronize(m->st));
  return KURA_OK;
}

extern "C" int kura_mlp_forward(kura_mlp* m, const float* x, int64_t n, float* y) {
  if (!m || !x || !y || n < 0) return mlp_fail(KURA_ERR_INVALID, "bad argument");
  MLPCU(cudaSetDevice(m->device));
  for (int64_t r0 = 0; r0 < n; r0 += m->Bt) {
    const int rows = (int)std::min<int64_t>(m->Bt, n - r0);
    MLPCU(cudaMemcpyAsync(m->Xin, x + r0 * m->in_dim, sizeof(float) * rows * m->in_dim, cudaMemcpyHostToDevice, m->st));
    MLPCU(gather(m, kura::GatherArgs{m->Xin, nullptr, nullptr, nullptr, 0, m->in_dim, m->out_dim, m->Bt, rows, m->H[0],
                                     m->HT[0], m->Tb}));
    MLPCU(forward(m, rows, 0, true));
    // outputs and error flag through pinned memory, one wait for both
    const size_t ny = (size_t)rows * m->out_dim;
    MLPCU(cudaMemcpyAsync(m->y_pin, m->Y, sizeof(float) * ny, cudaMemcpyDeviceToHost, m->st));
    MLPCU(cudaMemcpyAsync(m->y_pin + ny, m->err, sizeof(int), cudaMemcpyDeviceToHost, m->st));
    MLPCU(cudaStreamSynchronize(m->st));
    int flag;
    std::memcpy(&flag, m->y_pin + ny, sizeof flag);
    if (flag) {
      int rc = check_err(m);
      if (rc != KURA_OK) return rc;
    }
    std::memcpy(y + r0 * m->out_dim, m->y_pin, sizeof(float) * ny);
  }
  return KURA_OK;
}

extern "C" int kura_mlp_gradients(kura_mlp* m, const float* x, const float* target, int64_t n, float* grads,
                                  float* loss) {
  if (!m || !x || !target || !grads) return mlp_fail(KURA_ERR_INVALID, "NULL argument");
  if (n < 1 || n > m->Bt) return mlp_fail(KURA_ERR_INVALID, "n must be 1..batch");
  MLPCU(cudaSetDevice(m->device));
  MLPCU(cudaMemcpyAsync(m->Xin, x, sizeof(float) * n * m->in_dim, cudaMemcpyHostToDevice, m->st));
  MLPCU(cudaMemcpyAsync(m->Tin, target, sizeof(float) * n * m->out_dim, cudaMemcpyHostToDevice, m->st));
  MLPCU(gather(m, kura::GatherArgs{m->Xin, m->Tin, nullptr, nullptr, 0, m->in_dim, m->out_dim, m->Bt, (int)n, m->H[0],
                                   m->HT[0], m->Tb}));
  MLPCU(forward(m, m->Bt, (int)n, true));
  MLPCU(backward(m, (int)n, m->loss, nullptr));
  MLPCU(update(m, kura::AdamArgs{}, kura::UPD_BIAS_GRAD));
  std::vector<float> pad(m->nparam);
  float l = 0.f;
  MLPCU(cudaStreamSynchronize(m->st));
  int rc = check_err(m);
  if (rc != KURA_OK) return rc;
  MLPCU(cudaMemcpy(pad.data(), m->G, sizeof(float) * m->nparam, cudaMemcpyDeviceToHost));
  MLPCU(cudaMemcpy(&l, m->loss, sizeof(float), cudaMemcpyDeviceToHost));
  to_public(m, pad, grads);
  if (loss) *loss = l;
  return KURA_OK;
}

extern "C" int kura_mlp_train(kura_mlp* m, const float* x, const float* target, int64_t n_samples, int32_t epochs,
                              float lr, float lr_final, uint64_t shuffle_seed, float* epoch_loss, double* device_ms) {
  if (!m || !x || !target) return mlp_fail(KURA_ERR_INVALID, "NULL argument");
  if (n_samples < m->Bt) return mlp_fail(KURA_ERR_INVALID, "need at least one full batch of samples");
  if (epochs < 1) return mlp_fail(KURA_ERR_INVALID, "epochs must be >= 1");
  MLPCU(cudaSetDevice(m->device));
  const long long per_epoch = n_samples / m->Bt;
  const long long total = per_epoch * epochs;
  // the minibatch rows of every step: one shuffle per epoch (Fisher-Yates on splitmix64)
  std::vector<int> idx((size_t)total * m->Bt);
  std::vector<int> perm(n_samples);
  uint64_t s = shuffle_seed;
  for (int ep = 0; ep < epochs; ++ep) {
    for (long long i = 0; i < n_samples; ++i) perm[i] = (int)i;
    for (long long i = n_samples - 1; i > 0; --i) {
      const long long j = (long long)(kura::splitmix64(s) % (uint64_t)(i + 1));
      std::swap(perm[i], perm[j]);
    }
    std::memcpy(&idx[(size_t)ep * per_epoch * m->Bt], perm.data(), sizeof(int) * per_epoch * m->Bt);
  }
  float *dX = nullptr, *dT = nullptr, *dL = nullptr;
  int* dI = nullptr;
  int rc = KURA_OK;
  cudaGraph_t g = nullptr;
  cudaGraphExec_t ge = nullptr;
  auto run = [&]() -> int {
    MLPCU(cudaMalloc((void**)&dX, sizeof(float) * n_samples * m->in_dim));
    MLPCU(cudaMalloc((void**)&dT, sizeof(float) * n_samples * m->out_dim));
    MLPCU(cudaMalloc((void**)&dI, sizeof(int) * idx.size()));
    MLPCU(cudaMalloc((void**)&dL, sizeof(float) * total));
    MLPCU(cudaMemcpyAsync(dX, x, sizeof(float) * n_samples * m->in_dim, cudaMemcpyHostToDevice, m->st));
    MLPCU(cudaMemcpyAsync(dT, target, sizeof(float) * n_samples * m->out_dim, cudaMemcpyHostToDevice, m->st));
    MLPCU(cudaMemcpyAsync(dI, idx.data(), sizeof(int) * idx.size(), cudaMemcpyHostToDevice, m->st));
    // fresh Adam state
    MLPCU(cudaMemsetAsync(m->Mo, 0, sizeof(float) * m->nparam, m->st));
    MLPCU(cudaMemsetAsync(m->Vo, 0, sizeof(float) * m->nparam, m->st));
    MLPCU(cudaMemsetAsync(m->counter, 0, sizeof(int), m->st));
    MLPCU(cudaStreamSynchronize(m->st));
    const kura::GatherArgs ga{dX, dT, dI, m->counter, total, m->in_dim, m->out_dim, m->Bt, m->Bt, m->H[0], m->HT[0], m->Tb};
    MLPCU(gather(m, ga));
    // one training step, captured; its update gathers the rows of the next one
    MLPCU(cudaStreamBeginCapture(m->st, cudaStreamCaptureModeThreadLocal));
    cudaError_t e = forward(m, m->Bt, m->Bt, false);
    if (e == cudaSuccess) e = backward(m, m->Bt, dL, m->counter);
    if (e == cudaSuccess)
      e = update(m, kura::AdamArgs{m->Mo, m->Vo, m->counter, lr, lr_final, total, 0.9f, 0.999f, 1e-8f},
                 kura::UPD_ADAM | kura::UPD_PACK | kura::UPD_BIAS_GRAD | kura::UPD_GATHER, ga);
    cudaError_t ce = cudaStreamEndCapture(m->st, &g);
    MLPCU(e);
    MLPCU(ce);
    MLPCU(cudaGraphInstantiate(&ge, g, 0));
    MLPCU(cudaEventRecord(m->ev[0], m->st));
    for (long long i = 0; i < total; ++i) MLPCU(cudaGraphLaunch(ge, m->st));
    MLPCU(cudaEventRecord(m->ev[1], m->st));
    MLPCU(cudaStreamSynchronize(m->st));
    int r = check_err(m);
    if (r != KURA_OK) return r;
    float ms = 0.f;
    MLPCU(cudaEventElapsedTime(&ms, m->ev[0], m->ev[1]));
    if (device_ms) *device_ms = ms;
    if (epoch_loss) {
      std::vector<float> lh(total);
      MLPCU(cudaMemcpy(lh.data(), dL, sizeof(float) * total, cudaMemcpyDeviceToHost));
      for (int ep = 0; ep < epochs; ++ep) {
        double a = 0;
        for (long long i = 0; i < per_epoch; ++i) a += lh[(size_t)ep * per_epoch + i];
        epoch_loss[ep] = (float)(a / per_epoch);
      }
    }
    return KURA_OK;
  };
  rc = run();
  if (rc != KURA_OK) cudaGetLastError();
  if (ge) cudaGraphExecDestroy(ge);
  if (g) cudaGraphDestroy(g);
  cudaStreamSynchronize(m->st);
  for (void* p : {(void*)dX, (void*)dT, (void*)dI, (void*)dL})
    if (p) cudaFree(p);
  return rc;
}
