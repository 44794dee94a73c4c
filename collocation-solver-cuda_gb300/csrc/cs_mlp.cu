// Multilayer perceptron for the learned warm start: maps the parameters of
// an OCP instance to its state/costate/control trajectory at fixed
// normalised-time nodes (the Newton initial guess).
//
//   x -> L0 -> GELU -> L1 -> GELU -> ... -> L{D-1} -> y      (D linear layers)
//
// Weights are kept in FP32 (Adam master copy); every GEMM rounds its operands
// to BF16 when it stages them in shared memory and accumulates in FP32 on the
// tensor cores (mma.sync m16n8k16 BF16).  Forward, backward (input and weight
// gradients), MSE loss and Adam are all kernels here; the host only orders
// them.  The reference has no counterpart (it starts Newton from the
// constant guess of the OCP file).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>
#include <string>
#include <vector>

#include "cs_gb300.h"

int cs_internal_set_error(int code, const char* msg);

namespace {

#define MLP_CUDA(call)                                                                   \
  do {                                                                                   \
    cudaError_t e_ = (call);                                                             \
    if (e_ != cudaSuccess) return cs_internal_set_error(CS_ERR_CUDA, cudaGetErrorString(e_)); \
  } while (0)

// ---------------------------------------------------------------- GEMM ----
// C[m][n] (+)= sum_k A(m, k) B(k, n) (+ bias[n]), with strided FP32 operands:
// A(m, k) = A[m * sam + k * sak], B(k, n) = B[k * sbk + n * sbn].
// Tile 64 x 64 x 16 per CTA of 4 warps (2 x 2), each warp 32 x 32 = 2 x 4
// m16n8 tiles.  Epilogue: bias, then optionally GELU with the pre-activation
// kept in P.
constexpr int BM = 64, BN = 64, BK = 16;

struct GemmArgs {
  int M, N, K;
  const float* A;
  long long sam, sak;
  const float* B;
  long long sbk, sbn;
  float* C;
  long long ldc;
  const float* bias;  // [N] or null
  float* P;           // pre-activation out (GELU) or null
  int gelu;           // apply GELU
  int accumulate;     // C += result
};

__device__ __forceinline__ float gelu_f(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float x) {
  return 0.5f * (1.0f + erff(x * 0.70710678118654752f)) + x * 0.39894228040143268f * expf(-0.5f * x * x);
}

__global__ void __launch_bounds__(128) k_gemm_bf16(GemmArgs g) {
  // operand tiles in BF16: As[m][k], Bs[n][k] (K contiguous: the layout the
  // m16n8k16 row.col fragments read)
  __shared__ __nv_bfloat16 As[BM][BK + 8];
  __shared__ __nv_bfloat16 Bs[BN][BK + 8];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int gq = lane >> 2, tq = lane & 3;
  float acc[2][4][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[i][j][q] = 0.f;
  for (int k0 = 0; k0 < g.K; k0 += BK) {
    // stage: 64 x 16 elements of each operand, 8 per thread
    for (int e = tid; e < BM * BK; e += 128) {
      const int r = e / BK, k = e - r * BK;
      const int gm = m0 + r, gk = k0 + k;
      const float va = (gm < g.M && gk < g.K) ? g.A[gm * g.sam + gk * g.sak] : 0.f;
      As[r][k] = __float2bfloat16_rn(va);
      const int gn = n0 + r;
      const float vb = (gn < g.N && gk < g.K) ? g.B[gk * g.sbk + gn * g.sbn] : 0.f;
      Bs[r][k] = __float2bfloat16_rn(vb);
    }
    __syncthreads();
    unsigned af[2][4], bf[4][2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int r = wm + i * 16 + gq;
      af[i][0] = *reinterpret_cast<const unsigned*>(&As[r][2 * tq]);
      af[i][1] = *reinterpret_cast<const unsigned*>(&As[r + 8][2 * tq]);
      af[i][2] = *reinterpret_cast<const unsigned*>(&As[r][2 * tq + 8]);
      af[i][3] = *reinterpret_cast<const unsigned*>(&As[r + 8][2 * tq + 8]);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = wn + j * 8 + gq;
      bf[j][0] = *reinterpret_cast<const unsigned*>(&Bs[c][2 * tq]);
      bf[j][1] = *reinterpret_cast<const unsigned*>(&Bs[c][2 * tq + 8]);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        asm volatile(
            "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
            "{%0,%1,%2,%3};\n"
            : "+f"(acc[i][j][0]), "+f"(acc[i][j][1]), "+f"(acc[i][j][2]), "+f"(acc[i][j][3])
            : "r"(af[i][0]), "r"(af[i][1]), "r"(af[i][2]), "r"(af[i][3]), "r"(bf[j][0]), "r"(bf[j][1]));
      }
    __syncthreads();
  }
  // epilogue: c0 (gq, 2tq), c1 (gq, 2tq+1), c2 (gq+8, 2tq), c3 (gq+8, 2tq+1)
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int m = m0 + wm + i * 16 + gq + ((q & 2) ? 8 : 0);
        const int n = n0 + wn + j * 8 + 2 * tq + (q & 1);
        if (m >= g.M || n >= g.N) continue;
        float v = acc[i][j][q];
        if (g.bias) v += g.bias[n];
        float* c = g.C + (long long)m * g.ldc + n;
        if (g.gelu) {
          if (g.P) g.P[(long long)m * g.ldc + n] = v;
          v = gelu_f(v);
        }
        if (g.accumulate) *c += v; else *c = v;
      }
}

int gemm(cudaStream_t st, const GemmArgs& g) {
  dim3 grid((g.N + BN - 1) / BN, (g.M + BM - 1) / BM);
  k_gemm_bf16<<<grid, 128, 0, st>>>(g);
  MLP_CUDA(cudaGetLastError());
  return CS_OK;
}

// ------------------------------------------------------- fused network ----
// A layer of this network is a few hundred by a few hundred: as GEMMs of
// their own (stage, multiply, write, and read again for the next) the layers
// of a 1024-row step took 1.35 ms in 25 launches against ~10 us of operand
// traffic.  Rows are independent through the whole network, forward and
// backward, so one CTA carries a block of rows through every layer:
//
//   k_net     16 MT rows: normalise (gather), all layers; TRAIN: the loss and
//             the backward pass to the first layer's pre-activation as well
//   k_dw      weight gradients d^T x of all layers, 64 x 64 tiles, the rows
//             split kSplit ways
//   k_update  sums the splits, Adam, and the BF16 copies of the weights
//
// Activations pass from layer to layer in shared memory as the BF16 the tensor
// cores read (the rounding the operands had when they were staged from FP32);
// pre-activations, gradients, weights and sums stay FP32.  The weights are
// kept a second time in BF16 in the order of the mma B fragments (8 columns x
// 32 of k: 16 contiguous bytes per lane), for the forward and for the backward
// product, so a warp reads them from L2 in whole 512-byte lines without
// staging.  Every output element is the same sequence of m16n8k16 products
// over k as before.  Measured (4 -> 256 -> 256 -> 256 -> 322): an epoch of four
// 1024-row steps and the final loss, host copies included, 7.3 -> 0.43 ms; the
// prediction of 8192 rows 270 -> 46 us.  What bounds it now is the chain of
// layers in one CTA (about 5 us each: weights from L2, 16 k steps, GELU).
constexpr int kMaxDepth = 16;
constexpr int kNetDim = 2048;  // widest layer of the fused kernels (shared memory)
constexpr int kSplit = 4;      // row splits of the weight gradients

struct NetDesc {
  int depth, ld;                 // ld: row stride of the shared activations
  int din[kMaxDepth], dout[kMaxDepth];
  int kb[kMaxDepth], kbt[kMaxDepth];          // 32-wide k blocks of W (din) and W^T (dout)
  long long woff[kMaxDepth], boff[kMaxDepth]; // in the parameters
  long long fw[kMaxDepth], bw[kMaxDepth];     // packed weights (elements)
  long long xoff[kMaxDepth], doff[kMaxDepth]; // kept inputs / output gradients, BF16 [rows][pad64]
  long long poff[kMaxDepth];                  // pre-activations, FP32 [rows][dout]
  int soff[kMaxDepth], scols;                 // bias-gradient columns
  long long nparam;
};

__host__ __device__ inline int pad_to(int x, int m) { return (x + m - 1) / m * m; }

struct NetArgs {
  const float* X;
  const float* Y;
  const int* idx;
  const float* norm;  // xm, xs, ym, ys
  const float* w;     // FP32 parameters (biases)
  const __nv_bfloat16* pack;
  int n, rows_cap;
  float* out;         // denormalised predictions [n][nout] (inference)
  float scale;        // 1 / (n nout)
  double* loss;
  __nv_bfloat16* xk;  // kept layer inputs
  __nv_bfloat16* dk;  // kept output gradients
  float* pre;
  float* bsum;        // [CTA][scols]
};

__device__ __forceinline__ void mma_bf16(float* c, const unsigned* a, unsigned b0, unsigned b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void ldsm4(unsigned* r, const __nv_bfloat16* p) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
__device__ __forceinline__ void ldsm4_t(unsigned* r, const __nv_bfloat16* p) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}

// element (n, k) of a packed operand with kb k-blocks
__host__ __device__ inline long long pack_at(int n, int k, int kb) {
  const int lane = (n & 7) * 4 + ((k & 7) >> 1);
  const int e = ((k >> 4) & 1) * 4 + ((k >> 3) & 1) * 2 + (k & 1);
  return (((long long)(n >> 3) * kb + (k >> 5)) * 32 + lane) * 8 + e;
}

// acc = A (16 MT rows in shared memory) x packed B, tiles t0, t0 + NW, ... (KT
// of them) of this warp, NW warps; the weights of KA k blocks are loaded at a
// time (one L2 latency per KA blocks)
template <int MT, int NW, int kTiles, int kAhead>
__device__ __forceinline__ void net_product(const __nv_bfloat16* A, int ld, const __nv_bfloat16* B, int kb, int t0,
                                            int tiles, float (&acc)[MT][kTiles][4]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int j = 0; j < kTiles; ++j)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[i][j][q] = 0.f;
  const uint4* src[kTiles];
#pragma unroll
  for (int j = 0; j < kTiles; ++j) {
    const int t = min(t0 + NW * j, tiles - 1);
    src[j] = reinterpret_cast<const uint4*>(B) + (long long)t * kb * 32 + lane;
  }
  const __nv_bfloat16* arow = A + (lane & 15) * ld + (lane >> 4) * 8;
  for (int k0 = 0; k0 < kb; k0 += kAhead) {
    uint4 b[kAhead][kTiles];
#pragma unroll
    for (int u = 0; u < kAhead; ++u)
#pragma unroll
      for (int j = 0; j < kTiles; ++j)
        if (k0 + u < kb) b[u][j] = src[j][(long long)(k0 + u) * 32];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      if (k0 + u >= kb) break;
#pragma unroll
      for (int s = 0; s < 2; ++s)
#pragma unroll
        for (int i = 0; i < MT; ++i) {
          unsigned a[4];
          ldsm4(a, arow + i * 16 * ld + (k0 + u) * 32 + s * 16);
#pragma unroll
          for (int j = 0; j < kTiles; ++j)
            mma_bf16(acc[i][j], a, s ? b[u][j].z : b[u][j].x, s ? b[u][j].w : b[u][j].y);
        }
    }
  }
}

template <int MT, int NW, int kTiles, int kAhead, bool TRAIN>
__global__ void __launch_bounds__(32 * NW) k_net(NetDesc d, NetArgs g) {
  extern __shared__ __nv_bfloat16 sm[];
  __nv_bfloat16* cur = sm;
  __nv_bfloat16* nxt = sm + 16 * MT * d.ld;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int gq = lane >> 2, tq = lane & 3;
  const int r0 = blockIdx.x * 16 * MT, nin = d.din[0], nout = d.dout[d.depth - 1];
  const float *xm = g.norm, *xs = xm + nin, *ym = xs + nin, *ys = ym + nout;
  // columns past a layer's width stay zero (the packed weights' are zero too)
  for (int e = tid; e < 2 * 16 * MT * d.ld / 2; e += 32 * NW) reinterpret_cast<unsigned*>(sm)[e] = 0u;
  __syncthreads();
  for (int e = tid; e < 16 * MT * nin; e += 32 * NW) {
    const int r = e / nin, c = e - r * nin, row = r0 + r;
    if (row >= g.n) continue;
    const long long src = g.idx ? g.idx[row] : row;
    const __nv_bfloat16 v = __float2bfloat16_rn((g.X[src * nin + c] - xm[c]) / xs[c]);
    cur[r * d.ld + c] = v;
    if (TRAIN) g.xk[d.xoff[0] * g.rows_cap + (long long)row * pad_to(nin, 64) + c] = v;
  }
  __syncthreads();
  float acc[MT][kTiles][4];
  double loss = 0.0;
  for (int l = 0; l < d.depth; ++l) {
    const int dout = d.dout[l], tiles = (dout + 7) / 8;
    const bool last = l == d.depth - 1;
    const float* bias = g.w + d.boff[l];
    for (int t0 = warp; t0 < tiles; t0 += NW * kTiles) {
      net_product<MT, NW, kTiles, kAhead>(cur, d.ld, g.pack + d.fw[l], d.kb[l], t0, tiles, acc);
#pragma unroll
      for (int j = 0; j < kTiles; ++j) {
        float bs[2] = {0.f, 0.f};  // column sums of the output gradient
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int r = i * 16 + gq + ((q & 2) ? 8 : 0), row = r0 + r;
            const int c = (t0 + NW * j) * 8 + 2 * tq + (q & 1);
            if (t0 + NW * j >= tiles || c >= dout) continue;
            float v = acc[i][j][q];
            v += bias[c];
            if (!last) {
              if (TRAIN && row < g.n) g.pre[d.poff[l] * g.rows_cap + (long long)row * dout + c] = v;
              const __nv_bfloat16 h = __float2bfloat16_rn(gelu_f(v));
              nxt[r * d.ld + c] = h;
              if (TRAIN && row < g.n) g.xk[d.xoff[l + 1] * g.rows_cap + (long long)row * pad_to(dout, 64) + c] = h;
            } else if (TRAIN) {
              float dv = 0.f;
              if (row < g.n) {
                const long long src = g.idx ? g.idx[row] : row;
                const float df = v - (g.Y[src * nout + c] - ym[c]) / ys[c];
                dv = 2.0f * df * g.scale;
                loss += (double)df * df;
                g.dk[d.doff[l] * g.rows_cap + (long long)row * pad_to(dout, 64) + c] = __float2bfloat16_rn(dv);
              }
              bs[q & 1] += dv;
              nxt[r * d.ld + c] = __float2bfloat16_rn(dv);
            } else if (row < g.n) {
              g.out[(long long)row * nout + c] = v * ys[c] + ym[c];
            }
          }
        if (TRAIN && last) {
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            for (int o = 4; o < 32; o <<= 1) bs[q] += __shfl_xor_sync(0xffffffffu, bs[q], o);
            const int c = (t0 + NW * j) * 8 + 2 * tq + q;
            if (gq == 0 && t0 + NW * j < tiles && c < dout) g.bsum[(long long)blockIdx.x * d.scols + d.soff[l] + c] = bs[q];
          }
        }
      }
    }
    __syncthreads();
    // this layer's input buffer becomes the next output's: clear the columns
    // up to the next product's k blocks that it will not write
    __nv_bfloat16* t = cur;
    cur = nxt;
    nxt = t;
    if (l + 1 < d.depth || TRAIN) {
      for (int e = tid; e < 16 * MT * d.ld / 2; e += 32 * NW) reinterpret_cast<unsigned*>(nxt)[e] = 0u;
      __syncthreads();
    }
  }
  if constexpr (TRAIN) {
  for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
  if (lane == 0) atomicAdd(g.loss, loss * g.scale);
  // backward: cur holds the output gradient of layer l
  for (int l = d.depth - 1; l > 0; --l) {
    const int di = d.din[l], tiles = (di + 7) / 8;
    const float* pre = g.pre + d.poff[l - 1] * g.rows_cap;
    __nv_bfloat16* dk = g.dk + d.doff[l - 1] * g.rows_cap;
    for (int t0 = warp; t0 < tiles; t0 += NW * kTiles) {
      net_product<MT, NW, kTiles, kAhead>(cur, d.ld, g.pack + d.bw[l], d.kbt[l], t0, tiles, acc);
#pragma unroll
      for (int j = 0; j < kTiles; ++j) {
        float bs[2] = {0.f, 0.f};
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int r = i * 16 + gq + ((q & 2) ? 8 : 0), row = r0 + r;
            const int c = (t0 + NW * j) * 8 + 2 * tq + (q & 1);
            if (t0 + NW * j >= tiles || c >= di) continue;
            float dv = 0.f;
            if (row < g.n) {
              dv = acc[i][j][q] * gelu_grad(pre[(long long)row * di + c]);
              dk[(long long)row * pad_to(di, 64) + c] = __float2bfloat16_rn(dv);
            }
            bs[q & 1] += dv;
            nxt[r * d.ld + c] = __float2bfloat16_rn(dv);
          }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          for (int o = 4; o < 32; o <<= 1) bs[q] += __shfl_xor_sync(0xffffffffu, bs[q], o);
          const int c = (t0 + NW * j) * 8 + 2 * tq + q;
          if (gq == 0 && t0 + NW * j < tiles && c < di) g.bsum[(long long)blockIdx.x * d.scols + d.soff[l - 1] + c] = bs[q];
        }
      }
    }
    __syncthreads();
    __nv_bfloat16* t = cur;
    cur = nxt;
    nxt = t;
    for (int e = tid; e < 16 * MT * d.ld / 2; e += 32 * NW) reinterpret_cast<unsigned*>(nxt)[e] = 0u;
    __syncthreads();
  }
  }
}

// dW[o][i] = sum over rows d[r][o] x[r][i]: one 64 x 64 tile of one layer,
// rows of split blockIdx.y; both operands [row][column] BF16, transposed by
// ldmatrix.  part: [kSplit][nparam].
__global__ void __launch_bounds__(128) k_dw(NetDesc d, const __nv_bfloat16* xk, const __nv_bfloat16* dk, int n,
                                            int rows_cap, float* part) {
  constexpr int KR = 32, LD = 64 + 8;
  __shared__ __align__(16) __nv_bfloat16 Ds[2][KR][LD], Xs[2][KR][LD];
  int l = 0, t = blockIdx.x;
  for (; l < d.depth; ++l) {
    const int nt = ((d.dout[l] + 63) / 64) * ((d.din[l] + 63) / 64);
    if (t < nt) break;
    t -= nt;
  }
  if (l == d.depth) return;
  const int di = d.din[l], dd = d.dout[l], ct = (di + 63) / 64;
  const int o0 = (t / ct) * 64, i0 = (t % ct) * 64;
  const int ldd = pad_to(dd, 64), ldx = pad_to(di, 64);
  const __nv_bfloat16* D = dk + d.doff[l] * rows_cap + o0;
  const __nv_bfloat16* X = xk + d.xoff[l] * rows_cap + i0;
  const int per = pad_to((n + kSplit - 1) / kSplit, KR);
  const int ra = blockIdx.y * per, rb = min(n, ra + per);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32, gq = lane >> 2, tq = lane & 3;
  float acc[2][4][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[i][j][q] = 0.f;
  // 32 rows x 64 columns of each operand: two 16-byte pieces per thread
  uint4 dv[2], xv[2];
  auto fetch = [&](int r) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int e = tid + u * 128, row = r + (e >> 3), c = (e & 7) * 8;
      const bool in = row < rb;
      dv[u] = in ? *reinterpret_cast<const uint4*>(D + (long long)row * ldd + c) : make_uint4(0, 0, 0, 0);
      xv[u] = in ? *reinterpret_cast<const uint4*>(X + (long long)row * ldx + c) : make_uint4(0, 0, 0, 0);
    }
  };
  if (ra < rb) fetch(ra);
  int buf = 0;
  for (int r = ra; r < rb; r += KR, buf ^= 1) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int e = tid + u * 128;
      *reinterpret_cast<uint4*>(&Ds[buf][e >> 3][(e & 7) * 8]) = dv[u];
      *reinterpret_cast<uint4*>(&Xs[buf][e >> 3][(e & 7) * 8]) = xv[u];
    }
    __syncthreads();
    if (r + KR < rb) fetch(r + KR);
#pragma unroll
    for (int ks = 0; ks < KR; ks += 16) {
      unsigned a[2][4], b[2][4];
#pragma unroll
      for (int i = 0; i < 2; ++i)
        ldsm4_t(a[i], &Ds[buf][ks + ((lane >> 4) & 1) * 8 + (lane & 7)][wm + i * 16 + ((lane >> 3) & 1) * 8]);
#pragma unroll
      for (int j = 0; j < 2; ++j)
        ldsm4_t(b[j], &Xs[buf][ks + ((lane >> 3) & 1) * 8 + (lane & 7)][wn + j * 16 + ((lane >> 4) & 1) * 8]);
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) mma_bf16(acc[i][j], a[i], b[j >> 1][(j & 1) * 2], b[j >> 1][(j & 1) * 2 + 1]);
    }
  }
  float* out = part + (long long)blockIdx.y * d.nparam + d.woff[l];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int o = o0 + wm + i * 16 + gq + ((q & 2) ? 8 : 0), c = i0 + wn + j * 8 + 2 * tq + (q & 1);
        if (o < dd && c < di) out[(long long)o * di + c] = acc[i][j][q];
      }
}

// layer and position of parameter e: returns the layer; *o, *i (i = -1: bias o)
__device__ __forceinline__ int net_locate(const NetDesc& d, long long e, int* o, int* i) {
  int l = 0;
  while (l + 1 < d.depth && e >= d.woff[l + 1]) ++l;
  if (e >= d.boff[l]) {
    *o = (int)(e - d.boff[l]);
    *i = -1;
  } else {
    const int q = (int)(e - d.woff[l]);
    *o = q / d.din[l];
    *i = q - *o * d.din[l];
  }
  return l;
}

__device__ __forceinline__ void net_pack(const NetDesc& d, __nv_bfloat16* pack, int l, int o, int i, float w) {
  const __nv_bfloat16 v = __float2bfloat16_rn(w);
  pack[d.fw[l] + pack_at(o, i, d.kb[l])] = v;
  pack[d.bw[l] + pack_at(i, o, d.kbt[l])] = v;
}

__global__ void k_pack(NetDesc d, const float* w, __nv_bfloat16* pack) {
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < d.nparam; e += (long long)gridDim.x * blockDim.x) {
    int o, i;
    const int l = net_locate(d, e, &o, &i);
    if (i >= 0) net_pack(d, pack, l, o, i, w[e]);
  }
}

// gradient of every parameter from the splits (written to g), then Adam and
// the packed copies (step = 0: the gradient only)
__global__ void k_update(NetDesc d, const float* part, const float* bsum, int ctas, float* g, float* w, float* m1,
                         float* m2, __nv_bfloat16* pack, int step, float lr, float b1, float b2, float eps, float c1,
                         float c2) {
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < d.nparam; e += (long long)gridDim.x * blockDim.x) {
    int o, i;
    const int l = net_locate(d, e, &o, &i);
    float gg = 0.f;
    if (i >= 0) {
#pragma unroll
      for (int s = 0; s < kSplit; ++s) gg += part[(long long)s * d.nparam + e];
    } else {
      const float* b = bsum + d.soff[l] + o;
      float p[4] = {0.f, 0.f, 0.f, 0.f};
      int c = 0;
      for (; c + 3 < ctas; c += 4)
#pragma unroll
        for (int q = 0; q < 4; ++q) p[q] += b[(long long)(c + q) * d.scols];
      for (; c < ctas; ++c) p[0] += b[(long long)c * d.scols];
      gg = (p[0] + p[1]) + (p[2] + p[3]);
    }
    if (!step) {
      g[e] = gg;
      continue;
    }
    const float a = b1 * m1[e] + (1.f - b1) * gg;
    const float v = b2 * m2[e] + (1.f - b2) * gg * gg;
    m1[e] = a;
    m2[e] = v;
    const float nw = w[e] - lr * (a / c1) / (sqrtf(v / c2) + eps);
    w[e] = nw;
    if (i >= 0) net_pack(d, pack, l, o, i, nw);
  }
}

// ------------------------------------------------------- small kernels ----
// rows of X, Y by a permutation (mini-batch gather), normalised
__global__ void k_gather(const float* X, const float* Y, const int* idx, int n, int nin, int nout, const float* xm,
                         const float* xs, const float* ym, const float* ys, float* Xb, float* Yb) {
  const long long tot = (long long)n * (nin + nout);
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < tot; e += (long long)gridDim.x * blockDim.x) {
    const int r = (int)(e / (nin + nout)), c = (int)(e - (long long)r * (nin + nout));
    const long long src = idx ? idx[r] : r;
    if (c < nin) Xb[(long long)r * nin + c] = (X[src * nin + c] - xm[c]) / xs[c];
    else if (Y) {
      const int cc = c - nin;
      Yb[(long long)r * nout + cc] = (Y[src * nout + cc] - ym[cc]) / ys[cc];
    }
  }
}

// d = (pred - target) * 2 / (n * nout); loss partial sums
__global__ void k_mse_grad(const float* P, const float* T, long long total, float scale, float* D, double* loss) {
  double s = 0.0;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
    const float d = P[e] - T[e];
    D[e] = 2.0f * d * scale;
    s += (double)d * d;
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(loss, s * scale);
}

// dA = dH * gelu'(P)  (in place on dH)
__global__ void k_gelu_back(float* dH, const float* P, long long total) {
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x)
    dH[e] *= gelu_grad(P[e]);
}

// bias gradient: column sums of dH (rows n)
__global__ void k_colsum(const float* dH, int n, int cols, float* out) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= cols) return;
  float s = 0.f;
  for (int r = 0; r < n; ++r) s += dH[(long long)r * cols + c];
  out[c] = s;
}

__global__ void k_adam(float* w, const float* g, float* m1, float* m2, long long n, float lr, float b1, float b2,
                       float eps, float c1, float c2) {
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
    const float gg = g[e];
    const float a = b1 * m1[e] + (1.f - b1) * gg;
    const float v = b2 * m2[e] + (1.f - b2) * gg * gg;
    m1[e] = a;
    m2[e] = v;
    w[e] -= lr * (a / c1) / (sqrtf(v / c2) + eps);
  }
}

__global__ void k_denorm(float* Y, long long n, int nout, const float* ym, const float* ys) {
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < n * nout; e += (long long)gridDim.x * blockDim.x) {
    const int c = (int)(e % nout);
    Y[e] = Y[e] * ys[c] + ym[c];
  }
}

unsigned grid_for(long long n) { return (unsigned)std::max<long long>(1, std::min<long long>((n + 255) / 256, 4096)); }

}  // namespace

// ================================================================= MLP ===
struct cs_mlp {
  int nin, width, depth, nout;
  std::vector<int> din, dout;  // per layer
  std::vector<long long> woff, boff;
  long long nparam = 0;
  char* block = nullptr;  // the device memory of w .. pack
  float* w = nullptr;   // all weights and biases, FP32
  float* g = nullptr;   // gradients
  float* m1 = nullptr;  // Adam moments
  float* m2 = nullptr;
  float* norm = nullptr;  // xm, xs, ym, ys
  long long step = 0;
  float lr_final = -1.f;  // cosine decay of the learning rate to lr_final * lr (< 0: constant)
  cudaStream_t st = nullptr;
  // activations for a batch of up to cap rows
  int cap = 0;
  std::vector<float*> act, pre;  // act[l]: input of layer l (act[0] = x), act[depth] = output
  float* tgt = nullptr;
  float* dbuf[2] = {nullptr, nullptr};
  double* dloss = nullptr;
  int* didx = nullptr;
  // fused kernels (every layer at most kNetDim wide)
  bool fused = false;
  int sms = 1;        // of the network's device
  NetDesc net;
  __nv_bfloat16* pack = nullptr;
  bool stale = true;  // the packed weights are older than w
  int rows_cap = 0;   // training rows the buffers below hold
  __nv_bfloat16 *xk = nullptr, *dk = nullptr;
  float *kpre = nullptr, *bsum = nullptr, *part = nullptr;
  // device copies of the caller's arrays, kept from call to call
  struct Buf {
    void* p = nullptr;
    size_t bytes = 0;
  } in_x, in_y, in_perm, out_y;
};

static void mlp_free_acts(cs_mlp* M) {
  for (float* p : M->act) cudaFree(p);
  for (float* p : M->pre) cudaFree(p);
  M->act.clear();
  M->pre.clear();
  cudaFree(M->tgt);
  cudaFree(M->dbuf[0]);
  cudaFree(M->dbuf[1]);
  cudaFree(M->didx);
  M->tgt = M->dbuf[0] = M->dbuf[1] = nullptr;
  M->didx = nullptr;
  M->cap = 0;
}

static int mlp_reserve(cs_mlp* M, int rows) {
  if (rows <= M->cap) return CS_OK;
  mlp_free_acts(M);
  const int cap = std::max(rows, 256);
  M->act.resize(M->depth + 1, nullptr);
  M->pre.resize(M->depth, nullptr);
  for (int l = 0; l <= M->depth; ++l) {
    const int cols = (l == 0) ? M->nin : M->dout[l - 1];
    MLP_CUDA(cudaMalloc(&M->act[l], (size_t)cap * cols * sizeof(float)));
  }
  for (int l = 0; l < M->depth; ++l) MLP_CUDA(cudaMalloc(&M->pre[l], (size_t)cap * M->dout[l] * sizeof(float)));
  const int wmax = std::max(M->width, std::max(M->nout, M->nin));
  MLP_CUDA(cudaMalloc(&M->tgt, (size_t)cap * M->nout * sizeof(float)));
  MLP_CUDA(cudaMalloc(&M->dbuf[0], (size_t)cap * wmax * sizeof(float)));
  MLP_CUDA(cudaMalloc(&M->dbuf[1], (size_t)cap * wmax * sizeof(float)));
  MLP_CUDA(cudaMalloc(&M->didx, (size_t)cap * sizeof(int)));
  M->cap = cap;
  return CS_OK;
}

// grow-only device buffer of the network
static int mlp_buf(cs_mlp::Buf& b, size_t bytes) {
  if (b.bytes >= bytes) return CS_OK;
  cudaFree(b.p);
  b.p = nullptr;
  b.bytes = 0;
  MLP_CUDA(cudaMalloc(&b.p, bytes));
  b.bytes = bytes;
  return CS_OK;
}

// At the end of a call (its stream idle): copies of the caller's arrays stay for
// the next call up to this size each (four thousand samples of 322 outputs are
// 5 MB), larger ones go back to the device.
constexpr size_t kMlpKeep = 256ull << 20;
static void mlp_give_back(cs_mlp* M) {
  for (cs_mlp::Buf* b : {&M->in_x, &M->in_y, &M->in_perm, &M->out_y})
    if (b->bytes > kMlpKeep) {
      cudaFree(b->p);
      b->p = nullptr;
      b->bytes = 0;
    }
}

static void net_describe(cs_mlp* M) {
  NetDesc& d = M->net;
  memset(&d, 0, sizeof(d));
  d.depth = M->depth;
  d.nparam = M->nparam;
  long long pk = 0, xo = 0, dof = 0, po = 0;
  int so = 0, mx = 0;
  for (int l = 0; l < M->depth; ++l) {
    const int di = M->din[l], dd = M->dout[l];
    d.din[l] = di;
    d.dout[l] = dd;
    d.woff[l] = M->woff[l];
    d.boff[l] = M->boff[l];
    d.kb[l] = (di + 31) / 32;
    d.kbt[l] = (dd + 31) / 32;
    d.fw[l] = pk;
    pk += (long long)((dd + 7) / 8) * d.kb[l] * 256;
    d.bw[l] = pk;
    pk += (long long)((di + 7) / 8) * d.kbt[l] * 256;
    d.xoff[l] = xo;
    xo += pad_to(di, 64);
    d.doff[l] = dof;
    dof += pad_to(dd, 64);
    d.poff[l] = po;
    po += dd;
    d.soff[l] = so;
    so += dd;
    mx = std::max(mx, std::max(di, dd));
  }
  d.scols = so;
  d.ld = pad_to(mx, 32) + 8;
}

static long long net_pack_elems(const NetDesc& d) {
  const int l = d.depth - 1;
  return d.bw[l] + (long long)((d.din[l] + 7) / 8) * d.kbt[l] * 256;
}
static long long net_xcols(const NetDesc& d) { return d.xoff[d.depth - 1] + pad_to(d.din[d.depth - 1], 64); }
static long long net_dcols(const NetDesc& d) { return d.doff[d.depth - 1] + pad_to(d.dout[d.depth - 1], 64); }
static long long net_pcols(const NetDesc& d) { return d.poff[d.depth - 1] + d.dout[d.depth - 1]; }

static size_t net_smem(const NetDesc& d, int mt) { return (size_t)2 * 16 * mt * d.ld * sizeof(__nv_bfloat16); }

// Launch shapes of k_net <16-row blocks, warps, tiles per warp, k blocks ahead>
// by the rows of the call (4 -> 256^3 -> 322; us per prediction call, 1000 /
// 4000 / 8192 rows):
//   up to one 16-row block per SM: <1, 16, 2, 8>        24 / 36 / 60
//   up to one 32-row block per SM: <2, 16, 2, 8>        32 / 32 / 51
//   more:                          <2, 8, 4, 4>, two CTAs per SM: 38 / 40 / 46
// (64 rows per CTA: 59 / 61 / 61).  Training holds pre-activations and
// gradients back and keeps 16 warps throughout: <2, 16, 2, 4> above one block
// per SM.
static int net_rows(const NetDesc& d, int n, int sms) { return (n <= 16 * sms || net_smem(d, 2) > 200 * 1024) ? 16 : 32; }

static void net_free(cs_mlp* M) {
  cudaFree(M->xk);
  cudaFree(M->dk);
  cudaFree(M->kpre);
  cudaFree(M->bsum);
  cudaFree(M->part);
  M->xk = M->dk = nullptr;
  M->kpre = M->bsum = M->part = nullptr;
  M->rows_cap = 0;
}

// training buffers for n rows; the pad columns of the kept operands are zeroed
// once and never written
static int net_reserve(cs_mlp* M, int n) {
  if (n <= M->rows_cap) return CS_OK;
  net_free(M);
  const NetDesc& d = M->net;
  const size_t rows = (size_t)pad_to(n, 16);
  const size_t xb = rows * net_xcols(d) * sizeof(__nv_bfloat16), db = rows * net_dcols(d) * sizeof(__nv_bfloat16);
  MLP_CUDA(cudaMalloc(&M->xk, xb));
  MLP_CUDA(cudaMalloc(&M->dk, db));
  MLP_CUDA(cudaMalloc(&M->kpre, rows * net_pcols(d) * sizeof(float)));
  MLP_CUDA(cudaMalloc(&M->bsum, (rows / 16) * d.scols * sizeof(float)));
  MLP_CUDA(cudaMalloc(&M->part, (size_t)kSplit * d.nparam * sizeof(float)));
  MLP_CUDA(cudaMemsetAsync(M->xk, 0, xb, M->st));
  MLP_CUDA(cudaMemsetAsync(M->dk, 0, db, M->st));
  M->rows_cap = (int)rows;
  return CS_OK;
}

static int net_weights(cs_mlp* M, cudaStream_t st) {
  if (!M->stale) return CS_OK;
  k_pack<<<grid_for(M->nparam), 256, 0, st>>>(M->net, M->w, M->pack);
  MLP_CUDA(cudaGetLastError());
  M->stale = false;
  return CS_OK;
}

template <int MT, int NW, int KT, int KA, bool TRAIN>
static int net_launch(cs_mlp* M, const NetArgs& g, cudaStream_t st) {
  const size_t smem = net_smem(M->net, MT);
  auto k = k_net<MT, NW, KT, KA, TRAIN>;
  if (smem > 48 * 1024) MLP_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  k<<<(g.n + 16 * MT - 1) / (16 * MT), 32 * NW, smem, st>>>(M->net, g);
  MLP_CUDA(cudaGetLastError());
  return CS_OK;
}

// predictions of n rows (device arrays), denormalised
static int net_predict(cs_mlp* M, const float* dX, int n, float* dY, cudaStream_t st) {
  int rc = net_weights(M, st);
  if (rc != CS_OK) return rc;
  NetArgs g;
  memset(&g, 0, sizeof(g));
  g.X = dX;
  g.norm = M->norm;
  g.w = M->w;
  g.pack = M->pack;
  g.n = n;
  g.out = dY;
  if (net_rows(M->net, n, M->sms) == 16) return net_launch<1, 16, 2, 8, false>(M, g, st);
  if (n <= 32 * M->sms) return net_launch<2, 16, 2, 8, false>(M, g, st);
  return net_launch<2, 8, 4, 4, false>(M, g, st);
}

// loss and gradient (step = 0: into M->g), or one Adam step, on n rows of the
// device arrays (rows idx[0..n) of them when idx is given)
static int net_step(cs_mlp* M, const float* dX, const float* dY, const int* idx, int n, int step, float lr, float c1,
                    float c2) {
  int rc = net_weights(M, M->st);
  if (rc != CS_OK) return rc;
  const NetDesc& d = M->net;
  NetArgs g;
  memset(&g, 0, sizeof(g));
  g.X = dX;
  g.Y = dY;
  g.idx = idx;
  g.norm = M->norm;
  g.w = M->w;
  g.pack = M->pack;
  g.n = n;
  g.rows_cap = M->rows_cap;
  g.scale = 1.0f / (float)((long long)n * M->nout);
  g.loss = M->dloss;
  g.xk = M->xk;
  g.dk = M->dk;
  g.pre = M->kpre;
  g.bsum = M->bsum;
  const int rows = net_rows(d, n, M->sms);
  rc = rows == 16 ? net_launch<1, 16, 2, 8, true>(M, g, M->st) : net_launch<2, 16, 2, 4, true>(M, g, M->st);
  if (rc != CS_OK) return rc;
  int tiles = 0;
  for (int l = 0; l < d.depth; ++l) tiles += ((d.dout[l] + 63) / 64) * ((d.din[l] + 63) / 64);
  k_dw<<<dim3(tiles, kSplit), 128, 0, M->st>>>(d, M->xk, M->dk, n, M->rows_cap, M->part);
  k_update<<<grid_for(d.nparam), 256, 0, M->st>>>(d, M->part, M->bsum, (n + rows - 1) / rows, M->g, M->w, M->m1,
                                                  M->m2, M->pack, step, lr, 0.9f, 0.999f, 1e-8f, c1, c2);
  MLP_CUDA(cudaGetLastError());
  return CS_OK;
}

static int mlp_loss(cs_mlp* M, double* out) {
  MLP_CUDA(cudaMemcpyAsync(out, M->dloss, sizeof(double), cudaMemcpyDeviceToHost, M->st));
  MLP_CUDA(cudaStreamSynchronize(M->st));
  return CS_OK;
}

extern "C" int cs_mlp_create(int n_in, int width, int depth, int n_out, unsigned long long seed, cs_mlp** out) {
  if (!out || n_in < 1 || width < 1 || depth < 1 || n_out < 1 || depth > 16)
    return cs_internal_set_error(CS_ERR_INVALID, "cs_mlp_create: bad sizes");
  cs_mlp* M = new cs_mlp();
  M->nin = n_in;
  M->width = width;
  M->depth = depth;
  M->nout = n_out;
  long long off = 0;
  for (int l = 0; l < depth; ++l) {
    const int di = (l == 0) ? n_in : width;
    const int dd = (l == depth - 1) ? n_out : width;
    M->din.push_back(di);
    M->dout.push_back(dd);
    M->woff.push_back(off);
    off += (long long)di * dd;
    M->boff.push_back(off);
    off += dd;
  }
  M->nparam = off;
  M->fused = std::max(width, std::max(n_in, n_out)) <= kNetDim;
  if (M->fused) net_describe(M);
  // He-style uniform initialisation, seeded
  std::vector<float> hw(off, 0.f);
  std::mt19937_64 rng(seed);
  for (int l = 0; l < depth; ++l) {
    const float bound = std::sqrt(6.0f / (float)M->din[l]) * (l == depth - 1 ? 0.5f : 1.0f);
    std::uniform_real_distribution<float> U(-bound, bound);
    for (long long e = 0; e < (long long)M->din[l] * M->dout[l]; ++e) hw[M->woff[l] + e] = U(rng);
  }
  std::vector<float> nrm(2 * (n_in + n_out));
  for (int c = 0; c < n_in; ++c) { nrm[c] = 0.f; nrm[n_in + c] = 1.f; }
  for (int c = 0; c < n_out; ++c) { nrm[2 * n_in + c] = 0.f; nrm[2 * n_in + n_out + c] = 1.f; }
  // one block: parameters, gradients, Adam moments, normalisation, loss, packed
  // weights
  const size_t pb = (off * sizeof(float) + 255) / 256 * 256, nb = (nrm.size() * sizeof(float) + 255) / 256 * 256;
  const size_t kb = M->fused ? net_pack_elems(M->net) * sizeof(__nv_bfloat16) : 0;
  int dev = 0;
  if (cudaStreamCreateWithFlags(&M->st, cudaStreamNonBlocking) != cudaSuccess || cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&M->sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaMalloc(&M->block, 4 * pb + nb + 256 + kb) != cudaSuccess ||
      (kb && cudaMemsetAsync(M->block + 4 * pb + nb + 256, 0, kb, M->st) != cudaSuccess)) {
    cs_mlp_free(M);
    return cs_internal_set_error(CS_ERR_NOMEM, "cs_mlp_create: device allocation failed");
  }
  M->w = (float*)M->block;
  M->g = (float*)(M->block + pb);
  M->m1 = (float*)(M->block + 2 * pb);
  M->m2 = (float*)(M->block + 3 * pb);
  M->norm = (float*)(M->block + 4 * pb);
  M->dloss = (double*)(M->block + 4 * pb + nb);
  M->pack = (__nv_bfloat16*)(M->block + 4 * pb + nb + 256);
  cudaMemcpyAsync(M->w, hw.data(), off * sizeof(float), cudaMemcpyHostToDevice, M->st);
  cudaMemsetAsync(M->m1, 0, off * sizeof(float), M->st);
  cudaMemsetAsync(M->m2, 0, off * sizeof(float), M->st);
  cudaMemcpyAsync(M->norm, nrm.data(), nrm.size() * sizeof(float), cudaMemcpyHostToDevice, M->st);
  const cudaError_t e = cudaStreamSynchronize(M->st);
  if (e != cudaSuccess) {
    cs_mlp_free(M);
    return cs_internal_set_error(CS_ERR_CUDA, cudaGetErrorString(e));
  }
  *out = M;
  return CS_OK;
}

extern "C" void cs_mlp_free(cs_mlp* M) {
  if (!M) return;
  mlp_free_acts(M);
  net_free(M);
  for (cs_mlp::Buf* b : {&M->in_x, &M->in_y, &M->in_perm, &M->out_y}) cudaFree(b->p);
  cudaFree(M->block);
  if (M->st) cudaStreamDestroy(M->st);
  delete M;
}

extern "C" long long cs_mlp_num_params(const cs_mlp* M) { return M ? M->nparam : 0; }

extern "C" int cs_mlp_set_normalization(cs_mlp* M, const float* in_mean, const float* in_std, const float* out_mean,
                                        const float* out_std) {
  if (!M || !in_mean || !in_std || !out_mean || !out_std) return cs_internal_set_error(CS_ERR_INVALID, "null");
  std::vector<float> nrm;
  nrm.insert(nrm.end(), in_mean, in_mean + M->nin);
  nrm.insert(nrm.end(), in_std, in_std + M->nin);
  nrm.insert(nrm.end(), out_mean, out_mean + M->nout);
  nrm.insert(nrm.end(), out_std, out_std + M->nout);
  MLP_CUDA(cudaMemcpyAsync(M->norm, nrm.data(), nrm.size() * sizeof(float), cudaMemcpyHostToDevice, M->st));
  MLP_CUDA(cudaStreamSynchronize(M->st));
  return CS_OK;
}

extern "C" int cs_mlp_get_params(cs_mlp* M, float* host) {
  if (!M || !host) return cs_internal_set_error(CS_ERR_INVALID, "null");
  MLP_CUDA(cudaMemcpyAsync(host, M->w, M->nparam * sizeof(float), cudaMemcpyDeviceToHost, M->st));
  MLP_CUDA(cudaStreamSynchronize(M->st));
  return CS_OK;
}

extern "C" int cs_mlp_set_params(cs_mlp* M, const float* host) {
  if (!M || !host) return cs_internal_set_error(CS_ERR_INVALID, "null");
  MLP_CUDA(cudaMemcpyAsync(M->w, host, M->nparam * sizeof(float), cudaMemcpyHostToDevice, M->st));
  MLP_CUDA(cudaStreamSynchronize(M->st));
  M->stale = true;
  return CS_OK;
}

// forward on the normalised rows in act[0] (n rows)
static int mlp_forward(cs_mlp* M, int n) {
  for (int l = 0; l < M->depth; ++l) {
    GemmArgs g;
    memset(&g, 0, sizeof(g));
    g.M = n;
    g.N = M->dout[l];
    g.K = M->din[l];
    g.A = M->act[l];
    g.sam = M->din[l];
    g.sak = 1;
    g.B = M->w + M->woff[l];  // W[out][in]: B(k, n) = W[n][k]
    g.sbk = 1;
    g.sbn = M->din[l];
    g.C = M->act[l + 1];
    g.ldc = M->dout[l];
    g.bias = M->w + M->boff[l];
    const bool last = (l == M->depth - 1);
    g.gelu = last ? 0 : 1;
    g.P = last ? nullptr : M->pre[l];
    int rc = gemm(M->st, g);
    if (rc != CS_OK) return rc;
  }
  return CS_OK;
}

// loss and gradients for the rows in act[0] / tgt (n rows)
static int mlp_backward(cs_mlp* M, int n, double* loss_out) {
  const long long tot = (long long)n * M->nout;
  MLP_CUDA(cudaMemsetAsync(M->dloss, 0, sizeof(double), M->st));
  float* d = M->dbuf[0];
  k_mse_grad<<<grid_for(tot), 256, 0, M->st>>>(M->act[M->depth], M->tgt, tot, 1.0f / (float)tot, d, M->dloss);
  for (int l = M->depth - 1; l >= 0; --l) {
    const int di = M->din[l], dd = M->dout[l];
    if (l < M->depth - 1) k_gelu_back<<<grid_for((long long)n * dd), 256, 0, M->st>>>(d, M->pre[l], (long long)n * dd);
    // dW[o][i] = sum_r d[r][o] x[r][i]
    GemmArgs g;
    memset(&g, 0, sizeof(g));
    g.M = dd;
    g.N = di;
    g.K = n;
    g.A = d;
    g.sam = 1;
    g.sak = dd;
    g.B = M->act[l];
    g.sbk = di;
    g.sbn = 1;
    g.C = M->g + M->woff[l];
    g.ldc = di;
    int rc = gemm(M->st, g);
    if (rc != CS_OK) return rc;
    k_colsum<<<(dd + 127) / 128, 128, 0, M->st>>>(d, n, dd, M->g + M->boff[l]);
    if (l > 0) {
      // dx[r][i] = sum_o d[r][o] W[o][i]
      float* dn = (d == M->dbuf[0]) ? M->dbuf[1] : M->dbuf[0];
      GemmArgs h;
      memset(&h, 0, sizeof(h));
      h.M = n;
      h.N = di;
      h.K = dd;
      h.A = d;
      h.sam = dd;
      h.sak = 1;
      h.B = M->w + M->woff[l];
      h.sbk = di;
      h.sbn = 1;
      h.C = dn;
      h.ldc = di;
      rc = gemm(M->st, h);
      if (rc != CS_OK) return rc;
      d = dn;
    }
  }
  MLP_CUDA(cudaGetLastError());
  if (loss_out) {
    MLP_CUDA(cudaMemcpyAsync(loss_out, M->dloss, sizeof(double), cudaMemcpyDeviceToHost, M->st));
    MLP_CUDA(cudaStreamSynchronize(M->st));
  }
  return CS_OK;
}

extern "C" int cs_mlp_gradient(cs_mlp* M, const float* X, const float* Y, int n, double* loss, float* grad) {
  if (!M || !X || !Y || n < 1) return cs_internal_set_error(CS_ERR_INVALID, "cs_mlp_gradient: bad argument");
  int rc = M->fused ? net_reserve(M, n) : mlp_reserve(M, n);
  if (rc == CS_OK) rc = mlp_buf(M->in_x, (size_t)n * M->nin * sizeof(float));
  if (rc == CS_OK) rc = mlp_buf(M->in_y, (size_t)n * M->nout * sizeof(float));
  if (rc != CS_OK) return rc;
  float *dX = (float*)M->in_x.p, *dY = (float*)M->in_y.p;
  MLP_CUDA(cudaMemcpyAsync(dX, X, (size_t)n * M->nin * sizeof(float), cudaMemcpyHostToDevice, M->st));
  MLP_CUDA(cudaMemcpyAsync(dY, Y, (size_t)n * M->nout * sizeof(float), cudaMemcpyHostToDevice, M->st));
  if (M->fused) {
    MLP_CUDA(cudaMemsetAsync(M->dloss, 0, sizeof(double), M->st));
    rc = net_step(M, dX, dY, nullptr, n, 0, 0.f, 1.f, 1.f);
    if (rc == CS_OK && loss) rc = mlp_loss(M, loss);
  } else {
    const float* nr = M->norm;
    k_gather<<<grid_for((long long)n * (M->nin + M->nout)), 256, 0, M->st>>>(
        dX, dY, nullptr, n, M->nin, M->nout, nr, nr + M->nin, nr + 2 * M->nin, nr + 2 * M->nin + M->nout, M->act[0], M->tgt);
    rc = mlp_forward(M, n);
    if (rc == CS_OK) rc = mlp_backward(M, n, loss);
  }
  cudaError_t e = cudaSuccess;
  if (rc == CS_OK && grad) e = cudaMemcpyAsync(grad, M->g, M->nparam * sizeof(float), cudaMemcpyDeviceToHost, M->st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(M->st);
  if (rc == CS_OK && e != cudaSuccess) rc = cs_internal_set_error(CS_ERR_CUDA, cudaGetErrorString(e));
  mlp_give_back(M);
  return rc;
}

extern "C" int cs_mlp_train(cs_mlp* M, const float* X, const float* Y, int n, int epochs, int batch, float lr,
                            unsigned long long seed, double* final_loss) {
  if (!M || !X || !Y || n < 1 || epochs < 1 || batch < 1) return cs_internal_set_error(CS_ERR_INVALID, "cs_mlp_train: bad argument");
  batch = std::min(batch, n);
  int rc = M->fused ? net_reserve(M, batch) : mlp_reserve(M, batch);
  if (rc == CS_OK) rc = mlp_buf(M->in_x, (size_t)n * M->nin * sizeof(float));
  if (rc == CS_OK) rc = mlp_buf(M->in_y, (size_t)n * M->nout * sizeof(float));
  if (rc == CS_OK) rc = mlp_buf(M->in_perm, (size_t)n * sizeof(int));
  if (rc != CS_OK) return rc;
  float *dX = (float*)M->in_x.p, *dY = (float*)M->in_y.p;
  int* dperm = (int*)M->in_perm.p;
  MLP_CUDA(cudaMemcpyAsync(dX, X, (size_t)n * M->nin * sizeof(float), cudaMemcpyHostToDevice, M->st));
  MLP_CUDA(cudaMemcpyAsync(dY, Y, (size_t)n * M->nout * sizeof(float), cudaMemcpyHostToDevice, M->st));
  std::vector<int> perm(n);
  for (int i = 0; i < n; ++i) perm[i] = i;
  std::mt19937_64 rng(seed);
  const float* nr = M->norm;
  double last = 0.0;
  // learning rate of step q of this call: constant, or cosine from lr down to
  // lr_final * lr over the call's steps
  const long long total = (long long)epochs * (n / batch);
  long long q = 0;
  for (int ep = 0; ep < epochs && rc == CS_OK; ++ep) {
    std::shuffle(perm.begin(), perm.end(), rng);
    MLP_CUDA(cudaMemcpyAsync(dperm, perm.data(), (size_t)n * sizeof(int), cudaMemcpyHostToDevice, M->st));
    double ep_loss = 0.0;
    for (int s = 0; s + batch <= n && rc == CS_OK; s += batch) {
      if (!M->fused) {
        k_gather<<<grid_for((long long)batch * (M->nin + M->nout)), 256, 0, M->st>>>(
            dX, dY, dperm + s, batch, M->nin, M->nout, nr, nr + M->nin, nr + 2 * M->nin, nr + 2 * M->nin + M->nout,
            M->act[0], M->tgt);
        rc = mlp_forward(M, batch);
        if (rc == CS_OK) rc = mlp_backward(M, batch, nullptr);
        if (rc != CS_OK) break;
      }
      M->step += 1;
      const float b1 = 0.9f, b2 = 0.999f;
      const float c1 = 1.f - std::pow(b1, (float)M->step), c2 = 1.f - std::pow(b2, (float)M->step);
      float lq = lr;
      if (M->lr_final >= 0.f && total > 1) {
        const double f = M->lr_final + 0.5 * (1.0 - M->lr_final) * (1.0 + std::cos(3.14159265358979323846 * (double)q / (double)(total - 1)));
        lq = (float)(lr * f);
      }
      ++q;
      if (M->fused) rc = net_step(M, dX, dY, dperm + s, batch, 1, lq, c1, c2);
      else k_adam<<<grid_for(M->nparam), 256, 0, M->st>>>(M->w, M->g, M->m1, M->m2, M->nparam, lq, b1, b2, 1e-8f, c1, c2);
    }
    if (rc == CS_OK && ep == epochs - 1) {
      // loss of the final parameters on the last mini-batch
      if (M->fused) {
        MLP_CUDA(cudaMemsetAsync(M->dloss, 0, sizeof(double), M->st));
        rc = net_step(M, dX, dY, dperm + (n / batch - 1) * batch, batch, 0, 0.f, 1.f, 1.f);
        if (rc == CS_OK) rc = mlp_loss(M, &ep_loss);
      } else {
        rc = mlp_forward(M, batch);
        if (rc == CS_OK) rc = mlp_backward(M, batch, &ep_loss);
      }
      last = ep_loss;
    }
  }
  cudaError_t e = cudaStreamSynchronize(M->st);
  if (rc == CS_OK && e != cudaSuccess) rc = cs_internal_set_error(CS_ERR_CUDA, cudaGetErrorString(e));
  mlp_give_back(M);
  if (final_loss) *final_loss = last;
  return rc;
}

extern "C" int cs_mlp_set_schedule(cs_mlp* M, float lr_final) {
  if (!M || lr_final > 1.f) return cs_internal_set_error(CS_ERR_INVALID, "cs_mlp_set_schedule: bad argument");
  M->lr_final = lr_final;
  return CS_OK;
}

extern "C" int cs_mlp_predict_device(cs_mlp* M, const float* dX, int n, float* dY, void* stream) {
  if (!M || !dX || !dY || n < 1) return cs_internal_set_error(CS_ERR_INVALID, "cs_mlp_predict_device: bad argument");
  cudaStream_t st = stream ? (cudaStream_t)stream : M->st;
  if (M->fused) {
    const int rf = net_predict(M, dX, n, dY, st);
    const cudaError_t ef = cudaStreamSynchronize(st);
    return (rf == CS_OK && ef != cudaSuccess) ? cs_internal_set_error(CS_ERR_CUDA, cudaGetErrorString(ef)) : rf;
  }
  const int chunk = 65536;
  int rc = mlp_reserve(M, std::min(n, chunk));
  if (rc != CS_OK) return rc;
  cudaStream_t keep = M->st;
  M->st = st;
  const float* nr = M->norm;
  for (int s = 0; s < n && rc == CS_OK; s += chunk) {
    const int c = std::min(chunk, n - s);
    k_gather<<<grid_for((long long)c * M->nin), 256, 0, st>>>(dX + (size_t)s * M->nin, nullptr, nullptr, c, M->nin, 0,
                                                               nr, nr + M->nin, nullptr, nullptr, M->act[0], nullptr);
    rc = mlp_forward(M, c);
    if (rc != CS_OK) break;
    float* out = M->act[M->depth];
    k_denorm<<<grid_for((long long)c * M->nout), 256, 0, st>>>(out, c, M->nout, nr + 2 * M->nin,
                                                                nr + 2 * M->nin + M->nout);
    cudaMemcpyAsync(dY + (size_t)s * M->nout, out, (size_t)c * M->nout * sizeof(float), cudaMemcpyDeviceToDevice, st);
  }
  M->st = keep;
  cudaError_t e = cudaStreamSynchronize(st);
  if (rc == CS_OK && e != cudaSuccess) rc = cs_internal_set_error(CS_ERR_CUDA, cudaGetErrorString(e));
  return rc;
}

extern "C" int cs_mlp_predict(cs_mlp* M, const float* X, int n, float* Y) {
  if (!M || !X || !Y || n < 1) return cs_internal_set_error(CS_ERR_INVALID, "cs_mlp_predict: bad argument");
  const int chunk = 65536;
  int rc = M->fused ? mlp_buf(M->out_y, (size_t)std::min(n, chunk) * M->nout * sizeof(float)) : mlp_reserve(M, std::min(n, chunk));
  if (rc == CS_OK) rc = mlp_buf(M->in_x, (size_t)std::min(n, chunk) * M->nin * sizeof(float));
  if (rc != CS_OK) return rc;
  float* dX = (float*)M->in_x.p;
  const float* nr = M->norm;
  for (int s = 0; s < n && rc == CS_OK; s += chunk) {
    const int c = std::min(chunk, n - s);
    if (M->fused) {
      cudaMemcpyAsync(dX, X + (size_t)s * M->nin, (size_t)c * M->nin * sizeof(float), cudaMemcpyHostToDevice, M->st);
      rc = net_predict(M, dX, c, (float*)M->out_y.p, M->st);
      if (rc == CS_OK)
        cudaMemcpyAsync(Y + (size_t)s * M->nout, M->out_y.p, (size_t)c * M->nout * sizeof(float), cudaMemcpyDeviceToHost, M->st);
      continue;
    }
    cudaMemcpyAsync(dX, X + (size_t)s * M->nin, (size_t)c * M->nin * sizeof(float), cudaMemcpyHostToDevice, M->st);
    k_gather<<<grid_for((long long)c * M->nin), 256, 0, M->st>>>(dX, nullptr, nullptr, c, M->nin, 0, nr, nr + M->nin,
                                                                  nullptr, nullptr, M->act[0], nullptr);
    rc = mlp_forward(M, c);
    if (rc != CS_OK) break;
    float* out = M->act[M->depth];
    k_denorm<<<grid_for((long long)c * M->nout), 256, 0, M->st>>>(out, c, M->nout, nr + 2 * M->nin,
                                                                   nr + 2 * M->nin + M->nout);
    cudaMemcpyAsync(Y + (size_t)s * M->nout, out, (size_t)c * M->nout * sizeof(float), cudaMemcpyDeviceToHost, M->st);
  }
  cudaError_t e = cudaStreamSynchronize(M->st);
  if (rc == CS_OK && e != cudaSuccess) rc = cs_internal_set_error(CS_ERR_CUDA, cudaGetErrorString(e));
  mlp_give_back(M);
  return rc;
}
