// Standalone solve of one bordered almost-block-diagonal (BABD) system, the
// linear system of one Newton step after condensation:
//
//   A_i dy_i + C_i dy_{i+1} + H_i dp = b_i            i = 0 .. n-1
//   B_0 dy_0 + B_n dy_n     + V_n dp = -r              (ny + np rows)
//
// Reference: solve_babd_system.py (partition_factorization_parallel,
// construct_babd_mshoot, qr_decomposition, backward_substitution,
// recover_babd_solution, partition_backward_substitution_parallel,
// solve_babd_system.py:93-572), which sweeps 8 partitions sequentially and
// solves the reduced system on the host.  Here: a tree of pairwise Householder
// eliminations (one warp per merge, every level across the whole system), the
// dense top system with the boundary conditions, and back substitution down
// the tree, all on the device.  Sizes are run-time values (ny <= 32,
// np <= 32), unlike the problem-specialised solver kernels.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <mutex>
#include <string>

#include "cs_fp64.cuh"
#include "cs_gb300.h"

int cs_internal_set_error(int code, const char* msg);
int cs_internal_pool(cudaMemPool_t* out);

namespace {

struct BabdDims {
  int ny, np, n;  // block size, parameters, intervals
  int rowsz;      // ny * (2 ny + np + 1): a block row [A | C | H | b], column-major
  int treesz;     // ny * (3 ny + np + 1): a tree record [R | G | E | J | d]
  int qc, qld;    // merge columns, merge leading dimension
  int nt, tld;    // top system size, its leading dimension
};

BabdDims dims_of(int ny, int np, int n) {
  BabdDims d;
  d.ny = ny;
  d.np = np;
  d.n = n;
  d.rowsz = ny * (2 * ny + np + 1);
  d.treesz = ny * (3 * ny + np + 1);
  d.qc = 3 * ny + np + 1;
  d.qld = (2 * ny) | 1;
  d.nt = 2 * ny + np;
  d.tld = d.nt | 1;
  return d;
}

// scratch doubles: two block-row buffers and the tree records
size_t scratch_doubles(const BabdDims& d) {
  return 2 * (size_t)d.n * d.rowsz + (size_t)(d.n + 1) * d.treesz;
}

// A reflection is skipped only for a column that is zero below (and on) the
// diagonal (entries under about 1e-145): any other column is reflected whatever its scale, so a system
// multiplied by any factor gives the same solution (an absolute cut-off of
// the order of eps would leave the columns of a system scaled by 1e-9
// unreduced and the back substitution wrong).
constexpr double kZeroVs = 1e-290;

__device__ __forceinline__ int rows_at(int n0, int l) {
  int n = n0;
  for (int q = 0; q < l; ++q) n = (n + 1) >> 1;
  return n;
}

// inputs in the reference's row-major layout -> column-major block rows
__global__ void kb_pack(BabdDims d, const double* A, const double* C, const double* H, const double* b, double* rows) {
  const long long total = (long long)d.n * d.rowsz;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(e / d.rowsz);
    const int q = (int)(e - (long long)i * d.rowsz);
    const int c = q / d.ny, r = q - c * d.ny;
    double v;
    if (c < d.ny) v = A[((size_t)i * d.ny + r) * d.ny + c];
    else if (c < 2 * d.ny) v = C[((size_t)i * d.ny + r) * d.ny + (c - d.ny)];
    else if (c < 2 * d.ny + d.np) v = H[((size_t)i * d.ny + r) * d.np + (c - 2 * d.ny)];
    else v = b[(size_t)i * d.ny + r];
    rows[e] = v;
  }
}

// one merge (or the carried odd row) of tree level l, one warp per item
__global__ void kb_level(BabdDims d, int l, const double* src, double* dst, double* tree) {
  extern __shared__ double sm[];
  const int wpc = blockDim.x >> 5, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double* Q = sm + (size_t)w * d.qld * d.qc;
  const int nl = rows_at(d.n, l);
  const int merges = nl >> 1;
  const int items = (nl + 1) >> 1;
  const int ny = d.ny;
  for (int mi = blockIdx.x * wpc + w; mi < items; mi += gridDim.x * wpc) {
    if (mi >= merges) {
      const double* sr = src + (size_t)(nl - 1) * d.rowsz;
      double* dr = dst + (size_t)merges * d.rowsz;
      for (int q = lane; q < d.rowsz; q += 32) dr[q] = sr[q];
      continue;
    }
    const double* ra = src + (size_t)(2 * mi) * d.rowsz;
    const double* rb = src + (size_t)(2 * mi + 1) * d.rowsz;
    for (int c = lane; c < d.qc; c += 32) {
      double* col = Q + (size_t)c * d.qld;
      for (int r = 0; r < ny; ++r) {
        double top, bot;
        if (c < ny) { top = ra[(ny + c) * ny + r]; bot = rb[c * ny + r]; }
        else if (c < 2 * ny) { top = ra[(c - ny) * ny + r]; bot = 0.0; }
        else if (c < 3 * ny) { top = 0.0; bot = rb[(ny + c - 2 * ny) * ny + r]; }
        else { top = ra[(2 * ny + c - 3 * ny) * ny + r]; bot = rb[(2 * ny + c - 3 * ny) * ny + r]; }
        col[r] = top;
        col[ny + r] = bot;
      }
    }
    __syncwarp();
    for (int k = 0; k < ny; ++k) {
      const double* vk = Q + (size_t)k * d.qld;
      double ss = 0.0;
      for (int r = k + lane; r < 2 * ny; r += 32) ss += vk[r] * vk[r];
      for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      const double x0 = vk[k];
      const double g = (x0 >= 0.0) ? -sqrt(ss) : sqrt(ss);
      const double v0 = x0 - g;
      const double vs = ss - x0 * x0 + v0 * v0;
      __syncwarp();
      if (vs < kZeroVs) continue;
      const double beta = -2.0 / vs;
      for (int c = k + 1 + lane; c < d.qc; c += 32) {
        double* col = Q + (size_t)c * d.qld;
        double wv = v0 * col[k];
        for (int r = k + 1; r < 2 * ny; ++r) wv += vk[r] * col[r];
        const double bw = beta * wv;
        col[k] = fma(bw, v0, col[k]);
        for (int r = k + 1; r < 2 * ny; ++r) col[r] = fma(bw, vk[r], col[r]);
      }
      __syncwarp();
      if (lane == 0) {
        double* col = Q + (size_t)k * d.qld;
        col[k] = g;
        for (int r = k + 1; r < 2 * ny; ++r) col[r] = 0.0;
      }
      __syncwarp();
    }
    const int mid = (2 * mi + 1) << l;
    double* rec = tree + (size_t)mid * d.treesz;
    double* out = dst + (size_t)mi * d.rowsz;
    for (int c = lane; c < d.qc; c += 32) {
      const double* col = Q + (size_t)c * d.qld;
      for (int r = 0; r < ny; ++r) rec[(size_t)c * ny + r] = col[r];
      if (c >= ny)
        for (int r = 0; r < ny; ++r) out[(size_t)(c - ny) * ny + r] = col[ny + r];
    }
    __syncwarp();
  }
}

// top system [At Ct Ht; B_0 B_n V_n] [dy_0; dy_n; dp] = [bt; -r], one warp
__global__ void kb_top(BabdDims d, const double* row, const double* B0, const double* Bn, const double* Vn,
                       const double* r, double* dy, double* dp, int* singular) {
  extern __shared__ double top[];
  const int lane = threadIdx.x & 31;
  const int ny = d.ny, np = d.np, nt = d.nt, tld = d.tld;
  for (int c = lane; c < nt + 1; c += 32) {
    double* col = top + (size_t)c * tld;
    for (int q = 0; q < ny; ++q) col[q] = (c < 2 * ny + np) ? row[(size_t)c * ny + q] : row[(size_t)(2 * ny + np) * ny + q];
    for (int q = 0; q < ny + np; ++q) {
      double v;
      if (c < ny) v = B0[(size_t)q * ny + c];
      else if (c < 2 * ny) v = Bn[(size_t)q * ny + (c - ny)];
      else if (c < nt) v = Vn[(size_t)q * np + (c - 2 * ny)];
      else v = -r[q];
      col[ny + q] = v;
    }
  }
  __syncwarp();
  for (int k = 0; k < nt; ++k) {
    const double* vk = top + (size_t)k * tld;
    double ss = 0.0;
    for (int q = k + lane; q < nt; q += 32) ss += vk[q] * vk[q];
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const double x0 = vk[k];
    const double g = (x0 >= 0.0) ? -sqrt(ss) : sqrt(ss);
    const double v0 = x0 - g;
    const double vs = ss - x0 * x0 + v0 * v0;
    __syncwarp();
    if (vs < kZeroVs) continue;
    const double beta = -2.0 / vs;
    for (int c = k + 1 + lane; c < nt + 1; c += 32) {
      double* col = top + (size_t)c * tld;
      double wv = v0 * col[k];
      for (int q = k + 1; q < nt; ++q) wv += vk[q] * col[q];
      const double bw = beta * wv;
      col[k] = fma(bw, v0, col[k]);
      for (int q = k + 1; q < nt; ++q) col[q] = fma(bw, vk[q], col[q]);
    }
    __syncwarp();
    if (lane == 0) {
      double* col = top + (size_t)k * tld;
      col[k] = g;
      for (int q = k + 1; q < nt; ++q) col[q] = 0.0;
    }
    __syncwarp();
  }
  if (lane == 0) {
    double* rhs = top + (size_t)nt * tld;
    int sing = 0;
    for (int q = nt - 1; q >= 0; --q) {
      double v = rhs[q];
      for (int c = q + 1; c < nt; ++c) v -= top[(size_t)c * tld + q] * rhs[c];
      const double dd = top[(size_t)q * tld + q];
      if (dd == 0.0) sing = 1;
      rhs[q] = (dd != 0.0) ? v / dd : 0.0;
    }
    if (sing)
      for (int q = 0; q < nt; ++q) rhs[q] = 0.0;
    *singular = sing;
    for (int q = 0; q < ny; ++q) {
      dy[q] = rhs[q];
      dy[(size_t)d.n * ny + q] = rhs[ny + q];
    }
    for (int q = 0; q < np; ++q) dp[q] = rhs[2 * ny + q];
  }
}

// back substitution of tree level l: dy_m = R^-1 (d - G dy_l - E dy_r - J dp)
__global__ void kb_back(BabdDims d, int l, const double* tree, const double* dp, double* dy) {
  const int wpc = blockDim.x >> 5, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ny = d.ny, np = d.np;
  const int merges = rows_at(d.n, l) >> 1;
  for (int mi = blockIdx.x * wpc + w; mi < merges; mi += gridDim.x * wpc) {
    const int mid = (2 * mi + 1) << l, left = (2 * mi) << l;
    int right = (2 * mi + 2) << l;
    if (right > d.n) right = d.n;
    const double* rec = tree + (size_t)mid * d.treesz;
    const double* yl = dy + (size_t)left * ny;
    const double* yr = dy + (size_t)right * ny;
    double v = 0.0;
    if (lane < ny) {
      v = rec[(size_t)(3 * ny + np) * ny + lane];
      for (int c = 0; c < ny; ++c) v -= rec[(size_t)(ny + c) * ny + lane] * yl[c];
      for (int c = 0; c < ny; ++c) v -= rec[(size_t)(2 * ny + c) * ny + lane] * yr[c];
      for (int c = 0; c < np; ++c) v -= rec[(size_t)(3 * ny + c) * ny + lane] * dp[c];
    }
    for (int q = ny - 1; q >= 0; --q) {
      double xq = __shfl_sync(0xffffffffu, v, q);
      const double rr = rec[(size_t)q * ny + q];
      xq = (rr != 0.0) ? xq / rr : 0.0;
      if (lane == q) v = xq;
      if (lane < q) v -= rec[(size_t)q * ny + lane] * xq;
    }
    if (lane < ny) dy[(size_t)mid * ny + lane] = v;
  }
}

// ---------------------------------------------------------------------------
// Blocks up to 16 x 16: subtrees.  A merge is a chain of ny reflectors, a few
// microseconds whatever the machine, and a system of a thousand rows has eleven
// levels of them: launches and round trips to L2 between the levels cost as
// much again.  So a CTA takes kRows = 8 consecutive rows through three levels in
// shared memory (kb_sub; the first reads the caller's arrays), until one CTA
// holds what is left (kb_root: last levels, top system, first levels down), and
// the back substitution comes down the same chunks (kb_down).  A merge is one
// warp with its columns in registers (CPL columns per lane), rows unrolled to
// NYP >= ny (padding rows are zero); sums over rows run in four chains, since a
// dependent FP64 instruction waits ~64 cycles.  Eight rows: a warp's merge holds
// the SM's FP64 unit for 4 us (ny = 6), so sixteen rows a CTA cost more in the
// first level (8 merges on one SM) than they save in launches (296 us a call
// against 236).  Measured (ny = 6, np = 2, 1500 intervals): 24 launches, 390 us ->
// 7 launches, 190 us; the call, with its scratch from a pool instead of
// cudaMalloc, 650 -> 215 us.
constexpr int kRows = 8, kSubLevels = 3, kSubWarps = 4;
// |v|^2 / 2 below 1e-290 / 2 counts as zero (kZeroVs)
constexpr long long kLeast = 0x03a8f2b061aea072ll;

template <int I>
struct Ix {
  static constexpr int value = I;
};
template <int A, int B, typename F>
__device__ __forceinline__ void static_for(F&& f) {
  if constexpr (A < B) {
    f(Ix<A>());
    static_for<A + 1, B>(f);
  }
}

// one merge of block rows ra, rb (column-major in shared memory) by one warp
template <int NYP, int CPL>
__device__ void sub_merge(const BabdDims& d, const double* ra, const double* rb, double* out, double* rec) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31, ny = d.ny;
  double Q[CPL][2 * NYP];
  static_for<0, CPL>([&](auto sc) {
    constexpr int s = decltype(sc)::value;
    const int c = s * 32 + lane;
    const double *pt = nullptr, *pb = nullptr;
    if (c < ny) { pt = ra + (ny + c) * ny; pb = rb + c * ny; }
    else if (c < 2 * ny) { pt = ra + (c - ny) * ny; }
    else if (c < 3 * ny) { pb = rb + (c - ny) * ny; }
    else if (c < d.qc) { pt = ra + (c - ny) * ny; pb = rb + (c - ny) * ny; }
    static_for<0, NYP>([&](auto rc) {
      constexpr int r = decltype(rc)::value;
      Q[s][r] = (pt && r < ny) ? pt[r] : 0.0;
      Q[s][NYP + r] = (pb && r < ny) ? pb[r] : 0.0;
    });
  });
  static_for<0, NYP>([&](auto kc) {
    constexpr int k = decltype(kc)::value;
    if (k < ny) {
      // rows of the reflector: k .. NYP - 1 and the whole lower block; column k
      // to every lane, its products with the lane's columns (its own: the sum
      // of squares), the reflector in every lane
      double v[2 * NYP], p[CPL];
      static_for<k, 2 * NYP>([&](auto rc) {
        constexpr int r = decltype(rc)::value;
        v[r] = __shfl_sync(full, Q[0][r], k);
      });
      static_for<0, CPL>([&](auto sc) {
        constexpr int s = decltype(sc)::value;
        double a[4] = {0.0, 0.0, 0.0, 0.0};
        static_for<k, 2 * NYP>([&](auto rc) {
          constexpr int r = decltype(rc)::value;
          a[r & 3] = fma(v[r], Q[s][r], a[r & 3]);
        });
        p[s] = (a[0] + a[1]) + (a[2] + a[3]);
      });
      double g, v0, t;
      if (cs_reflector(__shfl_sync(full, p[0], k), v[k], &g, &v0, &t, kLeast)) {
        static_for<0, CPL>([&](auto sc) {
          constexpr int s = decltype(sc)::value;
          const double bw = (s * 32 + lane > k) ? -t * fma(-g, Q[s][k], p[s]) : 0.0;
          Q[s][k] = fma(bw, v0, Q[s][k]);
          static_for<k + 1, 2 * NYP>([&](auto rc) {
            constexpr int r = decltype(rc)::value;
            Q[s][r] = fma(bw, v[r], Q[s][r]);
          });
        });
        if (lane == k) Q[0][k] = g;  // (below it: never read again)
      }
    }
  });
  static_for<0, CPL>([&](auto sc) {
    constexpr int s = decltype(sc)::value;
    const int c = s * 32 + lane;
    if (c < d.qc) {
      static_for<0, NYP>([&](auto rc) {
        constexpr int r = decltype(rc)::value;
        if (r < ny) {
          rec[c * ny + r] = Q[s][r];
          if (c >= ny) out[(c - ny) * ny + r] = Q[s][NYP + r];
        }
      });
    }
  });
}

// The levels l0, l0 + 1, .. of rows [first, first + m) of level l0 (a multiple
// of kRows, m <= kRows), held in buf (kRows + kRows / 2 rows), down to one row
// or `levels` levels; returns the buffer position of the result.
template <int NYP, int CPL>
__device__ double* sub_up(const BabdDims& d, int l0, int first, int m, int levels, double* buf, double* tree) {
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double* in = buf;
  double* out = buf + (size_t)kRows * d.rowsz;
  for (int j = 0; j < levels && m > 1; ++j) {
    const int merges = m >> 1;
    for (int mi = w; mi < merges; mi += kSubWarps) {
      const int node = (2 * ((first >> (j + 1)) + mi) + 1) << (l0 + j);
      sub_merge<NYP, CPL>(d, in + 2 * mi * d.rowsz, in + (2 * mi + 1) * d.rowsz, out + mi * d.rowsz,
                          tree + (size_t)node * d.treesz);
    }
    if (m & 1)
      for (int q = threadIdx.x; q < d.rowsz; q += blockDim.x) out[merges * d.rowsz + q] = in[(m - 1) * d.rowsz + q];
    __syncthreads();
    m = (m + 1) >> 1;
    double* t = in;
    in = out;
    out = t;
  }
  (void)lane;
  return in;
}

// rows [first, first + m) into shared memory: from src (column-major block
// rows), or from the caller's row-major arrays
__device__ void sub_load(const BabdDims& d, const double* src, const double* A, const double* C, const double* H,
                         const double* b, int first, int m, double* buf) {
  if (src) {
    for (int e = threadIdx.x; e < m * d.rowsz; e += blockDim.x) buf[e] = src[(size_t)first * d.rowsz + e];
  } else {
    const int ny = d.ny, np = d.np, nn = ny * ny;
    for (int e = threadIdx.x; e < m * nn; e += blockDim.x) {
      const int i = e / nn, q = e - i * nn, r = q / ny, c = q - r * ny;
      double* row = buf + i * d.rowsz;
      row[c * ny + r] = A[(size_t)first * nn + e];
      row[(ny + c) * ny + r] = C[(size_t)first * nn + e];
    }
    for (int e = threadIdx.x; e < m * ny * np; e += blockDim.x) {
      const int i = e / (ny * np), q = e - i * ny * np, r = q / np, c = q - r * np;
      buf[i * d.rowsz + (2 * ny + c) * ny + r] = H[(size_t)first * ny * np + e];
    }
    for (int e = threadIdx.x; e < m * ny; e += blockDim.x)
      buf[(e / ny) * d.rowsz + (2 * ny + np) * ny + e % ny] = b[(size_t)first * ny + e];
  }
  __syncthreads();
}

template <int NYP, int CPL>
__global__ void __launch_bounds__(32 * kSubWarps) kb_sub(BabdDims d, int l0, int n, const double* src, const double* A,
                                                        const double* C, const double* H, const double* b, double* dst,
                                                        double* tree) {
  extern __shared__ double sm[];
  const int first = blockIdx.x * kRows, m = min(kRows, n - first);
  sub_load(d, src, A, C, H, b, first, m, sm);
  const double* r = sub_up<NYP, CPL>(d, l0, first, m, kSubLevels, sm, tree);
  for (int q = threadIdx.x; q < d.rowsz; q += blockDim.x) dst[(size_t)blockIdx.x * d.rowsz + q] = r[q];
}

// one merge's back substitution, one warp, lanes over rows: dy_m = R^-1 (d - G
// dy_l - E dy_r - J dp).  The record is read before anything waits on it.
template <int NYP>
__device__ __forceinline__ void sub_back(const BabdDims& d, const double* rec, const double* yl, const double* yr,
                                         const double* dp, double* ym) {
  const int ny = d.ny, np = d.np, lane = threadIdx.x & 31;
  const int a = lane < ny ? lane : 0;
  double gl[NYP], er[NYP], rr[NYP];
  static_for<0, NYP>([&](auto cc) {
    constexpr int c = decltype(cc)::value;
    const bool in = c < ny;
    rr[c] = in ? rec[c * ny + a] : 0.0;
    gl[c] = in ? rec[(ny + c) * ny + a] : 0.0;
    er[c] = in ? rec[(2 * ny + c) * ny + a] : 0.0;
  });
  double s = rec[(3 * ny + np) * ny + a], u = 0.0;
  const double diag = rec[a * ny + a];
  for (int c = 0; c < np; ++c) u = fma(rec[(3 * ny + c) * ny + a], dp[c], u);
  static_for<0, NYP>([&](auto cc) {
    constexpr int c = decltype(cc)::value;
    if (c < ny) {
      s = fma(-gl[c], yl[c], s);
      u = fma(er[c], yr[c], u);
    }
  });
  double v = s - u;
  const double inv = diag != 0.0 ? cs_rcp(diag) : 0.0;
  static_for<0, NYP>([&](auto cc) {
    constexpr int q = NYP - 1 - decltype(cc)::value;
    if (q < ny) {
      const double xq = __shfl_sync(0xffffffffu, v * inv, q);
      v = (lane == q) ? xq : (lane < q ? fma(-rr[q], xq, v) : v);
    }
  });
  if (lane < ny) ym[lane] = v;
}

// levels l0 + levels - 1 .. l0 of the chunk's rows, dy at the chunk's ends known
template <int NYP>
__device__ void sub_down(const BabdDims& d, int l0, int first, int m, int levels, const double* tree, const double* dp,
                         double* dy) {
  const int w = threadIdx.x >> 5;
  for (int j = levels - 1; j >= 0; --j) {
    int mj = m;
    for (int q = 0; q < j; ++q) mj = (mj + 1) >> 1;
    const int l = l0 + j;
    for (int mi = w; mi < (mj >> 1); mi += kSubWarps) {
      const int g = (first >> (j + 1)) + mi;
      const int mid = (2 * g + 1) << l, left = (2 * g) << l, right = min((2 * g + 2) << l, d.n);
      sub_back<NYP>(d, tree + (size_t)mid * d.treesz, dy + (size_t)left * d.ny, dy + (size_t)right * d.ny, dp,
               dy + (size_t)mid * d.ny);
    }
    __syncthreads();
  }
}

template <int NYP>
__global__ void __launch_bounds__(32 * kSubWarps) kb_down(BabdDims d, int l0, int n, const double* tree, const double* dp,
                                                         double* dy) {
  const int first = blockIdx.x * kRows;
  sub_down<NYP>(d, l0, first, min(kRows, n - first), kSubLevels, tree, dp, dy);
}

// top system [At Ct Ht; B_0 B_n V_n] [dy_0; dy_n; dp] = [bt; -r], one CTA, a
// column per thread (nt <= 64)
__device__ void sub_top(const BabdDims& d, const double* row, const double* B0, const double* Bn, const double* Vn,
                        const double* r, double* top, double* red, double* dy, double* dp, int* singular) {
  const int ny = d.ny, np = d.np, nt = d.nt, tld = d.tld, tid = threadIdx.x;
  for (int e = tid; e < (nt + 1) * nt; e += blockDim.x) {
    const int c = e / nt, q = e - c * nt;
    double v;
    if (q < ny) v = (c < nt) ? row[c * ny + q] : row[(2 * ny + np) * ny + q];
    else if (c < ny) v = B0[(size_t)(q - ny) * ny + c];
    else if (c < 2 * ny) v = Bn[(size_t)(q - ny) * ny + (c - ny)];
    else if (c < nt) v = Vn[(size_t)(q - ny) * np + (c - 2 * ny)];
    else v = cs_neg(r[q - ny]);
    top[(size_t)c * tld + q] = v;
  }
  __syncthreads();
  for (int k = 0; k < nt; ++k) {
    double* vk = top + (size_t)k * tld;
    const int c = k + tid;  // (nt + 1 <= 65 columns)
    double* col = top + (size_t)min(c, nt) * tld;
    double p = 0.0;
    if (c <= nt) {
      double w[4] = {0.0, 0.0, 0.0, 0.0};
      int q = k;
      for (; q + 3 < nt; q += 4)
#pragma unroll
        for (int u = 0; u < 4; ++u) w[u] = fma(vk[q + u], col[q + u], w[u]);
      for (; q < nt; ++q) w[3] = fma(vk[q], col[q], w[3]);
      p = (w[0] + w[1]) + (w[2] + w[3]);
      if (tid == 0) red[k & 1] = p;
    }
    __syncthreads();
    double g, v0, t;
    const bool on = cs_reflector(red[k & 1], vk[k], &g, &v0, &t, kLeast);
    if (on && c > k && c <= nt) {
      const double bw = -t * fma(-g, col[k], p);
      col[k] = fma(bw, v0, col[k]);
#pragma unroll 4
      for (int q = k + 1; q < nt; ++q) col[q] = fma(bw, vk[q], col[q]);
    }
    __syncthreads();
    if (on && tid == 0) vk[k] = g;  // (read again only after the next barrier; below it never)
  }
  __syncthreads();
  // back substitution, one warp, lanes over the rows of a column
  if (tid < 32) {
    double* rhs = top + (size_t)nt * tld;
    int sing = 0;
    for (int q = nt - 1; q >= 0; --q) {
      const double dd = top[(size_t)q * tld + q];
      sing |= dd == 0.0;
      const double x = dd != 0.0 ? rhs[q] * cs_rcp(dd) : 0.0;
      __syncwarp();
      for (int e = tid; e < q; e += 32) rhs[e] = fma(-top[(size_t)q * tld + e], x, rhs[e]);
      if (tid == 0) rhs[q] = x;
      __syncwarp();
    }
    for (int q = tid; q < nt; q += 32) {
      const double x = sing ? 0.0 : rhs[q];
      if (q < ny) dy[q] = x;
      else if (q < 2 * ny) dy[(size_t)d.n * ny + q - ny] = x;
      else dp[q - 2 * ny] = x;
    }
    if (tid == 0) *singular = sing;
  }
  __syncthreads();
}

// what is left (n <= kRows rows of level l0): the last levels, the top system,
// and those levels' back substitution
template <int NYP, int CPL>
__global__ void __launch_bounds__(32 * kSubWarps) kb_root(BabdDims d, int l0, int n, const double* src, const double* A,
                                                         const double* C, const double* H, const double* b,
                                                         const double* B0, const double* Bn, const double* Vn,
                                                         const double* r, double* tree, double* dy, double* dp,
                                                         int* singular) {
  extern __shared__ double sm[];
  double* top = sm + (size_t)(kRows + kRows / 2) * d.rowsz;
  double* red = top + (size_t)d.tld * (d.nt + 1);
  sub_load(d, src, A, C, H, b, 0, n, sm);
  const double* row = sub_up<NYP, CPL>(d, l0, 0, n, 32, sm, tree);
  sub_top(d, row, B0, Bn, Vn, r, top, red, dy, dp, singular);
  sub_down<NYP>(d, l0, 0, n, kSubLevels, tree, dp, dy);
}

size_t sub_smem(const BabdDims& d) { return (size_t)(kRows + kRows / 2) * d.rowsz * sizeof(double); }
size_t root_smem(const BabdDims& d) { return sub_smem(d) + ((size_t)d.tld * (d.nt + 1) + 4) * sizeof(double); }

// whether the subtree kernels take this system: blocks and shared memory
bool sub_fits(const BabdDims& d) {
  const int cols = d.ny <= 8 ? 64 : 96;
  return d.ny <= 16 && d.qc <= cols && root_smem(d) <= 220 * 1024;
}

template <int NYP, int CPL>
int sub_run(const BabdDims& d, const double* A, const double* C, const double* H, const double* b, const double* B0,
            const double* Bn, const double* Vn, const double* r, double* dy, double* dp, double* scratch, double* tree,
            int* d_singular, cudaStream_t stream) {
  const size_t ssm = sub_smem(d), rsm = root_smem(d);
  cudaError_t e = cudaSuccess;
  if (ssm > 48 * 1024) e = cudaFuncSetAttribute(kb_sub<NYP, CPL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ssm);
  if (e == cudaSuccess && rsm > 48 * 1024)
    e = cudaFuncSetAttribute(kb_root<NYP, CPL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)rsm);
  if (e != cudaSuccess) return cs_internal_set_error(CS_ERR_CUDA, cudaGetErrorString(e));
  int n = d.n, l0 = 0;
  const double* src = nullptr;
  double* dst = scratch;  // results of one chunk level after the other
  while (n > kRows) {
    const int chunks = (n + kRows - 1) / kRows;
    kb_sub<NYP, CPL><<<chunks, 32 * kSubWarps, ssm, stream>>>(d, l0, n, src, A, C, H, b, dst, tree);
    src = dst;
    dst += (size_t)chunks * d.rowsz;
    n = chunks;
    l0 += kSubLevels;
  }
  kb_root<NYP, CPL><<<1, 32 * kSubWarps, rsm, stream>>>(d, l0, n, src, A, C, H, b, B0, Bn, Vn, r, tree, dy, dp, d_singular);
  while (l0 > 0) {
    l0 -= kSubLevels;
    n = d.n;
    for (int l = 0; l < l0; ++l) n = (n + 1) >> 1;
    kb_down<NYP><<<(n + kRows - 1) / kRows, 32 * kSubWarps, 0, stream>>>(d, l0, n, tree, dp, dy);
  }
  e = cudaGetLastError();
  if (e != cudaSuccess) return cs_internal_set_error(CS_ERR_CUDA, cudaGetErrorString(e));
  return CS_OK;
}

int levels_of(int n) {
  int L = 0;
  while (n > 1) {
    n = (n + 1) >> 1;
    ++L;
  }
  return L;
}

int check_sizes(int ny, int np, int n) {
  if (ny < 1 || ny > 32 || np < 0 || np > 32 || n < 1)
    return cs_internal_set_error(CS_ERR_INVALID, "cs_babd_solve: need 1 <= ny <= 32, 0 <= np <= 32, n >= 1");
  return CS_OK;
}

// the whole solve on `stream`, with `scratch` holding scratch_doubles(d) doubles
int babd_run(const BabdDims& d, const double* A, const double* C, const double* H, const double* b, const double* B0,
             const double* Bn, const double* Vn, const double* r, double* dy, double* dp, double* scratch,
             int* d_singular, cudaStream_t stream) {
  double* rows0 = scratch;
  double* rows1 = rows0 + (size_t)d.n * d.rowsz;
  double* tree = rows1 + (size_t)d.n * d.rowsz;
  if (sub_fits(d)) {
#define CS_SUB(NYP, CPL) sub_run<NYP, CPL>(d, A, C, H, b, B0, Bn, Vn, r, dy, dp, rows0, tree, d_singular, stream)
    if (d.ny <= 4) return d.qc <= 32 ? CS_SUB(4, 1) : CS_SUB(4, 2);
    if (d.ny <= 6) return d.qc <= 32 ? CS_SUB(6, 1) : CS_SUB(6, 2);
    if (d.ny <= 8) return d.qc <= 32 ? CS_SUB(8, 1) : CS_SUB(8, 2);
    if (d.ny <= 12 && d.qc <= 64) return CS_SUB(12, 2);
    return d.qc <= 64 ? CS_SUB(16, 2) : CS_SUB(16, 3);
#undef CS_SUB
  }
  const long long pack = (long long)d.n * d.rowsz;
  kb_pack<<<(unsigned)std::min<long long>((pack + 255) / 256, 65535), 256, 0, stream>>>(d, A, C, H, b, rows0);
  const int L = levels_of(d.n);
  const size_t per_warp = (size_t)d.qld * d.qc * sizeof(double);
  const int wpc = (int)std::max<size_t>(1, std::min<size_t>(4, (size_t)(200 * 1024) / per_warp));
  const size_t lsm = per_warp * wpc;
  if (lsm > 48 * 1024) cudaFuncSetAttribute(kb_level, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)lsm);
  double* src = rows0;
  double* dst = rows1;
  for (int l = 0; l < L; ++l) {
    int items = d.n;
    for (int q = 0; q <= l; ++q) items = (items + 1) >> 1;
    const unsigned grid = (unsigned)std::max(1, std::min(65535, (items + wpc - 1) / wpc));
    kb_level<<<grid, 32 * wpc, lsm, stream>>>(d, l, src, dst, tree);
    std::swap(src, dst);
  }
  const size_t tsm = (size_t)d.tld * (d.nt + 1) * sizeof(double);
  if (tsm > 48 * 1024) cudaFuncSetAttribute(kb_top, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tsm);
  kb_top<<<1, 32, tsm, stream>>>(d, src, B0, Bn, Vn, r, dy, dp, d_singular);
  for (int l = L - 1; l >= 0; --l) {
    const int merges = ([&] {
      int m = d.n;
      for (int q = 0; q < l; ++q) m = (m + 1) >> 1;
      return m >> 1;
    })();
    const unsigned grid = (unsigned)std::max(1, std::min(65535, (merges + 3) / 4));
    kb_back<<<grid, 128, 0, stream>>>(d, l, tree, dp, dy);
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cs_internal_set_error(CS_ERR_CUDA, cudaGetErrorString(e));
  return CS_OK;
}

// ---------------------------------------------------------------------------
// Scratch for cs_babd_solve_noalloc: one array in the device image of this
// library, so that callers that cannot allocate device memory can still solve
// a BABD system.  Every GPU that loads the library holds it until the process
// exits.  Element 0 carries the singular flag; the block rows and tree records
// start at element 32 (256-byte aligned).
constexpr size_t kNoallocDoubles = (size_t)4 << 20;  // 32 MiB
__device__ __align__(256) double cs_babd_scratch[kNoallocDoubles];

std::mutex g_noalloc_mu;
void* g_noalloc_addr[128] = {nullptr};

// device address of the scratch array on the current device, looked up once
// per device (host code cannot use the symbol itself as an address)
int noalloc_scratch(double** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cs_internal_set_error(CS_ERR_CUDA, cudaGetErrorString(e));
  if (dev < 0 || dev >= 128) return cs_internal_set_error(CS_ERR_CUDA, "cs_babd_solve_noalloc: device index out of range");
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  if (!g_noalloc_addr[dev]) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, cs_babd_scratch);
    if (e != cudaSuccess || !p)
      return cs_internal_set_error(CS_ERR_CUDA, (std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e)).c_str());
    g_noalloc_addr[dev] = p;
  }
  *out = (double*)g_noalloc_addr[dev];
  return CS_OK;
}

}  // namespace

extern "C" int cs_babd_solve_noalloc(int ny, int np, int n, const double* A, const double* C, const double* H,
                                     const double* b, const double* B0, const double* Bn, const double* Vn,
                                     const double* r, double* dy, double* dp, int* singular, void* stream) {
  int rc = check_sizes(ny, np, n);
  if (rc != CS_OK) return rc;
  if (!A || !C || !b || !B0 || !Bn || !r || !dy || (np > 0 && (!H || !Vn || !dp)))
    return cs_internal_set_error(CS_ERR_INVALID, "cs_babd_solve_noalloc: null pointer");
  const BabdDims d = dims_of(ny, np, n);
  const size_t need = 32 + scratch_doubles(d);
  if (need > kNoallocDoubles)
    return cs_internal_set_error(
        CS_ERR_INVALID, ("cs_babd_solve_noalloc: the system needs " + std::to_string(need * sizeof(double)) +
                         " bytes of scratch, more than the fixed " + std::to_string(kNoallocDoubles * sizeof(double)) +
                         " bytes; use cs_babd_solve").c_str());
  double* base = nullptr;
  rc = noalloc_scratch(&base);
  if (rc != CS_OK) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  // every element read below is written earlier in the same call (packing,
  // tree levels, top system), so nothing needs clearing between calls
  int* dsing = (int*)base;
  rc = babd_run(d, A, C, H, b, B0, Bn, Vn, r, dy, dp, base + 32, dsing, st);
  int hs = 0;
  if (rc == CS_OK) {
    cudaError_t e = cudaMemcpyAsync(&hs, dsing, sizeof(int), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) rc = cs_internal_set_error(CS_ERR_CUDA, cudaGetErrorString(e));
  }
  if (singular) *singular = hs;
  return rc;
}

extern "C" int cs_babd_solve(int ny, int np, int n, const double* A, const double* C, const double* H,
                             const double* b, const double* B0, const double* Bn, const double* Vn, const double* r,
                             double* dy, double* dp, int* singular, void* stream) {
  const int bad = check_sizes(ny, np, n);
  if (bad != CS_OK) return bad;
  if (!A || !C || !b || !B0 || !Bn || !r || !dy || (np > 0 && (!H || !Vn || !dp)))
    return cs_internal_set_error(CS_ERR_INVALID, "cs_babd_solve: null pointer");
  const BabdDims d = dims_of(ny, np, n);
  cudaStream_t st = (cudaStream_t)stream;
  // scratch from the library's stream-ordered pool (element 0 carries the
  // singular flag)
  cudaMemPool_t pool = nullptr;
  int rc = cs_internal_pool(&pool);
  if (rc != CS_OK) return rc;
  void* mem = nullptr;
  cudaError_t e = cudaMallocFromPoolAsync(&mem, (32 + scratch_doubles(d)) * sizeof(double), pool, st);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return cs_internal_set_error(CS_ERR_NOMEM, "cs_babd_solve: device allocation failed");
  }
  int* dsing = (int*)mem;
  rc = babd_run(d, A, C, H, b, B0, Bn, Vn, r, dy, dp, (double*)mem + 32, dsing, st);
  int hs = 0;
  if (rc == CS_OK) {
    e = cudaMemcpyAsync(&hs, dsing, sizeof(int), cudaMemcpyDeviceToHost, st);
    if (e != cudaSuccess) rc = cs_internal_set_error(CS_ERR_CUDA, cudaGetErrorString(e));
  }
  cudaFreeAsync(mem, st);
  e = cudaStreamSynchronize(st);
  if (rc == CS_OK && e != cudaSuccess) rc = cs_internal_set_error(CS_ERR_CUDA, cudaGetErrorString(e));
  if (singular) *singular = hs;
  return rc;
}
