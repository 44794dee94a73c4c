// Solution files of a whole batch as text, formatted on the GPU.
//
// The reference writes each solution with a Python loop over every value
// ('{}'.format, BVPDAEReadWriteData.py:337-364).  Here a file is cut into
// chunks of kChunk values, a CTA each: the length of every value's shortest
// round-trip text (cs_dtoa.h), summed per chunk (k_text_sizes); the chunks'
// offsets (k_text_scan); and the text itself, assembled in shared memory and
// copied out in whole words (k_text_write).  Digits are generated again for the
// text: at about 100 integer instructions a value that costs less than keeping
// 25 bytes per value between the passes did, and it needs no scratch in
// proportion to the values.  The text is byte for byte the reference's file.
//
// Measured (512 instances, 3.2 M values, 62 MB of text): values and sizes
// 3.04 ms -> 0.11 ms, writing 3.6 ms -> 0.23 ms; with both calls of a caller that
// sizes first and the copy to page-locked memory 7.7 ms -> 0.87 ms.
#include <cuda_runtime.h>

#include <algorithm>
#include <string>
#include <vector>

#include "cs_dtoa.h"
#include "cs_gb300.h"
#include "cs_text.h"

int cs_internal_set_error(int code, const char* msg);

namespace {

// decimal text of a non-negative int; returns the length
__host__ __device__ inline int cs_itoa(int v, char* out) {
  char tmp[12];
  int n = 0;
  do {
    tmp[n++] = (char)('0' + v % 10);
    v /= 10;
  } while (v > 0);
  for (int i = 0; i < n; ++i) out[i] = tmp[n - 1 - i];
  return n;
}

__host__ __device__ inline int cs_itoa_len(int v) {
  int n = 1;
  while (v >= 10) {
    v /= 10;
    ++n;
  }
  return n;
}

// labels of a file: "nt:\n<N>\nt:\n", "\nny:\n<ny>\ny:\n", "nz:\n<nz>\nz:\n", "np:\n<np>\np:\n"
__host__ __device__ inline int cs_label(int which, int v, char* out) {
  const char* pre[4] = {"nt:\n", "\nny:\n", "nz:\n", "np:\n"};
  const char* post[4] = {"\nt:\n", "\ny:\n", "\nz:\n", "\np:\n"};
  int p = 0;
  for (const char* c = pre[which]; *c; ++c) out[p++] = *c;
  p += cs_itoa(v, out + p);
  for (const char* c = post[which]; *c; ++c) out[p++] = *c;
  return p;
}

__host__ __device__ inline int cs_label_len(int which, int v) { return (which == 1 ? 9 : 8) + cs_itoa_len(v); }

struct CsTextSrc {
  const double *t, *y, *z, *p;
  int B, ny, nz, np;
  const int *N, *off;
  const long long* cpre;  // [B+1] chunks before each instance
};

constexpr int kThreads = 256, kPer = 4, kChunk = kThreads * kPer;
constexpr int kStage = kChunk * (CS_DTOA_MAX + 2) + 160;  // a chunk's text, or it goes straight out

// the chunk's instance and its values [e0, e1) of the instance's list: t (N),
// y (N x ny), z (N x nz), p (np)
struct CsChunk {
  int b, N, o;
  long long e0, e1, total, by, bz, bp;  // sections start at 0, by, bz, bp
};

__device__ inline CsChunk cs_chunk(const CsTextSrc& s, long long c) {
  int lo = 0, hi = s.B - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (s.cpre[mid] <= c) lo = mid; else hi = mid - 1;
  }
  CsChunk k;
  k.b = lo;
  k.N = s.N[lo];
  k.o = s.off[lo];
  k.by = k.N;
  k.bz = k.by + (long long)k.N * s.ny;
  k.bp = k.bz + (long long)k.N * s.nz;
  k.total = k.bp + s.np;
  k.e0 = (c - s.cpre[lo]) * kChunk;
  k.e1 = min(k.total, k.e0 + kChunk);
  return k;
}

__device__ inline double cs_text_value(const CsTextSrc& s, const CsChunk& k, long long e) {
  if (e < k.by) return s.t[k.o + e];
  if (e < k.bz) return s.y[(long long)k.o * s.ny + (e - k.by)];
  if (e < k.bp) return s.z[(long long)k.o * s.nz + (e - k.bz)];
  return s.p[(long long)k.b * s.np + (e - k.bp)];
}

// bytes of the labels in front of value e (e = total: after the last one)
__device__ inline long long cs_insert_len(const CsTextSrc& s, const CsChunk& k, long long e) {
  long long n = 0;
  if (e == 0) n += cs_label_len(0, k.N);
  if (e == k.by) n += cs_label_len(1, s.ny);
  if (e == k.bz) n += cs_label_len(2, s.nz) + (s.nz == 0 ? k.N : 0);  // a row without values is its "\n"
  if (e == k.bp) n += cs_label_len(3, s.np);
  return n;
}
__device__ inline char* cs_insert(const CsTextSrc& s, const CsChunk& k, long long e, char* d) {
  if (e == 0) d += cs_label(0, k.N, d);
  if (e == k.by) d += cs_label(1, s.ny, d);
  if (e == k.bz) {
    d += cs_label(2, s.nz, d);
    if (s.nz == 0)
      for (int i = 0; i < k.N; ++i) *d++ = '\n';
  }
  if (e == k.bp) d += cs_label(3, s.np, d);
  return d;
}

// whether value e ends a row of y or z
__device__ inline bool cs_row_end(const CsTextSrc& s, const CsChunk& k, long long e) {
  if (e < k.by || e >= k.bp) return false;
  if (e < k.bz) return (unsigned)(e - k.by) % (unsigned)s.ny == (unsigned)(s.ny - 1);
  return (unsigned)(e - k.bz) % (unsigned)s.nz == (unsigned)(s.nz - 1);
}

// plans and bytes of this thread's kPer consecutive values
__device__ inline int cs_plan(const CsTextSrc& s, const CsChunk& k, CsText (&t)[kPer]) {
  int n = 0;
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const long long e = k.e0 + (long long)threadIdx.x * kPer + j;
    t[j].len = -1;
    if (e < k.e1) {
      cs_text_plan(cs_text_value(s, k, e), &t[j]);
      n += t[j].len + 1 + (cs_row_end(s, k, e) ? 1 : 0);
    }
  }
  return n;
}

// bytes of the labels among this thread's values
__device__ inline long long cs_plan_labels(const CsTextSrc& s, const CsChunk& k) {
  const long long a = k.e0 + (long long)threadIdx.x * kPer, z = min(k.e1, a + kPer);
  long long n = 0;
  for (long long e = a; e < z; ++e) n += cs_insert_len(s, k, e);
  if (a < k.e1 && z == k.total) n += cs_insert_len(s, k, k.total);
  return n;
}

// exclusive prefix sum over the CTA (at most 1024 threads); *total: its sum
__device__ long long cs_block_exscan(long long v, long long* sh, long long* total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  long long x = v;
  for (int o = 1; o < 32; o <<= 1) {
    const long long y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) sh[w] = x;
  __syncthreads();
  if (w == 0) {
    long long q = lane < nw ? sh[lane] : 0;
    for (int o = 1; o < 32; o <<= 1) {
      const long long y = __shfl_up_sync(0xffffffffu, q, o);
      if (lane >= o) q += y;
    }
    if (lane < nw) sh[lane] = q;  // inclusive sums of the warps
    if (lane == 31) sh[32] = q;
  }
  __syncthreads();
  const long long before = (w > 0 ? sh[w - 1] : 0) + x - v;
  *total = sh[32];
  __syncthreads();
  return before;
}

__global__ void __launch_bounds__(kThreads) k_text_sizes(CsTextSrc s, long long chunks, long long* csize) {
  __shared__ long long sh[33];
  for (long long c = blockIdx.x; c < chunks; c += gridDim.x) {
    const CsChunk k = cs_chunk(s, c);
    CsText t[kPer];
    long long tot;
    const long long n = cs_plan(s, k, t) + cs_plan_labels(s, k);
    cs_block_exscan(n, sh, &tot);
    if (threadIdx.x == 0) csize[c] = tot;
  }
}

// csize [chunks] -> offsets in place (csize[chunks]: all of it), and the first
// byte of every file
__global__ void __launch_bounds__(1024) k_text_scan(int B, const long long* cpre, long long chunks, long long* csize,
                                                    long long* offset) {
  __shared__ long long sh[33];
  long long at = 0;
  for (long long c0 = 0; c0 < chunks; c0 += 1024) {
    const long long c = c0 + threadIdx.x;
    long long tot;
    const long long v = c < chunks ? csize[c] : 0;
    const long long x = cs_block_exscan(v, sh, &tot);
    if (c < chunks) csize[c] = at + x;
    at += tot;
  }
  if (threadIdx.x == 0) csize[chunks] = at;
  __syncthreads();
  for (int b = threadIdx.x; b <= B; b += 1024) offset[b] = csize[cpre[b]];
}

__global__ void __launch_bounds__(kThreads) k_text_write(CsTextSrc s, long long chunks, const long long* coff, char* out) {
  __shared__ long long sh[33];
  __shared__ __align__(16) char stage[kStage + 16];
  for (long long c = blockIdx.x; c < chunks; c += gridDim.x) {
    const CsChunk k = cs_chunk(s, c);
    CsText t[kPer];
    long long tot;
    const long long n = cs_plan(s, k, t) + cs_plan_labels(s, k);
    long long pos = cs_block_exscan(n, sh, &tot);
    char* base = out + coff[c];
    const bool staged = tot <= kStage;
    const int lead = (int)((size_t)base & 15);  // the stage keeps the output's alignment
    char* d = (staged ? stage + lead : base) + pos;
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      const long long e = k.e0 + (long long)threadIdx.x * kPer + j;
      if (e < k.e1) {
        d = cs_insert(s, k, e, d);
        cs_text_put(t[j], d);
        d += t[j].len;
        *d++ = ' ';
        if (cs_row_end(s, k, e)) *d++ = '\n';
        if (e + 1 == k.total) cs_insert(s, k, k.total, d);
      }
    }
    __syncthreads();
    if (staged) {
      // bytes to the first 16-byte boundary, whole words, the rest
      const int end = lead + (int)tot, w0 = (lead + 15) >> 4, w1 = end >> 4;
      char* al = base - lead;
      for (int w = w0 + threadIdx.x; w < w1; w += kThreads)
        reinterpret_cast<uint4*>(al)[w] = reinterpret_cast<const uint4*>(stage)[w];
      for (int i = lead + threadIdx.x; i < min(end, 16 * w0); i += kThreads) al[i] = stage[i];
      for (int i = max(lead, 16 * max(w0, w1)) + threadIdx.x; i < end; i += kThreads) al[i] = stage[i];
    }
    __syncthreads();
  }
}

}  // namespace

extern "C" int cs_format_double(double v, char* out) {
  if (!out) {
    cs_internal_set_error(CS_ERR_INVALID, "cs_format_double: null output");
    return -1;
  }
  const int n = cs_format_double_text(v, out);
  out[n] = 0;
  return n;
}

#define CS_TRYC(call, what)                                                                          \
  do {                                                                                               \
    cudaError_t e_ = (call);                                                                         \
    if (e_ != cudaSuccess) return cs_internal_set_error(CS_ERR_CUDA, (std::string(what) + ": " + cudaGetErrorString(e_)).c_str()); \
  } while (0)

static void scratch_drop(CsTextScratch* s, int i) {
  cudaFree(s->p[i]);
  s->p[i] = nullptr;
  s->bytes[i] = 0;
}

void cs_text_scratch_free(CsTextScratch* s) {
  for (int i = 0; i < 2; ++i) scratch_drop(s, i);
}

static int scratch_grow(CsTextScratch* s, int i, size_t bytes) {
  if (s->bytes[i] >= bytes) return CS_OK;
  scratch_drop(s, i);
  CS_TRYC(cudaMalloc(&s->p[i], bytes), "cs_format_solutions: scratch");
  s->bytes[i] = bytes;
  return CS_OK;
}

// The text buffer stays with the batch up to this size (as the library's pool
// keeps); a larger one goes back to the device before the call returns.  Below it
// an allocation would cost as much as the writing: 62 MB of text take 0.9 ms.
static const size_t kTextKeep = 256ull << 20;

int cs_text_files(const CsTextArgs& a, char* out, long long cap, long long* offsets) {
  std::vector<long long> pre(a.B + 1);
  pre[0] = 0;
  for (int b = 0; b < a.B; ++b) {
    const long long values = (long long)a.hN[b] * (1 + a.ny + a.nz) + a.np;
    pre[b + 1] = pre[b] + (values + kChunk - 1) / kChunk;
  }
  const long long chunks = pre[a.B];
  // index [B + 1] | file offsets [B + 1] | chunk sizes, then offsets [chunks + 1]
  int rc = scratch_grow(a.scratch, 0, (size_t)(2 * (a.B + 1) + chunks + 1) * sizeof(long long));
  if (rc != CS_OK) return rc;
  long long* cpre = (long long*)a.scratch->p[0];
  long long* foff = cpre + a.B + 1;
  long long* coff = foff + a.B + 1;
  CsTextSrc s;
  s.t = a.t;
  s.y = a.y;
  s.z = a.z;
  s.p = a.p;
  s.B = a.B;
  s.ny = a.ny;
  s.nz = a.nz;
  s.np = a.np;
  s.N = a.dN;
  s.off = a.doff;
  s.cpre = cpre;
  cudaStream_t st = (cudaStream_t)a.stream;
  // numbers outside the fast range keep four ~160-byte integers per thread (a
  // 1.2 KB frame): make sure this context's per-thread stack holds it
  size_t stack = 0;
  CS_TRYC(cudaDeviceGetLimit(&stack, cudaLimitStackSize), "cs_format_solutions: stack limit");
  if (stack < 2048) CS_TRYC(cudaDeviceSetLimit(cudaLimitStackSize, 2048), "cs_format_solutions: stack limit");
  CS_TRYC(cudaMemcpyAsync(cpre, pre.data(), pre.size() * sizeof(long long), cudaMemcpyHostToDevice, st),
          "cs_format_solutions: index");
  const unsigned grid = (unsigned)std::min<long long>(chunks, 152ll * 64);
  k_text_sizes<<<grid, kThreads, 0, st>>>(s, chunks, coff);
  CS_TRYC(cudaGetLastError(), "k_text_sizes");
  k_text_scan<<<1, 1024, 0, st>>>(a.B, cpre, chunks, coff, foff);
  CS_TRYC(cudaGetLastError(), "k_text_scan");
  CS_TRYC(cudaMemcpyAsync(offsets, foff, (size_t)(a.B + 1) * sizeof(long long), cudaMemcpyDeviceToHost, st),
          "cs_format_solutions: offsets");
  CS_TRYC(cudaStreamSynchronize(st), "cs_format_solutions");
  const long long total = offsets[a.B];
  if (!out) return CS_OK;
  if (cap < total) return cs_internal_set_error(CS_ERR_INVALID, "cs_format_solutions: output buffer too small");
  rc = scratch_grow(a.scratch, 1, (size_t)std::max(total, 1ll));
  if (rc != CS_OK) return rc;
  k_text_write<<<grid, kThreads, 0, st>>>(s, chunks, coff, (char*)a.scratch->p[1]);
  CS_TRYC(cudaGetLastError(), "k_text_write");
  CS_TRYC(cudaMemcpyAsync(out, a.scratch->p[1], (size_t)total, cudaMemcpyDeviceToHost, st), "cs_format_solutions: text to host");
  CS_TRYC(cudaStreamSynchronize(st), "cs_format_solutions");
  if (a.scratch->bytes[1] > kTextKeep) scratch_drop(a.scratch, 1);
  return CS_OK;
}
