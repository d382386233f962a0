// Row movement of an expert layer whose experts are all on this GPU: which padded row each (token,
// expert) pair gets, the gather into the layout of the grouped GEMMs, and the weighted sum back.
//
// Layout: rows grouped by expert, every group starting at a multiple of `pad` rows; inside a group the
// pairs are in ascending pair order (pair = token * k + slot), so every result is the same from run to
// run.  Rows between a group's end and the next start are written as zeros by the gathers.
//
//   plan    hist     per chunk of 256 pairs: pairs per expert
//           scan     one CTA: per expert, prefix sums over the chunks and the group starts
//           tables   expert of each row block; padding rows named as such
//           place    pair -> row: start + chunk prefix + rank inside the chunk; row -> pair
//   gather  x[T, H] -> xp[rows, H]
//   combine / combine_bwd  the weighted fp32 sum of a token's k rows (one pass, no atomics); its gradient
//
// The last three stream 16-byte vectors and are bound by HBM.  The index_copy / index_select / index_add
// sequence they take the place of moved each row through memory eight times and added bf16 values
// atomically: 8.0 of 17.4 ms for 4096 tokens x 8 of 32 experts, hidden 7168, forward + backward.  With
// these kernels (0.5 ms) and the expert products on CTA pairs the layer takes 8.4-9.6 ms, and 1.90 instead
// of 3.70 ms on 77 tokens.
#include "sm100_common.cuh"

namespace hpb {
namespace moel {

constexpr int CHUNK = 256;

__device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8]) {
  const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = __bfloat1622float2(p[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  uint4 u;
  __nv_bfloat162* p = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) p[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return u;
}

// hist[e, chunk]; *bad != 0 when an id lies outside [0, E) (such a pair is counted nowhere)
__global__ void __launch_bounds__(CHUNK) hist_kernel(const int64_t* __restrict__ idx, int* __restrict__ hist,
                                                     int* __restrict__ bad, int64_t pairs, int E) {
  extern __shared__ int cnt[];
  for (int e = threadIdx.x; e < E; e += CHUNK) cnt[e] = 0;
  __syncthreads();
  const int64_t i = blockIdx.x * static_cast<int64_t>(CHUNK) + threadIdx.x;
  if (i < pairs) {
    const int64_t e = idx[i];
    if (e >= 0 && e < E) atomicAdd(&cnt[e], 1);
    else *bad = 1;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += CHUNK) hist[static_cast<int64_t>(e) * gridDim.x + blockIdx.x] = cnt[e];
}

// hist -> exclusive prefix over the chunks (in place); counts, group starts / ends.  One CTA, one warp
// per expert at a time, lanes over the chunks.
__global__ void __launch_bounds__(1024) scan_kernel(int* __restrict__ hist, int chunks, int E, int pad,
                                                    int* __restrict__ counts, int* __restrict__ starts,
                                                    int* __restrict__ ends) {
  extern __shared__ int sm[];       // padded sizes, then starts
  const int lane = threadIdx.x & 31;
  for (int e = threadIdx.x >> 5; e < E; e += blockDim.x >> 5) {
    int* h = hist + static_cast<int64_t>(e) * chunks;
    int run = 0;
    for (int c0 = 0; c0 < chunks; c0 += 32) {
      const int n = c0 + lane < chunks ? h[c0 + lane] : 0;
      int inc = n;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, inc, d);
        if (lane >= d) inc += up;
      }
      if (c0 + lane < chunks) h[c0 + lane] = run + inc - n;
      run += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (lane == 0) {
      counts[e] = run;
      sm[e] = (run + pad - 1) / pad * pad;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int off = 0;
    for (int e = 0; e < E; ++e) {
      const int n = sm[e];
      sm[e] = off;
      off += n;
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    starts[e] = sm[e];
    ends[e] = sm[e] + counts[e];
  }
}

// block_group[b] = expert of rows [b * pad, (b + 1) * pad); row_pair of the padding rows = -1
__global__ void tables_kernel(const int* __restrict__ starts, const int* __restrict__ ends, int E, int pad,
                              int* __restrict__ block_group, int* __restrict__ row_pair) {
  const int e = blockIdx.x;
  const int s = starts[e], n = ends[e];
  const int stop = s + (n - s + pad - 1) / pad * pad;
  for (int b = s / pad + threadIdx.x; b < stop / pad; b += blockDim.x) block_group[b] = e;
  for (int r = n + threadIdx.x; r < stop; r += blockDim.x) row_pair[r] = -1;
}

__global__ void __launch_bounds__(CHUNK) place_kernel(const int64_t* __restrict__ idx, const int* __restrict__ hist,
                                                      const int* __restrict__ starts, int* __restrict__ pos,
                                                      int* __restrict__ row_pair, int64_t pairs, int E, int64_t rows,
                                                      int* status) {
  __shared__ int ids[CHUNK];
  const int64_t i = blockIdx.x * static_cast<int64_t>(CHUNK) + threadIdx.x;
  const int e = i < pairs ? static_cast<int>(idx[i]) : -1;
  ids[threadIdx.x] = e;
  __syncthreads();
  if (e < 0 || e >= E) return;
  int rank = 0;
  for (int j = 0; j < threadIdx.x; ++j) rank += ids[j] == e;
  const int r = starts[e] + hist[static_cast<int64_t>(e) * gridDim.x + blockIdx.x] + rank;
  pos[i] = r;
  if (HPB_BOUNDS_OK(r >= 0 && r < rows, status, 0x800000 | e)) row_pair[r] = static_cast<int>(i);
}

// xp[row] = x[pair / k], zeros in padding rows; one row per blockIdx.x
__global__ void __launch_bounds__(256) gather_kernel(const uint4* __restrict__ x, const int* __restrict__ row_pair,
                                                     uint4* __restrict__ xp, int k, int vecs, int64_t pairs,
                                                     int* status) {
  const int64_t row = blockIdx.x;
  int pair = row_pair[row];
  if (!HPB_BOUNDS_OK(pair < pairs, status, 0x810000 | (blockIdx.x & 0xffff))) pair = -1;
  uint4* dst = xp + row * vecs;
  if (pair < 0) {
    for (int c = threadIdx.x; c < vecs; c += 256) dst[c] = make_uint4(0, 0, 0, 0);
    return;
  }
  const uint4* src = x + static_cast<int64_t>(pair / k) * vecs;
  for (int c0 = threadIdx.x; c0 < vecs; c0 += 4 * 256) {     // four vectors in flight per thread
    uint4 v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (c0 + u * 256 < vecs) v[u] = src[c0 + u * 256];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (c0 + u * 256 < vecs) dst[c0 + u * 256] = v[u];
  }
}

// out[t] = sum_j w[t, j] * yp[pos[t, j]] (w == nullptr: 1), fp32 sums; one token per blockIdx.x.
// Four rows are in flight per thread.
__global__ void __launch_bounds__(256) combine_kernel(const uint4* __restrict__ yp, const int* __restrict__ pos,
                                                      const float* __restrict__ w, uint4* __restrict__ out, int k,
                                                      int vecs, int64_t rows, int* status) {
  const int64_t t = blockIdx.x;
  const int* p = pos + t * k;
  for (int j = 0; j < k; ++j)      // (nothing in the normal build)
    if (!HPB_BOUNDS_OK(p[j] >= 0 && p[j] < rows, status, 0x820000 | (blockIdx.x & 0xffff))) return;
  for (int c = threadIdx.x; c < vecs; c += 256) {
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int j0 = 0; j0 < k; j0 += 4) {
      uint4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (j0 + u < k) v[u] = yp[static_cast<int64_t>(p[j0 + u]) * vecs + c];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (j0 + u < k) {
          const float s = w != nullptr ? w[t * k + j0 + u] : 1.f;
          float f[8];
          unpack8(v[u], f);
#pragma unroll
          for (int e = 0; e < 8; ++e) acc[e] += s * f[e];
        }
      }
    }
    out[t * vecs + c] = pack8(acc);
  }
}

// Gradient of the combine: dyp[row] = w[pair] * dout[token] (zeros in padding rows) and, with yp,
// dw[pair] = dout[token] . yp[row]; one row per blockIdx.x.
__global__ void __launch_bounds__(256) combine_bwd_kernel(const uint4* __restrict__ dout, const int* __restrict__ row_pair,
                                                          const float* __restrict__ w, const uint4* __restrict__ yp,
                                                          uint4* __restrict__ dyp, float* __restrict__ dw, int k,
                                                          int vecs, int64_t pairs, int* status) {
  __shared__ float red[8];
  const int64_t row = blockIdx.x;
  int pair = row_pair[row];
  if (!HPB_BOUNDS_OK(pair < pairs, status, 0x830000 | (blockIdx.x & 0xffff))) pair = -1;
  uint4* dst = dyp + row * vecs;
  if (pair < 0) {
    for (int c = threadIdx.x; c < vecs; c += 256) dst[c] = make_uint4(0, 0, 0, 0);
    return;
  }
  const uint4* src = dout + static_cast<int64_t>(pair / k) * vecs;
  const float s = w[pair];
  float dot = 0.f;
  for (int c0 = threadIdx.x; c0 < vecs; c0 += 4 * 256) {
    uint4 gv[4], yv[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (c0 + u * 256 < vecs) {
        gv[u] = src[c0 + u * 256];
        if (yp != nullptr) yv[u] = yp[row * vecs + c0 + u * 256];
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (c0 + u * 256 < vecs) {
        float g[8], o[8];
        unpack8(gv[u], g);
        if (yp != nullptr) {
          float y[8];
          unpack8(yv[u], y);
#pragma unroll
          for (int e = 0; e < 8; ++e) dot += g[e] * y[e];
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = s * g[e];
        dst[c0 + u * 256] = pack8(o);
      }
    }
  }
  if (dw == nullptr) return;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = dot;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) t += red[i];
    dw[pair] = t;
  }
}

}  // namespace moel
}  // namespace hpb

using namespace hpb::moel;

// First half of the plan: counts / starts / ends [E]; counts[E] becomes non-zero when an expert id is out
// of range.  E <= 8192; hist: E words for every 256 pairs.
extern "C" int hpb_moe_count(const int64_t* idx, int* hist, int* counts, int* starts, int* ends, int64_t pairs, int E,
                             int pad, cudaStream_t s) {
  if (pairs <= 0 || pairs > 0x3fffffff || E <= 0 || E > 8192 || pad <= 0) return -2;
  const int chunks = static_cast<int>((pairs + CHUNK - 1) / CHUNK);
  cudaError_t e = cudaMemsetAsync(counts + E, 0, sizeof(int), s);
  if (e != cudaSuccess) return static_cast<int>(e);
  hist_kernel<<<chunks, CHUNK, E * sizeof(int), s>>>(idx, hist, counts + E, pairs, E);
  scan_kernel<<<1, E < 32 ? E * 32 : 1024, E * sizeof(int), s>>>(hist, chunks, E, pad, counts, starts,
                                                                              ends);
  return static_cast<int>(cudaGetLastError());
}

// Second half (every id in range): block_group [rows / pad], row_pair [rows], pos [pairs].
extern "C" int hpb_moe_place(const int64_t* idx, const int* hist, const int* starts, const int* ends, int* block_group,
                             int* row_pair, int* pos, int64_t pairs, int E, int pad, int64_t rows, int* status,
                             cudaStream_t s) {
  if (pairs <= 0 || pairs > 0x3fffffff || E <= 0 || pad <= 0) return -2;
  tables_kernel<<<E, 128, 0, s>>>(starts, ends, E, pad, block_group, row_pair);
  place_kernel<<<static_cast<unsigned>((pairs + CHUNK - 1) / CHUNK), CHUNK, 0, s>>>(idx, hist, starts, pos, row_pair,
                                                                                 pairs, E, rows, status);
  return static_cast<int>(cudaGetLastError());
}

static bool aligned16(const void* a, const void* b, const void* c = nullptr) {
  return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c)) & 15) == 0;
}

// (rows / pairs and status below: what the index checks of the debug build compare with and report to)
extern "C" int hpb_moe_gather(const void* x, const int* row_pair, void* xp, int64_t rows, int k, int H, int64_t pairs,
                              int* status, cudaStream_t s) {
  if (H % 8 || k <= 0 || rows > 0x7fffffff || !aligned16(x, xp)) return -2;
  if (rows <= 0) return 0;
  gather_kernel<<<static_cast<unsigned>(rows), 256, 0, s>>>(reinterpret_cast<const uint4*>(x), row_pair,
                                                            reinterpret_cast<uint4*>(xp), k, H / 8, pairs, status);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int hpb_moe_combine(const void* yp, const int* pos, const float* w, void* out, int64_t T, int k, int H,
                               int64_t rows, int* status, cudaStream_t s) {
  if (H % 8 || k <= 0 || T > 0x7fffffff || !aligned16(yp, out)) return -2;
  if (T <= 0) return 0;
  combine_kernel<<<static_cast<unsigned>(T), 256, 0, s>>>(reinterpret_cast<const uint4*>(yp), pos, w,
                                                          reinterpret_cast<uint4*>(out), k, H / 8, rows, status);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int hpb_moe_combine_bwd(const void* dout, const int* row_pair, const float* w, const void* yp, void* dyp,
                                   float* dw, int64_t rows, int k, int H, int64_t pairs, int* status, cudaStream_t s) {
  if (H % 8 || k <= 0 || rows > 0x7fffffff || !aligned16(dout, dyp, yp)) return -2;
  if (rows <= 0) return 0;
  combine_bwd_kernel<<<static_cast<unsigned>(rows), 256, 0, s>>>(
      reinterpret_cast<const uint4*>(dout), row_pair, w, reinterpret_cast<const uint4*>(yp),
      reinterpret_cast<uint4*>(dyp), dw, k, H / 8, pairs, status);
  return static_cast<int>(cudaGetLastError());
}
