// Token embedding for sm_100a: the row gather of the forward pass and a deterministic dense
// weight gradient for the backward pass (bf16 rows, fp32 accumulation).
//
// Backward.  dW[v, :] = sum over the tokens t with idx[t] == v of dY[t, :], every row of dW written
// exactly once (rows that no token names are written as zeros, so the caller passes uninitialised
// memory).  No sort over the tokens and no floating-point atomics:
//
//   1. count   cnt[v] += 1 per token (integer atomics: the result does not depend on the order)
//   2. scan    off[v] = exclusive prefix sum of cnt over the vocabulary: sums of 1024 counts, and every
//              CTA adds up the sums in front of its 1024 and scans them (one CTA that walked the whole
//              vocabulary took 280 us for 128256 rows; the two launches take 7)
//   3. fill    bucket[off[v] + k] = t, k handed out by an integer atomic (order inside a bucket varies)
//   4. sum     one CTA per one or two vocabulary rows and 256 of their vectors: the bucket is rank-sorted by
//              token index in shared memory (token indices are distinct, buckets are short), then the rows are
//              added in that order -- the same order, hence the same bits, on every run.  Buckets longer than
//              kMaxSorted tokens are added in bucket order (still correct, order not fixed).  Bound by writing
//              dW where most rows have no token (193 us for 128256 x 4096 and 8192 uniform tokens, 215 us when
//              they are Zipf-distributed; 5.4 TB/s), by the load latency along a bucket where they are long.
//
// Indices outside [0, V) contribute nothing (forward: a zero row) and record kBadArgument in the
// status word.
#include "sm100_common.cuh"

namespace hpb {
namespace emb {

constexpr int kMaxSorted = 1024;

__global__ void embed_fwd_kernel(const int64_t* __restrict__ idx, const uint4* __restrict__ w, uint4* __restrict__ out,
                                 int64_t T, int V, int vec_per_row, int* status) {
  const int64_t total = T * vec_per_row;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t t = i / vec_per_row;
    const int c = static_cast<int>(i - t * vec_per_row);
    const int64_t v = idx[t];
    if (v < 0 || v >= V) {
      if (c == 0) report_error(status, kBadArgument, static_cast<int>(t));
      out[i] = make_uint4(0, 0, 0, 0);
    } else {
      out[i] = w[v * vec_per_row + c];
    }
  }
}

__global__ void embed_count_kernel(const int64_t* __restrict__ idx, int* __restrict__ cnt, int64_t T, int V,
                                   int* status) {
  for (int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; t < T;
       t += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t v = idx[t];
    if (v < 0 || v >= V)
      report_error(status, kBadArgument, static_cast<int>(t));
    else
      atomicAdd(&cnt[v], 1);
  }
}

constexpr int kScan = 1024;      // counts per CTA of the scan

__device__ __forceinline__ int block_sum_1024(int v, int* red) {      // every thread gets the sum
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  v = red[threadIdx.x & 31];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  return v;
}

// part[b] = sum of the 1024 counts of block b
__global__ void __launch_bounds__(kScan) embed_part_kernel(const int* __restrict__ cnt, int* __restrict__ part, int V) {
  __shared__ int red[32];
  const int v = blockIdx.x * kScan + threadIdx.x;
  const int s = block_sum_1024(v < V ? cnt[v] : 0, red);
  if (threadIdx.x == 0) part[blockIdx.x] = s;
}

// off[v] = cursor[v] = sum of cnt[0..v); without `part` the CTA adds up the counts in front of its own
__global__ void __launch_bounds__(kScan) embed_scan_kernel(const int* __restrict__ cnt, const int* __restrict__ part,
                                                           int* __restrict__ off, int* __restrict__ cursor, int V) {
  __shared__ int red[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int before = 0;
  if (part != nullptr) {
    for (int b = threadIdx.x; b < static_cast<int>(blockIdx.x); b += kScan) before += part[b];
  } else {
    for (int b = 0; b < static_cast<int>(blockIdx.x); ++b) before += cnt[b * kScan + threadIdx.x];
  }
  before = block_sum_1024(before, red);
  const int v = blockIdx.x * kScan + threadIdx.x;
  const int n = v < V ? cnt[v] : 0;
  int inc = n;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int up = __shfl_up_sync(0xffffffffu, inc, d);
    if (lane >= d) inc += up;
  }
  if (lane == 31) red[warp] = inc;
  __syncthreads();
  int w = lane < warp ? red[lane] : 0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
  if (v < V) off[v] = cursor[v] = before + w + inc - n;
}

__global__ void embed_fill_kernel(const int64_t* __restrict__ idx, int* __restrict__ cursor, int* __restrict__ bucket,
                                  int64_t T, int V) {
  for (int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; t < T;
       t += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t v = idx[t];
    if (v < 0 || v >= V) continue;
    bucket[atomicAdd(&cursor[v], 1)] = static_cast<int>(t);
  }
}

__device__ __forceinline__ void add_row(float (&acc)[8], const uint4& x) {
  const __nv_bfloat162* xb = reinterpret_cast<const __nv_bfloat162*>(&x);
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float2 f = __bfloat1622float2(xb[e]);
    acc[2 * e] += f.x;
    acc[2 * e + 1] += f.y;
  }
}

// ROWS vocabulary rows per CTA, a `stride` apart: ids follow frequency in most vocabularies, so that
// neighbouring rows have long buckets together.  The 256 threads own one vector each of 256 neighbouring ones.
// CTAS per SM sets the registers: with 8 (32 registers) each token row of a bucket waits for the one before
// it; with 4 (up to 64) eight are in flight, but rows without a token are cleared by half the threads.  Eight
// rows per CTA left a vocabulary of a few thousand rows with too few CTAs (256 rows of 512, 65536 tokens:
// 244 us; 60 now), and with more rows it was no faster than two.
template <int ROWS, int CTAS>
__global__ void __launch_bounds__(256, CTAS) embed_sum_kernel(const uint4* __restrict__ dy, const int* __restrict__ cnt,
                                                        const int* __restrict__ off, const int* __restrict__ bucket,
                                                        uint4* __restrict__ dw, int V, int stride, int vec_per_row,
                                                        int64_t T, int* status) {
  __shared__ int raw[kMaxSorted];
  __shared__ int sorted[kMaxSorted];
  const int c = (blockIdx.z * gridDim.y + blockIdx.y) * 256 + threadIdx.x;
  const bool live = c < vec_per_row;
  for (int v0 = blockIdx.x; v0 < stride; v0 += gridDim.x) {
    int counts[ROWS];
#pragma unroll
    for (int i = 0; i < ROWS; ++i) counts[i] = v0 + i * static_cast<int64_t>(stride) < V ? cnt[v0 + i * stride] : -1;
#pragma unroll
    for (int i = 0; i < ROWS; ++i)
      if (counts[i] == 0 && live) dw[static_cast<int64_t>(v0 + i * stride) * vec_per_row + c] = make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
      const int n = counts[i];
      if (n <= 0) continue;                    // uniform over the CTA
      const int* b = bucket + off[v0 + i * stride];
      const int* order = b;
      bool ok = true;                          // (nothing in the normal build)
      for (int k = 0; k < n; ++k)
        ok = ok && HPB_BOUNDS_OK(b[k] >= 0 && b[k] < T, status, 0x900000 | (blockIdx.x & 0xffff));
      if (!ok) continue;                       // uniform over the CTA
      if (n > 1 && n <= kMaxSorted) {
        __syncthreads();                       // the previous row's readers are done with the arrays
        for (int k = threadIdx.x; k < n; k += 256) raw[k] = b[k];
        __syncthreads();
        for (int k = threadIdx.x; k < n; k += 256) {
          const int t = raw[k];
          int rank = 0;
          for (int j = 0; j < n; ++j) rank += raw[j] < t;
          sorted[rank] = t;
        }
        __syncthreads();
        order = sorted;
      }
      if (!live) continue;
      float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      int k = 0;
      for (; k + 8 <= n; k += 8) {
        uint4 x[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) x[u] = dy[static_cast<int64_t>(order[k + u]) * vec_per_row + c];
#pragma unroll
        for (int u = 0; u < 8; ++u) add_row(acc, x[u]);
      }
      for (; k < n; ++k) add_row(acc, dy[static_cast<int64_t>(order[k]) * vec_per_row + c]);
      uint4 o;
      __nv_bfloat162* ob = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
      for (int e = 0; e < 4; ++e) ob[e] = __floats2bfloat162_rn(acc[2 * e], acc[2 * e + 1]);
      dw[static_cast<int64_t>(v0 + i * stride) * vec_per_row + c] = o;
    }
  }
}

}  // namespace emb
}  // namespace hpb

using namespace hpb;

// out[T, H] = w[idx[T], :]; bf16, H % 8 == 0, 16-byte aligned pointers.
extern "C" int hpb_embedding_fwd(const int64_t* idx, const void* w, void* out, int64_t T, int V, int H, int* status,
                                 int num_sms, cudaStream_t s) {
  if (H <= 0 || H % 8 || V <= 0) return -2;
  if ((reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(out)) & 15) return -2;
  if (T == 0) return 0;
  const int64_t total = T * (H / 8);
  const int64_t want = (total + 255) / 256;
  const int64_t cap = static_cast<int64_t>(num_sms > 0 ? num_sms : 148) * 16;
  emb::embed_fwd_kernel<<<static_cast<unsigned>(want < cap ? want : cap), 256, 0, s>>>(
      idx, reinterpret_cast<const uint4*>(w), reinterpret_cast<uint4*>(out), T, V, H / 8, status);
  return static_cast<int>(cudaGetLastError());
}

// dw[V, H] = scatter-add of dy[T, H] by idx (every row written); scratch: 3 V + T + ceil(V / 1024) ints.
extern "C" int hpb_embedding_bwd(const int64_t* idx, const void* dy, void* dw, int* scratch, int64_t T, int V, int H,
                                 int* status, int num_sms, cudaStream_t s) {
  if (H <= 0 || H % 8 || V <= 0 || T < 0 || T > 0x7fffffff) return -2;
  if ((reinterpret_cast<uintptr_t>(dy) | reinterpret_cast<uintptr_t>(dw)) & 15) return -2;
  int* cnt = scratch;
  int* off = scratch + V;
  int* cursor = scratch + 2ll * V;
  int* bucket = scratch + 3ll * V;
  int* part = bucket + T;
  const int scan_blocks = (V + emb::kScan - 1) / emb::kScan;
  cudaError_t e = cudaMemsetAsync(cnt, 0, sizeof(int) * static_cast<size_t>(V), s);
  if (e != cudaSuccess) return static_cast<int>(e);
  const int sms = num_sms > 0 ? num_sms : 148;
  if (T > 0) {
    const int64_t want = (T + 255) / 256;
    emb::embed_count_kernel<<<static_cast<unsigned>(want < sms * 8 ? want : sms * 8), 256, 0, s>>>(idx, cnt, T, V,
                                                                                                 status);
  }
  // up to 16384 rows a CTA of the scan adds up all counts in front of its own, which is shorter than a launch
  // (1000 rows, 1000 tokens: 14.7 -> 12.6 us)
  const bool direct = scan_blocks <= 16;
  if (!direct) emb::embed_part_kernel<<<scan_blocks, emb::kScan, 0, s>>>(cnt, part, V);
  emb::embed_scan_kernel<<<scan_blocks, emb::kScan, 0, s>>>(cnt, direct ? nullptr : part, off, cursor, V);
  if (T > 0) {
    const int64_t want = (T + 255) / 256;
    emb::embed_fill_kernel<<<static_cast<unsigned>(want < sms * 8 ? want : sms * 8), 256, 0, s>>>(idx, cursor, bucket,
                                                                                                T, V);
  }
  // Long buckets (more than 16 tokens per row on average): one row per CTA, and registers for eight token rows in
  // flight.  Otherwise two rows per CTA and as many CTAs as fit.  Measured, one / two rows: 256 rows of 512, 65536
  // tokens 60 / 93 us; 5000 rows of 512, 100000 tokens 43 / 47; 1024 rows of 4096, 8192 tokens 23.6 / 20.7; 32000 rows
  // of 5120, 8192 tokens 137 / 86.
  const bool dense = T > 16ll * V;
  const int groups = dense ? V : (V + 1) / 2;
  const int slices = (H / 8 + 255) / 256, planes = (slices + 65534) / 65535;
  const dim3 grid(groups < sms * 32 ? groups : sms * 32, (slices + planes - 1) / planes, planes);
  auto kern = dense ? emb::embed_sum_kernel<1, 4> : emb::embed_sum_kernel<2, 8>;
  kern<<<grid, 256, 0, s>>>(reinterpret_cast<const uint4*>(dy), cnt, off, bucket, reinterpret_cast<uint4*>(dw), V, groups,
                            H / 8, T, status);
  return static_cast<int>(cudaGetLastError());
}
