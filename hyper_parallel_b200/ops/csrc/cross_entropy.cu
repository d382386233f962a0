// Fused softmax cross entropy, forward and backward in one kernel (sm_100a).
//
// Reads logits[row, :V] (bf16), writes loss[row] (fp32) and overwrites the row IN PLACE with
// d(loss_sum * grad_scale)/dlogits = (softmax - onehot) * grad_scale.  Rows with target < 0 or >= V get
// zero loss and gradient.
//
//   ce_reg_kernel     up to 8192 logits: 128 threads hold the row in registers
//   ce_stream_kernel  longer rows: persistent CTAs, two per SM.  A producer warp streams the row twice
//                     through a ring of 32 KB bulk copies -- from HBM for the running maximum and sum of
//                     exponentials, from L2 (296 rows of 256 KB are in flight at 128256 logits, 76 MB) for
//                     the gradient -- and runs ahead into the next row, so that copies never wait for the
//                     reductions between the passes.
//
// Bound by HBM: one read and one write of every logit.  The gradient is stored evict-first, which keeps the
// rows that are still to be read a second time in L2 (without: 23 % more DRAM reads, 921 us).  Measured, 8192
// rows of 128256 / 32000 and 512 of 128256: 852 / 191 / 58 us (4.9 / 5.5 / 4.5 TB/s); the three-pass kernel with
// plain loads that this one replaces took 1036 / 302 / 83 us, and 1593 instead of 964 us behind a GEMM, at the
// lower clock that the power limit leaves.
#include "sm100_common.cuh"

namespace hpb {

typedef __nv_bfloat16 bf16;
typedef __nv_bfloat162 bf162;

namespace {

__device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8]) {
  const bf162* p = reinterpret_cast<const bf162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = __bfloat1622float2(p[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  uint4 u;
  bf162* p = reinterpret_cast<bf162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) p[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return u;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
template <int THREADS>
__device__ __forceinline__ void consumer_sync() {
  asm volatile("bar.sync 1, %0;" ::"n"(THREADS) : "memory");
}
// Reductions over the first THREADS threads; `red` holds 32 floats and is free again after the next one.
template <int THREADS>
__device__ __forceinline__ float group_max(float v, float* red) {
  const int lane = threadIdx.x & 31;
  v = warp_max(v);
  if (lane == 0) red[threadIdx.x >> 5] = v;
  consumer_sync<THREADS>();
  return warp_max(lane < THREADS / 32 ? red[lane] : -INFINITY);
}
template <int THREADS>
__device__ __forceinline__ float group_sum(float v, float* red) {
  const int lane = threadIdx.x & 31;
  v = warp_sum(v);
  if (lane == 0) red[threadIdx.x >> 5] = v;
  consumer_sync<THREADS>();
  return warp_sum(lane < THREADS / 32 ? red[lane] : 0.f);
}
__device__ __forceinline__ float2 ce_add2(float2 a, float2 b) {
  unsigned long long d;
  asm("add.rn.f32x2 %0, %1, %2;"
      : "=l"(d)
      : "l"(*reinterpret_cast<unsigned long long*>(&a)), "l"(*reinterpret_cast<unsigned long long*>(&b)));
  return *reinterpret_cast<float2*>(&d);
}
__device__ __forceinline__ float2 ce_mul2(float2 a, float2 b) {
  unsigned long long d;
  asm("mul.rn.f32x2 %0, %1, %2;"
      : "=l"(d)
      : "l"(*reinterpret_cast<unsigned long long*>(&a)), "l"(*reinterpret_cast<unsigned long long*>(&b)));
  return *reinterpret_cast<float2*>(&d);
}
__device__ __forceinline__ float ce_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

struct CeRow {
  bf16* lr;
  uint4* lv;
  int nvec, tail, tgt_vec;     // tgt_vec: vector of the target, -1 without one
  int64_t tgt;
  bool valid;
  float at_target;     // thread 0 only; read before anything is overwritten
};
__device__ __forceinline__ CeRow ce_row(bf16* logits, const int64_t* target, int64_t row, int V, int64_t ld) {
  CeRow r;
  r.lr = logits + row * ld;
  r.lv = reinterpret_cast<uint4*>(r.lr);
  r.nvec = V >> 3;
  r.tail = V - r.nvec * 8;
  r.tgt = target[row];
  r.valid = r.tgt >= 0 && r.tgt < V;
  r.tgt_vec = r.valid ? static_cast<int>(r.tgt >> 3) : -1;
  r.at_target = threadIdx.x == 0 && r.valid ? __bfloat162float(r.lr[r.tgt]) : 0.f;
  return r;
}
// e^(f - shift): the difference first, so that a row at the type's lowest value does not overflow.
constexpr float kLog2e = 1.4426950408889634f;
__device__ __forceinline__ float ce_exp(float f, float shift) { return ce_ex2((f - shift) * kLog2e); }

__device__ __forceinline__ bf162 ce_vec_max(const uint4& v) {
  const bf162* p = reinterpret_cast<const bf162*>(&v);
  return __hmax2(__hmax2(p[0], p[1]), __hmax2(p[2], p[3]));
}
__device__ __forceinline__ float ce_max(bf162 a) { return fmaxf(__low2float(a), __high2float(a)); }

__device__ __forceinline__ float2 ce_add_exps(float2 s, const uint4& v, float shift) {
  const float2 l2e = make_float2(kLog2e, kLog2e), ns = make_float2(-shift, -shift);
  float f[8];
  unpack8(v, f);
#pragma unroll
  for (int e = 0; e < 8; e += 2) {
    float2 x = ce_mul2(ce_add2(make_float2(f[e], f[e + 1]), ns), l2e);
    x.x = ce_ex2(x.x);
    x.y = ce_ex2(x.y);
    s = ce_add2(s, x);
  }
  return s;
}
// Gradient of vector c of the row, written in place.  The target's logit is patched behind the vector store
// (a conditional on one of the eight values would push all of them through local memory).
__device__ __forceinline__ void ce_grad(const uint4& v, const CeRow& r, int c, float lse, float gs) {
  const float2 l2e = make_float2(kLog2e, kLog2e), nl = make_float2(-lse, -lse), g2 = make_float2(gs, gs);
  float f[8];
  unpack8(v, f);
#pragma unroll
  for (int e = 0; e < 8; e += 2) {
    const float2 x = ce_mul2(ce_add2(make_float2(f[e], f[e + 1]), nl), l2e);
    f[e] = ce_ex2(x.x);
    f[e + 1] = ce_ex2(x.y);
  }
#pragma unroll
  for (int e = 0; e < 8; e += 2) {
    const float2 x = ce_mul2(make_float2(f[e], f[e + 1]), g2);
    f[e] = x.x;
    f[e + 1] = x.y;
  }
  __stcs(&r.lv[c], pack8(f));
  if (c == r.tgt_vec) {
    const int e = static_cast<int>(r.tgt & 7);
    const uint32_t w = e & 4 ? (e & 2 ? v.w : v.z) : (e & 2 ? v.y : v.x);
    const float ft = __uint_as_float(e & 1 ? w & 0xffff0000u : w << 16);
    r.lr[r.tgt] = __float2bfloat16((ce_exp(ft, lse) - 1.f) * gs);
  }
}
// The last V % 8 logits, one per thread.
__device__ __forceinline__ void ce_tail_grad(const CeRow& r, float ft, float lse, float gs) {
  const int c = r.nvec * 8 + threadIdx.x;
  float pr = ce_exp(ft, lse);
  if (c == r.tgt) pr -= 1.f;
  r.lr[c] = __float2bfloat16(pr * gs);
}

// Keeps the packed vectors packed: without it the compiler holds their unpacked form across the phases
// (twice the registers) and spills.
template <int NV>
__device__ __forceinline__ void ce_pin(uint4 (&v)[NV]) {
#pragma unroll
  for (int i = 0; i < NV; ++i) asm volatile("" : "+r"(v[i].x), "+r"(v[i].y), "+r"(v[i].z), "+r"(v[i].w));
}

template <int THREADS, int NV>
__global__ void __launch_bounds__(THREADS)
ce_reg_kernel(bf16* __restrict__ logits, const int64_t* __restrict__ target, float* __restrict__ loss, int V,
              int64_t ld, float grad_scale) {
  __shared__ float red[64];
  const CeRow r = ce_row(logits, target, blockIdx.x, V, ld);
  const bool has_tail = static_cast<int>(threadIdx.x) < r.tail;
  uint4 v[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = i * THREADS + threadIdx.x;
    if (c < r.nvec) v[i] = r.lv[c];
    else v[i] = make_uint4(0xff80ff80u, 0xff80ff80u, 0xff80ff80u, 0xff80ff80u);      // -inf
  }
  const float ft = has_tail ? __bfloat162float(r.lr[r.nvec * 8 + threadIdx.x]) : -INFINITY;
  bf162 m2 = ce_vec_max(v[0]);
#pragma unroll
  for (int i = 1; i < NV; ++i) m2 = __hmax2(m2, ce_vec_max(v[i]));
  const float mx = group_max<THREADS>(fmaxf(ft, ce_max(m2)), red);
  ce_pin(v);
  float2 s2 = make_float2(has_tail ? ce_exp(ft, mx) : 0.f, 0.f);
#pragma unroll
  for (int i = 0; i < NV; ++i)
    if (i * THREADS + static_cast<int>(threadIdx.x) < r.nvec) s2 = ce_add_exps(s2, v[i], mx);
  const float lse = mx + __logf(group_sum<THREADS>(s2.x + s2.y, red + 32));
  if (threadIdx.x == 0) loss[blockIdx.x] = r.valid ? lse - r.at_target : 0.f;
  ce_pin(v);
  const float gs = r.valid ? grad_scale : 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = i * THREADS + threadIdx.x;
    if (c < r.nvec) ce_grad(v[i], r, c, lse, gs);
  }
  if (has_tail) ce_tail_grad(r, ft, lse, gs);
}


constexpr int CS_THREADS = 512;                   // consumers; one producer warp on top
constexpr int CS_VECS = 2048;                     // 16-byte vectors per stage
constexpr int CS_STAGES = 3;
constexpr int CS_SMEM = CS_STAGES * CS_VECS * 16 + 128;
constexpr int CS_PER_THREAD = CS_VECS / CS_THREADS;

__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

__global__ void __launch_bounds__(CS_THREADS + 32, 2)
ce_stream_kernel(bf16* __restrict__ logits, const int64_t* __restrict__ target, float* __restrict__ loss, int64_t T,
                 int V, int64_t ld, float grad_scale, int* status) {
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ float red[64];
  __shared__ int abort_word;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + CS_STAGES * CS_VECS * 16);
  uint64_t* empty = full + CS_STAGES;
  volatile int* abort_flag = &abort_word;
  const int lane = threadIdx.x & 31;
  const int nvec = V >> 3, chunks = (nvec + CS_VECS - 1) / CS_VECS;
  if (threadIdx.x == 0) {
    for (int s = 0; s < CS_STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], CS_THREADS / 32);
    }
    abort_word = 0;
    fence_barrier_init();
  }
  __syncthreads();
  int stage = 0;
  uint32_t phase = 0;
  bool ok = true;
  if (threadIdx.x >= CS_THREADS) {
    if (lane == 0) {
      int64_t issued = 0;
      for (int64_t row = blockIdx.x; row < T && ok; row += gridDim.x) {
        const uint4* lv = reinterpret_cast<const uint4*>(logits + row * ld);
        for (int i = 0; i < 2 * chunks && ok; ++i) {
          const int c0 = (i < chunks ? i : i - chunks) * CS_VECS;
          const uint32_t bytes = min(CS_VECS, nvec - c0) * 16;
          ok = mbar_wait_bounded(&empty[stage], phase ^ 1, abort_flag, status, kTimeoutEmptyBarrier, blockIdx.x);
          if (!ok) break;
          mbar_arrive_expect_tx(&full[stage], bytes);
          bulk_load(smem + stage * CS_VECS * 16, lv + c0, bytes, &full[stage]);
          ++issued;
          if (++stage == CS_STAGES) { stage = 0; phase ^= 1; }
        }
      }
      if (!ok) {       // no copy may land after the CTA has gone
        for (int64_t i = 0; i < min(issued, static_cast<int64_t>(CS_STAGES)); ++i) {
          if (--stage < 0) { stage = CS_STAGES - 1; phase ^= 1; }
          const uint64_t t0 = globaltimer_ns();
          while (!mbar_try_wait(&full[stage], phase) && globaltimer_ns() - t0 < 100000000ull) {}
        }
      }
    }
    return;
  }
  for (int64_t row = blockIdx.x; row < T; row += gridDim.x) {
    const CeRow r = ce_row(logits, target, row, V, ld);
    const bool has_tail = static_cast<int>(threadIdx.x) < r.tail;
    const float ft = has_tail ? __bfloat162float(r.lr[nvec * 8 + threadIdx.x]) : -INFINITY;
    // shift: the running maximum, 0 while every logit seen is -inf (the sum is then 0, not NaN)
    float m = ft, shift = ft == -INFINITY ? 0.f : ft;
    float2 s = make_float2(has_tail ? ce_exp(ft, shift) : 0.f, 0.f);
    uint4 v[CS_PER_THREAD];
    auto next = [&](int k) {
      if (ok) ok = mbar_wait_bounded(&full[stage], phase, abort_flag, status, kTimeoutFullBarrier, blockIdx.x);
      const uint4* sv = reinterpret_cast<const uint4*>(smem + stage * CS_VECS * 16) + threadIdx.x;
      if ((k + 1) * CS_VECS <= nvec) {
#pragma unroll
        for (int u = 0; u < CS_PER_THREAD; ++u) v[u] = sv[u * CS_THREADS];
      } else {
#pragma unroll
        for (int u = 0; u < CS_PER_THREAD; ++u)
          v[u] = k * CS_VECS + static_cast<int>(threadIdx.x) + u * CS_THREADS < nvec
                     ? sv[u * CS_THREADS]
                     : make_uint4(0xff80ff80u, 0xff80ff80u, 0xff80ff80u, 0xff80ff80u);      // -inf: adds nothing
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[stage]);
      if (++stage == CS_STAGES) { stage = 0; phase ^= 1; }
    };
    for (int k = 0; k < chunks; ++k) {
      next(k);
      bf162 m2 = ce_vec_max(v[0]);
#pragma unroll
      for (int u = 1; u < CS_PER_THREAD; ++u) m2 = __hmax2(m2, ce_vec_max(v[u]));
      const float vm = ce_max(m2);
      if (vm > m) {
        if (m > -INFINITY) {                                 // (before any finite logit s is 0, or NaN)
          const float a = ce_exp(shift, vm);
          s = ce_mul2(s, make_float2(a, a));
        }
        m = shift = vm;
      }
#pragma unroll
      for (int u = 0; u < CS_PER_THREAD; ++u) s = ce_add_exps(s, v[u], shift);
    }
    const float mx = group_max<CS_THREADS>(m, red);
    const float st = s.x + s.y;
    const float se = group_sum<CS_THREADS>(m == -INFINITY && mx > -INFINITY ? st : st * ce_exp(m, mx), red + 32);
    const float lse = mx + __logf(se);
    if (threadIdx.x == 0) loss[row] = r.valid ? lse - r.at_target : 0.f;
    const float gs = r.valid ? grad_scale : 0.f;
    for (int k = 0; k < chunks; ++k) {
      next(k);
#pragma unroll
      for (int u = 0; u < CS_PER_THREAD; ++u) {
        const int c = k * CS_VECS + threadIdx.x + u * CS_THREADS;
        if (c < nvec) ce_grad(v[u], r, c, lse, gs);
      }
    }
    if (has_tail) ce_tail_grad(r, ft, lse, gs);
  }
}

}  // namespace
}  // namespace hpb

using namespace hpb;

extern "C" int hpb_cross_entropy(void* logits, const int64_t* target, float* loss, int64_t T, int V, int64_t ld,
                                 float grad_scale, int* status, int num_sms, cudaStream_t s) {
  if (ld % 8 || (reinterpret_cast<uintptr_t>(logits) & 15)) return -2;
  if (T == 0) return 0;
  const int nvec = V >> 3;
  const unsigned g = static_cast<unsigned>(T);
  bf16* l = reinterpret_cast<bf16*>(logits);
  if (nvec <= 128) ce_reg_kernel<128, 1><<<g, 128, 0, s>>>(l, target, loss, V, ld, grad_scale);
  else if (nvec <= 256) ce_reg_kernel<128, 2><<<g, 128, 0, s>>>(l, target, loss, V, ld, grad_scale);
  else if (nvec <= 512) ce_reg_kernel<128, 4><<<g, 128, 0, s>>>(l, target, loss, V, ld, grad_scale);
  else if (nvec <= 1024) ce_reg_kernel<128, 8><<<g, 128, 0, s>>>(l, target, loss, V, ld, grad_scale);
  else {
    static bool configured[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !configured[dev]) {
      cudaError_t e = cudaFuncSetAttribute(ce_stream_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, CS_SMEM);
      if (e != cudaSuccess) return static_cast<int>(e);
      if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    const int64_t ctas = 2ll * num_sms;
    ce_stream_kernel<<<static_cast<unsigned>(T < ctas ? T : ctas), CS_THREADS + 32, CS_SMEM, s>>>(
        l, target, loss, T, V, ld, grad_scale, status);
  }
  return static_cast<int>(cudaGetLastError());
}
