// FP8 (e4m3) GEMM with block scaling, 128x256 output tile per CTA.
//
// Same contract as hpb_gemm_fp8_blockscale (gemm_fp8_sm100.cu): C = dequant(A) * dequant(B)^T with one
// activation scale per 1x128 tile, sa [K/128, M], and one weight scale per 128x128 tile, sb [N/128, K/128].
//
// Two-level accumulation as there: every 128-deep partial product (256 fp32 columns of tensor memory, two
// buffers) is scaled and added to a sum in registers.  What bounds this loop is the turn-round of a buffer
// -- product, commit, tensor-memory load, release -- and the shared-memory pipe: while the tensor core reads
// its operands, even a wait on a completed barrier takes 200 to 400 cycles.  Hence twice the columns per turn
// of the 128x128 kernel, sixteen promotion warps of 32 rows x 64 columns, one wait and two scale reads per warp
// and block, and scales that travel with the operands (fetched by the promotion warps they cost an L2 round
// trip per block, with barriers of their own 10 %).  Measured against the 128x128 kernel: 4096 x 36864 x 7168
// 1466-1612 -> 1034-1052 us (2.1 PFLOP/s), 4096 x 7168 x 18432 781 -> 561 us, 1024 x 7168 x 7168 113 -> 75 us,
// 203 x 36864 x 7168 110 -> 78 us.
// (Tried: 256x256 tiles on CTA pairs.  The release then crosses the cluster, 1300-1900 cycles per turn, and
// the kernel was slower than the 128x128 one from K = 7168 on.)
//
//   warp 0       producer: operand tiles by TMA, the block's 128 + 2 scales by cp.async into an eight-slot ring
//                (both complete on the stage's barrier)
//   warp 1       MMA issuer
//   warps 4-19   promotion; C leaves through swizzled shared memory and TMA stores
// Every wait is bounded (see sm100_common.cuh).
#include "epilogue_store.cuh"
#include "sm100_common.cuh"

namespace hpb {
namespace f8w {

constexpr int TILE_M = 128, TILE_N = 256;
constexpr int GROUP_M = 16;                      // raster: row blocks that share the weight tiles in L2
constexpr int BK = 128;                          // elements = bytes: one scale block, one swizzle row
constexpr int UMMA_K = 32;
constexpr int STAGES = 3;
constexpr int A_BYTES = TILE_M * BK;             // 16 KB
constexpr int B_BYTES = TILE_N * BK;             // 32 KB
constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int PROMO_WARPS = 16;
constexpr int THREADS = 128 + PROMO_WARPS * 32;
// 640 threads launch with 96 registers each = 61440; 128 x 56 + 512 x 104 = 60416
constexpr int PRODUCER_REGS = 56, PROMO_REGS = 104;
constexpr int TMEM_COLS = 512;
constexpr int EPI8_BYTES = PROMO_WARPS * EPI_TILE_BYTES;     // one 4 KB store tile per warp
constexpr int SC_SLOTS = 8;
constexpr int SC_FLOATS = TILE_M + 4;          // 128 activation scales, then the weight scales of both column halves
constexpr int SC_BYTES = SC_SLOTS * SC_FLOATS * 4;
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + EPI8_BYTES + SC_BYTES + 1024 + 512;

struct Params {
  int M, N, K;
  const float* sa;
  const float* sb;
  int* status;
};

__device__ __forceinline__ void tile_coords(int t, int num_m, int num_n, int& m_blk, int& n_blk) {
  const int per_group = GROUP_M * num_n;
  const int group = t / per_group;
  const int first_m = group * GROUP_M;
  const int gsz = min(num_m - first_m, GROUP_M);
  const int r = t - group * per_group;
  m_blk = first_m + r % gsz;
  n_blk = r / gsz;
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(d)
      : "l"(*reinterpret_cast<unsigned long long*>(&a)), "l"(*reinterpret_cast<unsigned long long*>(&b)),
        "l"(*reinterpret_cast<unsigned long long*>(&c)));
  return *reinterpret_cast<float2*>(&d);
}

// The operand `bytes` further into shared memory: one 32-bit add (the address field cannot carry out).
__device__ __forceinline__ uint64_t desc_at(uint64_t desc, uint32_t bytes) {
  return (desc & 0xffffffff00000000ull) | (static_cast<uint32_t>(desc) + (bytes >> 4));
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void cp_async4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
// One arrival of this thread on `bar` once its cp.asyncs so far have landed.
__device__ __forceinline__ void cp_async_arrive(uint64_t* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__global__ void __launch_bounds__(THREADS, 1)
gemm_fp8_wide_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                 const __grid_constant__ CUtensorMap tmap_c, const Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* epi = smem + STAGES * STAGE_BYTES;
  float* scales = reinterpret_cast<float*>(epi + EPI8_BYTES);
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(epi + EPI8_BYTES + SC_BYTES);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* part_full = empty_bar + STAGES;   // [2]
  uint64_t* part_empty = part_full + 2;       // [2]
  uint64_t* drain_bar = part_empty + 2;
  uint32_t* tmem_base_slot = reinterpret_cast<uint32_t*>(drain_bar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_base_slot + 1);

  const int warp = uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int num_m = (p.M + TILE_M - 1) / TILE_M, num_n = (p.N + TILE_N - 1) / TILE_N;
  const int num_tiles = num_m * num_n;
  const int num_k = p.K / BK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1 + 32);     // operand bytes; the 32 lanes that copy the scales
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&part_full[b], 1);
      mbar_init(&part_empty[b], PROMO_WARPS);
    }
    mbar_init(drain_bar, 1);
    *abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
    tma_prefetch_desc(&tmap_c);
  }
  if (warp == 1) {
    tmem_alloc(tmem_base_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_base_slot;

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(PRODUCER_REGS));
    if (warp == 0) {
      int stage = 0, slot = 0;
      uint32_t phase = 0;
      int64_t issued = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < num_tiles && ok; t += gridDim.x) {
        int m_blk, n_blk;
        tile_coords(t, num_m, num_n, m_blk, n_blk);
        const int m0 = m_blk * TILE_M, n0 = n_blk * TILE_N;
        const int sb_row = min(n_blk * 2 + (lane & 1), (p.N - 1) / 128);
        for (int kb = 0; kb < num_k; ++kb) {
          // The slot is free too: a free stage means that block i - STAGES has been multiplied, so that the
          // promotion of block i - STAGES - 2 has released its buffer, and STAGES + 2 < SC_SLOTS.
          ok = mbar_wait_warp(&empty_bar[stage], phase ^ 1, abort_flag, p.status, kTimeoutEmptyBarrier, blockIdx.x);
          if (!ok) break;
          uint8_t* sa = smem + stage * STAGE_BYTES;
          if (lane == 0) {
            mbar_arrive_expect_tx(&full_bar[stage], STAGE_BYTES);
            tma_load_2d(sa, &tmap_a, &full_bar[stage], kb * BK, m0);
            tma_load_2d(sa + A_BYTES, &tmap_b, &full_bar[stage], kb * BK, n0);
          }
          float* dst = scales + slot * SC_FLOATS;
          const float* ga = p.sa + static_cast<int64_t>(kb) * p.M;
#pragma unroll
          for (int i = 0; i < 4; ++i) cp_async4(dst + i * 32 + lane, ga + min(m0 + i * 32 + lane, p.M - 1));
          if (lane < 2) cp_async4(dst + TILE_M + lane, p.sb + static_cast<int64_t>(sb_row) * num_k + kb);
          cp_async_arrive(&full_bar[stage]);
          ++issued;
          if (++slot == SC_SLOTS) slot = 0;
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
      if (!ok) {       // no copy may land after the CTA has gone
        for (int i = 0; i < STAGES && i < issued; ++i) {
          if (--stage < 0) { stage = STAGES - 1; phase ^= 1; }
          const uint64_t t0 = globaltimer_ns();
          while (!mbar_try_wait(&full_bar[stage], phase) && globaltimer_ns() - t0 < 100000000ull) {}
        }
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
    }
    if (warp == 1) {
      // the whole warp walks the loop, one elected lane issues
      constexpr uint32_t idesc = make_idesc(0, 0, 0, 0, TILE_M, TILE_N);      // e4m3 x e4m3 -> fp32
      const uint32_t base = uniform(smem_u32(smem));
      const uint64_t a_desc = make_smem_desc_sw128(base, 0, 1024);
      const uint64_t b_desc = make_smem_desc_sw128(base + A_BYTES, 0, 1024);
      const uint32_t tbase = uniform(tmem_base);
      const bool issuer = elect_one();
      int stage = 0, buf = 0;
      uint32_t phase = 0, bphase = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < num_tiles && ok; t += gridDim.x) {
        for (int kb = 0; kb < num_k; ++kb) {
          ok = mbar_wait_warp(&part_empty[buf], bphase ^ 1, abort_flag, p.status, kTimeoutTmemEmpty, blockIdx.x);
          if (ok) ok = mbar_wait_warp(&full_bar[stage], phase, abort_flag, p.status, kTimeoutFullBarrier, blockIdx.x);
          if (!ok) break;
          tc_fence_after();
          const uint64_t da = desc_at(a_desc, stage * STAGE_BYTES), db = desc_at(b_desc, stage * STAGE_BYTES);
          const uint32_t tmem_d = tbase + buf * TILE_N;
          if (issuer) {
#pragma unroll
            for (int kk = 0; kk < BK / UMMA_K; ++kk)
              umma_f8f6f4(tmem_d, desc_at(da, kk * UMMA_K), desc_at(db, kk * UMMA_K), idesc, kk > 0 ? 1u : 0u);
            umma_commit(&empty_bar[stage]);
            umma_commit(&part_full[buf]);
          }
          __syncwarp();
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
          buf ^= 1;
          if (buf == 0) bphase ^= 1;
        }
      }
      if (!ok && issuer) {
        umma_commit(drain_bar);
        const uint64_t t0 = globaltimer_ns();
        while (!mbar_try_wait(drain_bar, 0) && globaltimer_ns() - t0 < 100000000ull) {}
      }
      __syncwarp();
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(PROMO_REGS));
    const int q = warp & 3;                    // tensor-memory lane quarter
    const int part = (warp - 4) >> 2;          // 64 of the 256 columns
    uint8_t* tile = epi + (warp - 4) * EPI_TILE_BYTES;
    const uint32_t lane_off = static_cast<uint32_t>(q * 32) << 16;
    int buf = 0, slot = 0;
    uint32_t bphase = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < num_tiles && ok; t += gridDim.x) {
      int m_blk, n_blk;
      tile_coords(t, num_m, num_n, m_blk, n_blk);
      const int row0 = m_blk * TILE_M + q * 32, col0 = n_blk * TILE_N + part * 64;
      float2 acc[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) acc[j] = make_float2(0.f, 0.f);
      for (int kb = 0; kb < num_k; ++kb) {
        ok = mbar_wait_bounded(&part_full[buf], bphase, abort_flag, p.status, kTimeoutTmemFull, blockIdx.x);
        if (!ok) break;
        tc_fence_after();
        const uint32_t taddr = tmem_base + buf * TILE_N + part * 64 + lane_off;
        // (the product was issued behind the stage's barrier, on which the scales have landed as well)
        const float* sc = scales + slot * SC_FLOATS;
        const float scale = sc[q * 32 + lane] * sc[TILE_M + (part >> 1)];
        const float2 s2 = make_float2(scale, scale);
        if (++slot == SC_SLOTS) slot = 0;
        uint32_t r[2][16];                     // the load of 16 columns runs under the multiply-adds of the 16 before
        tmem_ld16(taddr, r[0]);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          tmem_ld_wait();
          if (c < 3) {
            tmem_ld16(taddr + (c + 1) * 16, r[(c + 1) & 1]);
          } else {                             // the partial product is in registers
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&part_empty[buf]);
          }
#pragma unroll
          for (int j = 0; j < 8; ++j)
            acc[c * 8 + j] = fma2(make_float2(__uint_as_float(r[c & 1][2 * j]), __uint_as_float(r[c & 1][2 * j + 1])),
                                  s2, acc[c * 8 + j]);
        }
        buf ^= 1;
        if (buf == 0) bphase ^= 1;
      }
      if (!ok) break;
      if (row0 >= p.M) continue;
      if (col0 < p.N) {                        // 64 columns = one 128-byte store row
        if (lane == 0) tma_store_wait_read<0>();
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          uint4 u;
          __nv_bfloat162* b = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
          for (int e = 0; e < 4; ++e) b[e] = __floats2bfloat162_rn(acc[j * 4 + e].x, acc[j * 4 + e].y);
          *reinterpret_cast<uint4*>(tile + lane * 128 + ((j ^ (lane & 7)) << 4)) = u;
        }
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) {
          tma_store_3d(&tmap_c, tile, col0, row0, 0);
          tma_store_commit();
        }
      }
    }
    if (lane == 0) tma_store_wait<0>();
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

}  // namespace f8w

int make_tmap_2d(CUtensorMap* map, const void* ptr, CUtensorMapDataType dtype, int elem_bytes, uint64_t inner,
                 uint64_t outer, uint64_t ld, uint32_t box_inner, uint32_t box_outer);

}  // namespace hpb

// Arguments as hpb_gemm_fp8_blockscale; C 16-byte aligned with ldc % 8 == 0.
extern "C" int hpb_gemm_fp8_blockscale_wide(const void* Aq, const float* sa, const void* Bq, const float* sb, void* C,
                                        long long ldc, int M, int N, int K, int* status, int num_sms,
                                        cudaStream_t stream) {
  using namespace hpb;
  using namespace hpb::f8w;
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if ((K % BK) || (reinterpret_cast<uintptr_t>(Aq) & 15) || (reinterpret_cast<uintptr_t>(Bq) & 15)) return -2;
  cudaFree(nullptr);
  CUtensorMap ta, tb, tc;
  int r = make_tmap_2d(&ta, Aq, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, K, M, K, BK, TILE_M);
  if (r) return r;
  r = make_tmap_2d(&tb, Bq, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, K, N, K, BK, TILE_N);
  if (r) return r;
  if (!make_tmap_c(&tc, C, false, N, M, 1, ldc)) return -2;
  static bool configured[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    // the promotion warps' registers come out of what the CTA launches with: less would leave them waiting for good
    cudaFuncAttributes fa;
    cudaError_t e = cudaFuncGetAttributes(&fa, gemm_fp8_wide_kernel);
    if (e != cudaSuccess) return static_cast<int>(e);
    if (fa.numRegs * THREADS < 128 * PRODUCER_REGS + PROMO_WARPS * 32 * PROMO_REGS) return -6;
    e = cudaFuncSetAttribute(gemm_fp8_wide_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
    if (e != cudaSuccess) return static_cast<int>(e);
    if (dev >= 0 && dev < 64) configured[dev] = true;
  }
  const int64_t tiles = static_cast<int64_t>((M + TILE_M - 1) / TILE_M) * ((N + TILE_N - 1) / TILE_N);
  if (tiles > 0x3fffffff) return -2;
  Params p{M, N, K, sa, sb, status};
  gemm_fp8_wide_kernel<<<tiles < num_sms ? static_cast<int>(tiles) : num_sms, THREADS, SMEM_BYTES, stream>>>(ta, tb, tc,
                                                                                                          p);
  return static_cast<int>(cudaGetLastError());
}
