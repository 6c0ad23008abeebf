// Router logits of many bf16 rows on tcgen05 at fp32 precision: a fp32 weight is the exact sum of three bf16 parts (8 + 8 + 8 bits), bf16 rows are exact, so
// every product is exact in fp32 and only the sums round.
//   CTA = 128 tokens x 128 experts x a part of the columns, 64 columns a round.  8 warps bring the rows and split the weights on their way into a three-stage
//   ring, one warp issues 12 UMMA 128x128x16 a round (lowest parts first) into one of two accumulators, 8 warps add the round's sums up in fp32
//   registers: the tensor core adds without rounding to nearest (2e-6 .. 7e-6 off over 2048 .. 6144 columns when it carries the sum alone).
// What bounds it: a few rounds of 768 MMA clocks and the first loads' latency.  Logits and choice together, us, here / the same parts on mma.sync in blocks of
// 32 tokens (bound by those MMAs): 4096 tokens x 128 experts of 2048 columns 24 / 61, 1000 tokens 18 / 25, 256 tokens 17 / 24, 4096 x 512 54 / 195.
#include <cuda_bf16.h>

#include <algorithm>
#include <stdexcept>

#include "api.h"
#include "common.cuh"
#include "mbar_wait.cuh"
#include "seqmix.h"

namespace nxdi {
namespace {

constexpr int RT_T = 128, RT_E = 128, RT_K = 64, RT_STAGES = 3;
constexpr int RT_TILE = 128 * RT_K * 2, RT_STAGE = 4 * RT_TILE;          // rows | weights' three parts, 128-byte rows, SWIZZLE_128B
constexpr int RT_THREADS = 17 * 32, RT_SMEM = RT_STAGES * RT_STAGE + 1024;

__device__ __forceinline__ uint64_t rt_desc(const void* smem) {
  uint64_t d = 0;
  d |= (uint64_t)((mbar_s32(smem) & 0x3FFFF) >> 4);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
__device__ __forceinline__ uint32_t rt_swz(int row, int piece) { return (uint32_t)(row * 128 + ((piece ^ (row & 7)) << 4)); }

__global__ void __launch_bounds__(RT_THREADS, 1) router_logits_tc_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ w, float* __restrict__ logits,
                                                                         float* __restrict__ parts, int N, int W, int E, unsigned* wait_word) {
  extern __shared__ __align__(1024) uint8_t rt_raw[];
  uint8_t* smem = rt_raw + ((1024u - (mbar_s32(rt_raw) & 1023u)) & 1023u);
  __shared__ uint64_t full[RT_STAGES], empty[RT_STAGES], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int s_stop;
  volatile int* stop = &s_stop;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < RT_STAGES; ++s) {
      mbar_init(&full[s], 8);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 8);
    }
    s_stop = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 16) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(mbar_s32(&tmem_slot)), "n"(256));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot;
  const int t0 = blockIdx.x * RT_T, e0 = blockIdx.y * RT_E;
  // this block's part of the columns: part 0 goes to `logits`, the others to `parts`, router_select_kernel adds them in order
  const int rounds = W / RT_K, r0 = (int)((long long)rounds * blockIdx.z / gridDim.z), nr = (int)((long long)rounds * (blockIdx.z + 1) / gridDim.z) - r0;
  if (blockIdx.z > 0) logits = parts + (size_t)(blockIdx.z - 1) * N * E;

  if (warp < 8) {
    // ================= rows and weights =================
    uint4 xr[4];
    float4 wr[4][2];
    auto fetch = [&](int r) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int u = threadIdx.x + 256 * j, row = u >> 3, k = (r0 + r) * RT_K + (u & 7) * 8;
        xr[j] = t0 + row < N ? __ldg(reinterpret_cast<const uint4*>(x + (size_t)(t0 + row) * W + k)) : make_uint4(0u, 0u, 0u, 0u);
        const float4* q = reinterpret_cast<const float4*>(w + (size_t)min(e0 + row, E - 1) * W + k);
        wr[j][0] = __ldg(q);
        wr[j][1] = __ldg(q + 1);
      }
    };
    if (nr > 0) fetch(0);
    for (int r = 0; r < nr; ++r) {
      const int s = r % RT_STAGES;
      if (!mbar_wait_warp(&empty[s], (uint32_t)((r / RT_STAGES) & 1) ^ 1u, stop, wait_word)) break;
      uint8_t* st = smem + s * RT_STAGE;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int u = threadIdx.x + 256 * j;
        const uint32_t at = rt_swz(u >> 3, u & 7);
        *reinterpret_cast<uint4*>(st + at) = xr[j];
        float v[8] = {wr[j][0].x, wr[j][0].y, wr[j][0].z, wr[j][0].w, wr[j][1].x, wr[j][1].y, wr[j][1].z, wr[j][1].w};
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          uint32_t p[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            p[k] = pack_bf16(v[2 * k], v[2 * k + 1]);
            v[2 * k] -= bf16lo(p[k]);
            v[2 * k + 1] -= bf16hi(p[k]);
          }
          *reinterpret_cast<uint4*>(st + (1 + q) * RT_TILE + at) = make_uint4(p[0], p[1], p[2], p[3]);
        }
      }
      if (r + 1 < nr) fetch(r + 1);
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&full[s]);
    }
  } else if (warp < 16) {
    // ================= sums: thread = token x half of the experts =================
    const int half = (warp - 8) >> 2, row = (warp & 3) * 32 + lane;
    const uint32_t at = tmem + ((uint32_t)((warp & 3) * 32) << 16) + half * 64;
    float sum[64];
#pragma unroll
    for (int e = 0; e < 64; ++e) sum[e] = 0.f;
    bool ok = true;
    for (int r = 0; r < nr && ok; ++r) {
      const int b = r & 1;
      ok = mbar_wait_warp(&acc_full[b], (uint32_t)((r >> 1) & 1), stop, wait_word);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int c = 0; c < 64; c += 16) {
        uint32_t v[16];
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                     : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]),
                       "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                     : "r"(at + (uint32_t)(b * 128 + c)));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int e = 0; e < 16; ++e) sum[c + e] += __uint_as_float(v[e]);
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[b]);
    }
    const int t = t0 + row, e_first = e0 + half * 64;
    if (ok && t < N) {
      float* dst = logits + (size_t)t * E + e_first;
      if (E % 4 == 0) {
#pragma unroll
        for (int e = 0; e < 64; e += 4)
          if (e_first + e < E) *reinterpret_cast<float4*>(dst + e) = make_float4(sum[e], sum[e + 1], sum[e + 2], sum[e + 3]);
      } else {
#pragma unroll
        for (int e = 0; e < 64; ++e)
          if (e_first + e < E) dst[e] = sum[e];
      }
    }
  } else {
    // ================= MMAs =================
    uint32_t on;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(on));
    // D = f32, A = B = bf16, both K-major, M = N = 128
    constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(RT_E >> 3) << 17) | ((uint32_t)(RT_T >> 4) << 24);
    auto commit = [&](uint64_t* bar) {
      asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(mbar_s32(bar)),
                   "r"(on) : "memory");
    };
    for (int r = 0; r < nr; ++r) {
      const int s = r % RT_STAGES, b = r & 1;
      if (!mbar_wait_warp(&full[s], (uint32_t)((r / RT_STAGES) & 1), stop, wait_word) ||
          !mbar_wait_warp(&acc_empty[b], (uint32_t)((r >> 1) & 1) ^ 1u, stop, wait_word))
        break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint64_t da = rt_desc(smem + s * RT_STAGE);
#pragma unroll
      for (int i = 0; i < 12; ++i) {
        const int q = 2 - i / 4, k = i & 3;              // 16 k = 32 bytes inside the swizzle atom
        const uint64_t db = da + (uint64_t)((1 + q) * (RT_TILE >> 4) + k * 2);
        asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(
                         tmem + (uint32_t)(b * 128)), "l"(da + (uint64_t)(k * 2)), "l"(db), "r"(idesc), "r"(i != 0 ? 1u : 0u), "r"(on) : "memory");
      }
      commit(&empty[s]);
      commit(&acc_full[b]);
    }
  }
  if (*stop) __nanosleep(1000000);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 16) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(256));
  }
}

}  // namespace

// Column parts of the tensor-core kernel, up to one block per SM and at least two rounds each; 0: the CUDA-core kernels.  A block computes 128 experts whether
// they exist or not, so fewer than 64 stay with the CUDA cores, and so do a few tokens (N = 128: 17 us there).
int router_parts(int N, int W, int E, bool lp) {
  if (!lp || N < 256 || E < 64 || W % RT_K != 0) return 0;
  const long long blocks = (long long)((N + RT_T - 1) / RT_T) * ((E + RT_E - 1) / RT_E);
  return (int)std::max<long long>(1, std::min<long long>({8, kNumSMs / blocks, W / (2 * RT_K)}));
}
void router_logits_tc_launch(const void* x, const float* w, float* logits, float* parts, int N, int W, int E, int n_parts, cudaStream_t st) {
  check_waits();
  count_launch(COUNT_ROUTER);
  if (cudaFuncSetAttribute(router_logits_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, RT_SMEM) != cudaSuccess)
    throw std::runtime_error("router: shared memory size refused");
  router_logits_tc_kernel<<<dim3((N + RT_T - 1) / RT_T, (E + RT_E - 1) / RT_E, n_parts), RT_THREADS, RT_SMEM, st>>>(
      (const __nv_bfloat16*)x, w, logits, parts, N, W, E, wait_word(WAIT_ROUTER));
}

}  // namespace nxdi
