// GEMM of a few tokens with large weights (9 .. 128 tokens of a batched decode step; the tokens of one expert of a small MoE step):
// Y[t, n] = act(X W^T).  The weights are the M operand of the tensor cores and the tokens the N operand (swapped against gemm_tcgen05.cu, whose
// 128-row token tiles would be mostly padding and whose tile grid leaves a last wave nearly empty).
//
// What bounds it: the weight stream from HBM.  So
//   * CTA c of G takes the k-blocks [total c / G, total (c + 1) / G) of the concatenated (segment, 128-feature tile, k) space: every SM streams the
//     same number of bytes whatever the shape (stream-K).  Tiles cut by a boundary meet in fp32 partials; the CTA that arrives last adds them in
//     k order (deterministic) and runs the epilogue.
//   * a stage is a weight box of 128 rows x 64 k (two for gate | up; 128 k for one plain bf16 weight) plus the tokens' columns; the ring takes all of shared
//     memory (100 .. 180 KB of weights in flight per SM), weights and tokens have a TMA producer warp each.  4096 x 4096 at 9 tokens 11.7 us with 128 k a stage,
//     13.3 with 64.
//   * int8 / e4m3 weights come as bytes, 128 k a box; eight warps expand them to bf16 (exactly) into TMEM, from where the MMAs read them as their A operand; the scale is
//     applied to the fp32 sum.
//   * accumulators (128 features x tokens) sit in TMEM twice, so a tile's epilogue overlaps the stream of the next one.  A lane holds one output
//     feature: a warp's store of one token is 64 contiguous bytes, gate and up of a feature meet in one thread.
//   * 16 epilogue warps: the last tile's epilogue is the tail of the launch, and so is the fix-up of its parts.  Both are round trips to L2 and cold
//     instructions, so: every load of a group of 8 tokens (residual, parts) before the first use, the activation chosen outside of the loops, one code path.
//     With 8 warps, groups of 16 tokens, three copies of the epilogue and the residual read where it was added, the tail after the last weights was
//     25 us at 37 tokens, 28672 x 4096 gate | up (now 8) and 17 us at 4096 x 14336 with a residual (now 6).
// Measured (us, here / 128-row token tiles): see skinny_pays in bindings.cpp, 8-bit weights: linear8_few.  28672 x 4096 gate | up at 9 tokens 42.5 us = 5.5 TB/s
// (46 before), a gated MLP of 8B sizes with norm and residual at 37 tokens 77 us in a graph (100 before); six of eight Mixtral-sized experts, 6 tokens, with permutation
// and sum: 336 us = 6.3 TB/s (one warp per weight row and (token, slot) pair: 744 us).
#include <algorithm>
#include <stdexcept>
#include <string>

#include "api.h"
#include "common.cuh"
#include "mbar_wait.cuh"

namespace nxdi {

constexpr int SK_BM = 128, SK_BK = 64;                 // weight rows, k elements per stage box (128-byte rows)
constexpr int SK_W_BYTES = SK_BM * SK_BK * 2;
constexpr int SK_THREADS = 640;                        // 4 warps: weights, MMA, TMEM, tokens; 16 epilogue warps, or 8 that expand 8-bit weights and 8 epilogue warps
constexpr int SK_A_BUFS = 4, SK_A_COLS = 64;           // 8-bit weights: expanded boxes in TMEM, 128 k each
__host__ __device__ constexpr int sk_epi(int wt) { return wt ? 8 : 16; }
// k elements of a stage: with 128, one copy brings 32 KB of bf16 weights (or 16 KB of bytes) and one the tokens' columns.  A thread issues a copy in 0.25 us, in which an
// SM's share of HBM brings 11 KB.
__host__ __device__ constexpr int sk_bk(int wt, bool wide) { return wt || wide ? 128 : SK_BK; }
constexpr int SK_MAX_STAGES = 12;
constexpr int SK_SMEM = 220 * 1024;
// the warps that expand 8-bit weights count on as many stages as there are expanded boxes, for the largest blocks too (128 tokens; 64 beside two weight boxes)
static_assert((SK_SMEM - 1024) / (SK_W_BYTES + SKINNY_MAX_T * 128 * 2) >= SK_A_BUFS && (SK_SMEM - 1024) / (2 * SK_W_BYTES + SKINNY_MAX_T / 2 * 128 * 2) >= SK_A_BUFS, "ring of 8-bit weights");

struct SkinnyKernelParams {
  CUtensorMap tm_w;        // [experts * rows, K], box {64, 128} (bytes: {128, 128}); wide: as {64, rows, K / 64}, box {64, 128, 2}
  CUtensorMap tm_x;        // [token rows, K], box {64, xbox}: xb rows for one expert, 16 when grouped (an expert loads as many as it has tokens for); 128 k: {64, xb, 2}
  CUtensorMap tm_x64;      // grouped, segments of more than 48 rows: box {64, 64}
  const int *n_active, *active, *seg_start, *seg_count;     // grouped: segments (expert, first row of x, rows <= xb); null: one expert, T rows
  const __nv_bfloat16 *bias, *residual;                      // [experts * rows]; [T, n_out] (one expert)
  const float* scale;      // 8-bit weights: [rows], or [1] with scale_step 0
  int scale_step;
  void* y;                 // [token rows, n_out] bf16, or fp32 (y_f32)
  float* ws;               // [G][2][cols / 4][128][4] partial tiles
  unsigned* tickets;       // [G], zero at launch
  int T, n_out, rows, K, act, xb, xbox, stages, y_f32, tmem_cols, w_fresh;
  float limit, alpha;
  unsigned* wait_word;     // mbar_wait.cuh
};

__device__ __forceinline__ void sk_tma3(void* dst, const CUtensorMap* tm, int row, int group, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(mbar_s32(dst)), "l"(tm),
               "r"(0), "r"(row), "r"(group), "r"(mbar_s32(bar)) : "memory");
}
__device__ __forceinline__ void sk_tma(void* dst, const CUtensorMap* tm, int c0, int c1, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(mbar_s32(dst)), "l"(tm),
               "r"(c0), "r"(c1), "r"(mbar_s32(bar)) : "memory");
}
// K-major operand tile of 128-byte rows, SWIZZLE_128B; 8-row groups are 1024 B apart
__device__ __forceinline__ uint64_t sk_desc(const void* smem) {
  uint64_t d = 0;
  d |= (uint64_t)((mbar_s32(smem) & 0x3FFFF) >> 4);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
// Called by a whole warp, issued by the lane whose `on` is 1: in code that all lanes run the descriptors stay in uniform registers.  (In a branch for one lane each
// is moved there before its instruction: the issuing thread took 0.8 us for a box of 128 rows and eight instructions, more than its bytes take from HBM.)
__device__ __forceinline__ void sk_umma(uint32_t on, uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc) {
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d), "l"(da),
               "l"(db), "r"(idesc), "r"(acc), "r"(on) : "memory");
}
__device__ __forceinline__ void sk_umma_ts(uint32_t on, uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t idesc, uint32_t acc) {
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
               "r"(tmem_a), "l"(db), "r"(idesc), "r"(acc), "r"(on) : "memory");
}
__device__ __forceinline__ void sk_commit(uint32_t on, uint64_t* bar) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(mbar_s32(bar)),
               "r"(on) : "memory");
}
__device__ __forceinline__ uint32_t sk_elect() {
  uint32_t r;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r));
  return r;
}
__device__ __forceinline__ void sk_ld8(uint32_t taddr, uint32_t (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]) : "r"(taddr));
}

__device__ __forceinline__ void sk_st32(uint32_t taddr, const uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]),
      "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]),
      "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]),
      "r"(v[31])
      : "memory");
}
// four one-byte weights (k ascending) -> two bf16 pairs, exact
template <int WT>
__device__ __forceinline__ void sk_expand4(uint32_t w, uint32_t& lo, uint32_t& hi) {
  if constexpr (WT == 2) {        // e4m3
    uint32_t a, b;
    asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(a) : "h"((unsigned short)(w & 0xffffu)));
    asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(b) : "h"((unsigned short)(w >> 16)));
    const float2 fa = __half22float2(*reinterpret_cast<const __half2*>(&a)), fb = __half22float2(*reinterpret_cast<const __half2*>(&b));
    lo = pack_bf16(fa.x, fa.y);
    hi = pack_bf16(fb.x, fb.y);
  } else {                        // int8: 128 + the low seven bits under the exponent of 128, minus 128 or (negative) 256
    const uint32_t a = __byte_perm(w, 0x43434343u, 0x5140), b = __byte_perm(w, 0x43434343u, 0x5342);
    asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(lo) : "r"(a & 0xff7fff7fu), "r"(a & 0xff80ff80u));
    asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(hi) : "r"(b & 0xff7fff7fu), "r"(b & 0xff80ff80u));
  }
}

// WT: 0 bf16 weights, 1 int8, 2 e4m3.  WIDE (bf16, one weight without a gate product): 128 k a stage
template <bool GLU, int WT, bool WIDE>
__global__ void __launch_bounds__(SK_THREADS, 1) skinny_gemm_kernel(const __grid_constant__ SkinnyKernelParams p) {
  constexpr int NW = GLU ? 2 : 1, EPI = sk_epi(WT), W_EPI = SK_THREADS / 32 - EPI, T_EPI = W_EPI * 32, BK = sk_bk(WT, WIDE), XBOX = BK / SK_BK;
  constexpr int W_BYTES = WIDE ? 2 * SK_W_BYTES : SK_W_BYTES;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (mbar_s32(smem_raw) & 1023u)) & 1023u);
  __shared__ uint64_t full_bar[SK_MAX_STAGES], empty_bar[SK_MAX_STAGES], tmem_full[2], tmem_empty[2], a_full[SK_A_BUFS], a_empty[SK_A_BUFS];
  __shared__ uint32_t tmem_slot;
  __shared__ int s_stop, s_last;
  volatile int* stop = &s_stop;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ST = p.stages, x_bytes = p.xb * BK * 2, stage_bytes = NW * W_BYTES + x_bytes;     // xb % 16 == 0: multiples of 1024

  if (warp == 0 && lane == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&p.tm_w) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&p.tm_x) : "memory");
    if (p.n_active) asm volatile("prefetch.tensormap [%0];" ::"l"(&p.tm_x64) : "memory");
    for (int s = 0; s < ST; ++s) {
      mbar_init(&full_bar[s], 2);         // the two producers
      mbar_init(&empty_bar[s], WT ? 1 + 4 * NW : 1);      // the MMAs' commit, and the warps that expand the weights
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tmem_full[b], 1);
      mbar_init(&tmem_empty[b], EPI);
    }
    for (int b = 0; b < SK_A_BUFS && WT; ++b) {
      mbar_init(&a_full[b], 4);
      mbar_init(&a_empty[b], 1);
    }
    s_stop = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(mbar_s32(&tmem_slot)), "r"(p.tmem_cols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot;
  pdl_launch_dependents();
  // a dense weight that is a parameter does not depend on earlier kernels; everything else does
  const bool grouped = p.n_active != nullptr;
  bool early = warp == 0 && !grouped && !p.w_fresh;
  if (!early) pdl_wait();

  const int n_tiles = (p.n_out + SK_BM - 1) / SK_BM, nkb = p.K / BK;
  // 8-bit weights: more tokens than a token tile holds are blocks of xb rows, which share the weights in L2
  const int n_seg = grouped ? *p.n_active : WT ? (p.T + p.xb - 1) / p.xb : 1;
  const long long total = (long long)n_seg * n_tiles * nkb;
  const long long G = max(1ll, min((long long)gridDim.x, total / 4));                // at least four k-blocks per CTA that works
  const long long u0 = blockIdx.x < G ? total * blockIdx.x / G : 0, u1 = blockIdx.x < G ? total * (blockIdx.x + 1) / G : 0;
  const int acc_cols = NW * p.xb;

  if (warp == 0 || warp == 3) {
    // ================= TMA producers: weights, tokens =================
    if (lane == 0) {
      int s = 0;                 // counted, not divided out of a 64-bit count: 4096 x 14336, 9 tokens, 30.1 -> 26.1 us
      uint32_t phase = 0;
      bool go = true;
      for (long long u = u0; u < u1 && go;) {
        const int tile = (int)(u / nkb), kb0 = (int)(u % nkb), kb1 = (int)min((long long)nkb, kb0 + (u1 - u));
        const int ei = tile / n_tiles, n0 = (tile % n_tiles) * SK_BM, e = grouped ? p.active[ei] : 0;
        const int row_w = e * p.rows + n0, row_x = grouped ? p.seg_start[ei] : ei * p.xb;
        // a segment's rows in boxes of 64 as far as they go, the rest in one more (where it fits) or in up to two of 16: each copy costs the issuing thread 0.25 us
        int boxes = 1, big = 0;
        const int box_bytes = p.xbox * SK_BK * 2;
        if (grouped) {
          const int cnt = p.seg_count[ei];
          big = cnt / 64 + (cnt % 64 > 32 && (cnt / 64 + 1) * 64 <= p.xb ? 1 : 0);
          boxes = max(0, (cnt - big * 64 + 15) / 16);
        }
        for (int kb = kb0; kb < kb1; ++kb) {
          if (early && phase != 0) {       // the ring is full: from here on a wait depends on the warps that wait for earlier kernels
            pdl_wait();
            early = false;
          }
          go = mbar_wait(&empty_bar[s], phase ^ 1u, stop, p.wait_word);
          if (!go) break;
          uint8_t* st = smem + (size_t)s * stage_bytes;
          if (warp == 0) {
            mbar_expect(&full_bar[s], NW * W_BYTES);
            if (WIDE) sk_tma3(st, &p.tm_w, row_w, kb * 2, &full_bar[s]);
            else sk_tma(st, &p.tm_w, kb * BK, row_w, &full_bar[s]);
            if (GLU) sk_tma(st + W_BYTES, &p.tm_w, kb * BK, row_w + p.n_out, &full_bar[s]);
          } else {
            mbar_expect(&full_bar[s], boxes * box_bytes * XBOX + big * (64 * SK_BK * 2));
            uint8_t* xs = st + NW * W_BYTES;
            if (XBOX == 2) {
              sk_tma3(xs, &p.tm_x, row_x, kb * 2, &full_bar[s]);
            } else {
              for (int q = 0; q < big; ++q) sk_tma(xs + q * (64 * SK_BK * 2), &p.tm_x64, kb * BK, row_x + q * 64, &full_bar[s]);
              for (int q = 0; q < boxes; ++q) sk_tma(xs + big * (64 * SK_BK * 2) + q * box_bytes, &p.tm_x, kb * BK, row_x + big * 64 + q * p.xbox, &full_bar[s]);
            }
          }
          if (++s == ST) {
            s = 0;
            phase ^= 1u;
          }
        }
        u += kb1 - kb0;
      }
    }
  } else if (warp == 1) {
    // ================= MMA issuer =================
    const uint32_t on = sk_elect();
    const uint64_t dw0 = sk_desc(smem), dx0 = sk_desc(smem + NW * W_BYTES);
    const uint32_t half = (uint32_t)(x_bytes / XBOX) >> 4, stage = (uint32_t)stage_bytes >> 4;
    uint32_t at = 0;                                       // of the ring's next stage, in 16-byte units like a descriptor
    int seg = 0, s = 0, ab = 0;
    uint32_t phase = 0, aphase = 0;
    bool go = true;
    for (long long u = u0; u < u1 && go; ++seg) {
      const int kb0 = (int)(u % nkb), kb1 = (int)min((long long)nkb, kb0 + (u1 - u)), buf = seg & 1;
      // D = f32, A = B = bf16, both K-major, M = 128, N = the tokens in whole boxes (a multiple of 16)
      const int nx = grouped ? (p.seg_count[(int)(u / nkb) / n_tiles] + 15) / 16 * 16 : p.xb;
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(nx >> 3) << 17) | ((uint32_t)(SK_BM >> 4) << 24);
      const uint32_t d0 = tmem + (uint32_t)(buf * acc_cols);
      go = mbar_wait_warp(&tmem_empty[buf], (uint32_t)((seg >> 1) & 1) ^ 1u, stop, p.wait_word);
      if (!go) break;
      for (int kb = kb0; kb < kb1; ++kb) {
        go = mbar_wait_warp(&full_bar[s], phase, stop, p.wait_word);
        if (!go) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t db = dx0 + at;
#pragma unroll
        for (int w = 0; w < NW; ++w) {
          const uint32_t d = d0 + (uint32_t)(w * p.xb), first = kb != kb0 ? 1u : 0u;
          if constexpr (WT == 0) {
            const uint64_t da = dw0 + at + (uint64_t)(w * (W_BYTES >> 4));
#pragma unroll
            for (int k = 0; k < BK / 16; ++k)         // 16 k = 32 bytes inside the swizzle atom of 64
              sk_umma(on, d, da + (uint64_t)((k >> 2) * (SK_W_BYTES >> 4) + (k & 3) * 2), db + (uint64_t)((k >> 2) * half + (k & 3) * 2), idesc, k != 0 ? 1u : first);
          } else {
            go = mbar_wait_warp(&a_full[ab], aphase, stop, p.wait_word);
            if (!go) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t a = tmem + 2 * acc_cols + ab * SK_A_COLS;
#pragma unroll
            for (int k = 0; k < BK / 16; ++k)
              sk_umma_ts(on, d, a + 8 * k, db + (uint64_t)((k >> 2) * half + (k & 3) * 2), idesc, k != 0 ? 1u : first);
            sk_commit(on, &a_empty[ab]);
            if (++ab == SK_A_BUFS) {
              ab = 0;
              aphase ^= 1u;
            }
          }
        }
        if (!go) break;
        sk_commit(on, &empty_bar[s]);
        at += stage;
        if (++s == ST) {
          s = 0;
          at = 0;
          phase ^= 1u;
        }
      }
      if (go) sk_commit(on, &tmem_full[buf]);
      u += kb1 - kb0;
    }
  } else if (WT != 0 && warp >= 4 && warp < W_EPI) {
    // ================= 8-bit weights -> bf16 in TMEM, the MMAs' A operand =================
    // Two sets of four warps (32 weight rows each) take the boxes in turn.  Through TMEM, because shared memory has no room for it: a box is written and read
    // once there as bytes; as bf16 it would be written and read twice more.
    if constexpr (WT != 0) {
      const int set = (warp - 4) >> 2, row = (warp & 3) * 32 + lane;
      const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
      const int n = (int)(u1 - u0) * NW;                  // boxes
      int s = NW == 1 ? set : 0, ab = set;                // counted: divisions of the box's number cost more than its expansion
      uint32_t phase = 0, aphase = 1;
      for (int it = set; it < n; it += 2) {
        // the buffer first: that its last MMAs are done tells that the stage's phase before this one is over, which its parity (this set sees every second
        // phase) does not
        if (!mbar_wait_warp(&a_empty[ab], aphase, stop, p.wait_word)) break;
        if (!mbar_wait_warp(&full_bar[s], phase, stop, p.wait_word)) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t src = mbar_s32(smem + (size_t)s * stage_bytes + (NW == 1 ? 0 : set) * W_BYTES) + row * 128;
#pragma unroll
        for (int h = 0; h < 2; ++h) {                      // 64 k: four 16-byte chunks of the row, XOR-swizzled by TMA
          uint32_t v[32];
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint32_t q[4];
            asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(q[0]), "=r"(q[1]), "=r"(q[2]), "=r"(q[3]) : "r"(src + (((4 * h + c) ^ (row & 7)) << 4)));
#pragma unroll
            for (int k = 0; k < 4; ++k) sk_expand4<WT>(q[k], v[8 * c + 2 * k], v[8 * c + 2 * k + 1]);
          }
          sk_st32(tmem + lanes + 2 * acc_cols + ab * SK_A_COLS + 32 * h, v);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty_bar[s]);
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(&a_full[ab]);
        ab += 2;
        if (ab >= SK_A_BUFS) {
          ab = set;
          aphase ^= 1u;
        }
        s += 2 / NW;
        if (s >= ST) {
          s -= ST;
          phase ^= 1u;
        }
      }
    }
  } else if (warp >= W_EPI) {
    // ================= epilogue: lane = output feature =================
    // One code path for whole tiles and for tiles that meet in the workspace, the activation chosen outside of the loop over the tokens: the epilogue runs once or
    // twice per CTA, so every instruction of it is fetched cold.
    const int n_in = (warp & 3) * 32 + lane, c0 = ((warp - W_EPI) >> 2) * 8;      // the warps of 32 features take groups of 8 tokens in turn
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    int seg = 0;
    bool live = true;          // false once a wait ran out: the warp still takes part in the barriers of the eight
    for (long long u = u0; u < u1; ++seg) {
      const int tile = (int)(u / nkb), kb0 = (int)(u % nkb), kb1 = (int)min((long long)nkb, kb0 + (u1 - u)), buf = seg & 1;
      u += kb1 - kb0;
      const int ei = tile / n_tiles, n = (tile % n_tiles) * SK_BM + n_in, e = grouped ? p.active[ei] : 0;
      const int row0 = grouped ? p.seg_start[ei] : ei * p.xb, cnt = grouped ? p.seg_count[ei] : WT ? min(p.xb, p.T - row0) : p.T;
      const float bg = (p.bias && n < p.n_out) ? __bfloat162float(p.bias[(size_t)e * p.rows + n]) : 0.f;
      const float bu = (GLU && p.bias && n < p.n_out) ? __bfloat162float(p.bias[(size_t)e * p.rows + p.n_out + n]) : 0.f;
      const float sg = WT && n < p.n_out ? __ldcg(p.scale + (size_t)n * p.scale_step) : 1.f, su = WT && GLU && n < p.n_out ? __ldcg(p.scale + (size_t)(p.n_out + n) * p.scale_step) : 1.f;
      const bool whole = kb0 == 0 && kb1 == nkb;
      // CTAs that share the tile: those of its first and last k-block and all between
      const long long f = (long long)tile * nkb;
      const int c_first = whole ? blockIdx.x : (int)(((f + 1) * G - 1) / total), c_last = whole ? blockIdx.x : (int)(((f + nkb) * G - 1) / total);
      if (live) live = mbar_wait_warp(&tmem_full[buf], (uint32_t)((seg >> 1) & 1), stop, p.wait_word);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t acc = tmem + lanes + (uint32_t)(buf * acc_cols);
      bool own = whole;          // this CTA's part comes straight from TMEM (it is the first in k order), the others' from the workspace
      if (!whole) {
        if (kb0 == 0) {
          // the tile's first part is its CTA's last segment, so the other parts are often there already: then they are added to the sums in TMEM, which
          // needs neither slot nor ticket
          if (threadIdx.x == T_EPI) {
            unsigned v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p.tickets + c_first) : "memory");
            s_last = v == (unsigned)(c_last - c_first);
          }
          asm volatile("bar.sync 1, %0;" ::"n"(EPI * 32) : "memory");
          own = s_last != 0;
          asm volatile("bar.sync 1, %0;" ::"n"(EPI * 32) : "memory");     // s_last reusable
        }
        if (!own) {
          // slot 0 of this CTA if the tile began in an earlier one, else slot 1
          float4* mine = reinterpret_cast<float4*>(p.ws + ((size_t)blockIdx.x * 2 + (kb0 == 0 ? 1 : 0)) * acc_cols * SK_BM) + n_in;
#pragma unroll 1
          for (int c = c0; c < cnt && live; c += 2 * EPI) {
#pragma unroll
            for (int w = 0; w < NW; ++w) {
              uint32_t v[8];
              sk_ld8(acc + w * p.xb + c, v);
              asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
              for (int k = 0; k < 8; k += 4)
                __stcg(mine + (size_t)((w * p.xb + c + k) >> 2) * SK_BM, make_float4(__uint_as_float(v[k]), __uint_as_float(v[k + 1]), __uint_as_float(v[k + 2]), __uint_as_float(v[k + 3])));
            }
          }
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(&tmem_empty[buf]);
          __threadfence();
          asm volatile("bar.sync 1, %0;" ::"n"(EPI * 32) : "memory");
          if (threadIdx.x == T_EPI) s_last = atomicAdd(&p.tickets[c_first], 1u) == (unsigned)(c_last - c_first);
          asm volatile("bar.sync 1, %0;" ::"n"(EPI * 32) : "memory");
          const bool last = s_last != 0;
          asm volatile("bar.sync 1, %0;" ::"n"(EPI * 32) : "memory");     // s_last reusable
          if (!last) continue;
        }
        __threadfence();
      }
#pragma unroll 1
      for (int c = c0; c < cnt && live; c += 2 * EPI) {
        float g[8], up[8];
        uint32_t res[8];
        const bool in = n < p.n_out;
        const size_t at = (size_t)(row0 + c) * p.n_out + n;
        if (!GLU && p.residual) {
#pragma unroll
          for (int k = 0; k < 8; ++k)
            if (in && c + k < cnt) res[k] = ldg_act_u16(p.residual + at + (size_t)k * p.n_out);
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) g[k] = up[k] = 0.f;
        if (own) {
          uint32_t vg[8], vu[8];
          sk_ld8(acc + c, vg);
          if (GLU) sk_ld8(acc + p.xb + c, vu);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            g[k] = __uint_as_float(vg[k]);
            if (GLU) up[k] = __uint_as_float(vu[k]);
          }
        }
        // the other parts in k order, 8 or 12 16-byte loads in flight per thread: a round trip to L2 is most of the cost
        constexpr int NP = GLU ? 2 : 6;
#pragma unroll 1
        for (int q0 = own ? c_first + 1 : c_first; q0 <= c_last; q0 += NP) {
          float4 a[NP][2], b[NP][2];
#pragma unroll
          for (int i = 0; i < NP; ++i) {
            const int q = q0 + i;
            const float4* src = reinterpret_cast<const float4*>(p.ws + ((size_t)q * 2 + (q == c_first ? 1 : 0)) * acc_cols * SK_BM) + n_in + (size_t)(c >> 2) * SK_BM;
#pragma unroll
            for (int k = 0; k < 2; ++k) {
              if (q <= c_last) a[i][k] = __ldcg(src + k * SK_BM);
              if (GLU && q <= c_last) b[i][k] = __ldcg(src + (size_t)((p.xb >> 2) + k) * SK_BM);
            }
          }
#pragma unroll
          for (int i = 0; i < NP; ++i) {
            if (q0 + i > c_last) break;
#pragma unroll
            for (int k = 0; k < 2; ++k) {
              g[4 * k] += a[i][k].x; g[4 * k + 1] += a[i][k].y; g[4 * k + 2] += a[i][k].z; g[4 * k + 3] += a[i][k].w;
              if (GLU) { up[4 * k] += b[i][k].x; up[4 * k + 1] += b[i][k].y; up[4 * k + 2] += b[i][k].z; up[4 * k + 3] += b[i][k].w; }
            }
          }
        }
        if constexpr (WT != 0) {
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            g[k] *= sg;
            if (GLU) up[k] *= su;
          }
        }
        if (GLU) {
          if (p.act == 4) {       // clamped, shifted gate product
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              const float gc = fminf(g[k] + bg, p.limit), uc = fminf(fmaxf(up[k] + bu, -p.limit), p.limit);
              g[k] = (uc + 1.f) * gc * (1.f / (1.f + __expf(-p.alpha * gc)));
            }
          } else if (p.act == 1) {
#pragma unroll
            for (int k = 0; k < 8; ++k) g[k] = silu(g[k] + bg) * (up[k] + bu);
          } else if (p.act == 2) {
#pragma unroll
            for (int k = 0; k < 8; ++k) g[k] = gelu_tanh(g[k] + bg) * (up[k] + bu);
          } else {
#pragma unroll
            for (int k = 0; k < 8; ++k) g[k] = gelu_erf(g[k] + bg) * (up[k] + bu);
          }
        } else {
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            g[k] += bg;
            if (p.residual) g[k] += __uint_as_float(res[k] << 16);
          }
        }
#pragma unroll
        for (int k = 0; k < 8; ++k)
          if (in && c + k < cnt) {
            if (p.y_f32) reinterpret_cast<float*>(p.y)[at + (size_t)k * p.n_out] = g[k];
            else reinterpret_cast<__nv_bfloat16*>(p.y)[at + (size_t)k * p.n_out] = __float2bfloat16(g[k]);
          }
      }
      if (own) {
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(&tmem_empty[buf]);
      }
    }
  }
  if (*stop) __nanosleep(1000000);        // gave up: let copies in flight land before the shared memory goes away
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 2) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(p.tmem_cols));
  }
}

typedef CUresult (*SkEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                               const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
// rows of K elements, `groups` boxes of 64 elements (128 bytes, also for byte elements) side by side in one copy; groups > 1: as {64, rows, K / 64}
static void sk_map(CUtensorMap* tm, const void* ptr, long long rows, int K, long long ld, int box_rows, bool bytes = false, int groups = 1) {
  static SkEncodeFn fn = [] {
    void* q = nullptr;
    cudaDriverEntryPointQueryResult r;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &q, cudaEnableDefault, &r) != cudaSuccess || q == nullptr)
      throw std::runtime_error("cuTensorMapEncodeTiled not available");
    return reinterpret_cast<SkEncodeFn>(q);
  }();
  const cuuint64_t es = bytes ? 1 : 2;
  cuuint64_t gdim[3] = {(cuuint64_t)(groups > 1 ? SK_BK : K), (cuuint64_t)rows, (cuuint64_t)(K / SK_BK)}, gstride[2] = {(cuuint64_t)ld * es, 128};
  cuuint32_t box[3] = {(cuuint32_t)(128 / es), (cuuint32_t)box_rows, (cuuint32_t)groups}, estr[3] = {1, 1, 1};
  CUresult r = fn(tm, bytes ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, groups > 1 ? 3 : 2, const_cast<void*>(ptr), gdim, gstride, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) throw std::runtime_error("cuTensorMapEncodeTiled (skinny gemm) failed: " + std::to_string((int)r));
}

static int sk_grid() {
  static int n = [] {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    return v;
  }();
  return n;
}
int skinny_gemm_rows(int tokens) { return std::max(16, (tokens + 15) / 16 * 16); }

// floats of partial tiles a launch may need
long long skinny_gemm_ws_floats(int tokens, bool glu) { return (long long)sk_grid() * 2 * skinny_gemm_rows(tokens) * (glu ? 2 : 1) * SK_BM; }
int skinny_gemm_tickets() { return sk_grid(); }

// one block between the kernel that produces x and the GEMM: the GEMM's CTAs are already filling their rings meanwhile
__global__ void __launch_bounds__(256) skinny_clear_kernel(unsigned* __restrict__ tickets, int n) {
  pdl_launch_dependents();
  pdl_wait();
  for (int i = threadIdx.x; i < n; i += 256) tickets[i] = 0u;
}
void skinny_clear_launch(unsigned* tickets, int n, cudaStream_t stream) { launch_pdl(skinny_clear_kernel, dim3(1), dim3(256), 0, stream, tickets, n); }

bool skinny_gemm8_supported(int tokens, int K, bool glu) { return tokens >= 1 && tokens <= (glu ? SKINNY_MAX_T / 2 : SKINNY8_MAX_T) && K % sk_bk(1, false) == 0; }
int skinny_gemm8_block(int tokens) { return (tokens + (tokens + SKINNY_MAX_T - 1) / SKINNY_MAX_T - 1) / ((tokens + SKINNY_MAX_T - 1) / SKINNY_MAX_T); }

void skinny_gemm_launch(const SkinnyGemm& a, cudaStream_t stream) {
  const bool glu = a.act != 0;
  if (a.K % SK_BK != 0 || a.tokens < 1 || (a.wt == 0 && a.tokens > SKINNY_MAX_T)) throw std::runtime_error("skinny gemm: K % 64 == 0, 1 .. 128 tokens per expert");
  if (a.wt != 0 && (!skinny_gemm8_supported(a.tokens, a.K, glu) || a.n_active != nullptr || a.scale == nullptr))
    throw std::runtime_error("skinny gemm, 8-bit weights: one weight with scales, K % 128 == 0, 1 .. 512 tokens (64 with a gate product)");
  SkinnyKernelParams p{};
  p.rows = glu ? 2 * a.n_out : a.n_out;
  p.xb = skinny_gemm_rows(a.wt ? skinny_gemm8_block(a.tokens) : a.tokens);
  const bool wide = a.wt == 0 && !glu && a.n_active == nullptr && a.K % 128 == 0;
  sk_map(&p.tm_w, a.w, (long long)a.experts * p.rows, a.K, a.K, SK_BM, a.wt != 0, wide ? 2 : 1);
  p.xbox = a.n_active ? 16 : p.xb;
  sk_map(&p.tm_x, a.x, a.x_rows, a.K, a.ldx, p.xbox, false, wide || a.wt ? 2 : 1);
  if (a.n_active) sk_map(&p.tm_x64, a.x, a.x_rows, a.K, a.ldx, 64);
  p.n_active = a.n_active; p.active = a.active; p.seg_start = a.seg_start; p.seg_count = a.seg_count;
  p.bias = reinterpret_cast<const __nv_bfloat16*>(a.bias);
  p.residual = reinterpret_cast<const __nv_bfloat16*>(a.residual);
  p.scale = a.scale; p.scale_step = a.scale_n > 1 ? 1 : 0;
  p.y = a.y; p.y_f32 = a.y_f32; p.ws = a.ws; p.tickets = a.tickets;
  p.T = a.tokens; p.n_out = a.n_out; p.K = a.K; p.act = a.act; p.limit = a.limit; p.alpha = a.alpha; p.w_fresh = a.w_fresh;
  check_waits();
  p.wait_word = wait_word(WAIT_SKINNY);
  count_launch(COUNT_SKINNY);
  const int stage = (glu || wide ? 2 : 1) * SK_W_BYTES + p.xb * sk_bk(a.wt, wide) * 2;
  p.stages = std::min(SK_MAX_STAGES, (SK_SMEM - 1024) / stage);       // (8-bit weights: at least SK_A_BUFS, asserted above)
  int cols = 32;
  while (cols < 2 * (glu ? 2 : 1) * p.xb + (a.wt ? SK_A_BUFS * SK_A_COLS : 0)) cols *= 2;
  p.tmem_cols = cols;
  const size_t smem = (size_t)p.stages * stage + 1024;
  auto go = [&](auto kernel) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SK_SMEM) != cudaSuccess)
      throw std::runtime_error("skinny gemm: shared memory size refused");
    launch_pdl(kernel, dim3(sk_grid()), dim3(SK_THREADS), smem, stream, p);
  };
  if (a.wt == 0) glu ? go(skinny_gemm_kernel<true, 0, false>) : wide ? go(skinny_gemm_kernel<false, 0, true>) : go(skinny_gemm_kernel<false, 0, false>);
  else if (a.wt == 1) glu ? go(skinny_gemm_kernel<true, 1, false>) : go(skinny_gemm_kernel<false, 1, false>);
  else glu ? go(skinny_gemm_kernel<true, 2, false>) : go(skinny_gemm_kernel<false, 2, false>);
}

// ---- routed experts of a small step -------------------------------------------------------------------------------------------------------
// One block per (token, slot) entry: its row among the entries sorted by (expert, entry) — counted, so the order is the same every time —
// and a copy of the token's row to that place.  Block 0 also writes the segments (an expert's rows, cut every seg_rows of them) and clears the tickets
// of the two GEMMs.
__global__ void __launch_bounds__(256) moe_small_gather_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ topk_w,
                                                               const int* __restrict__ topk_i, int id_step, int entries, int k, int H, int expert_offset, int e_local,
                                                               int seg_rows, int scale_input, __nv_bfloat16* __restrict__ xp, int* __restrict__ pos,
                                                               int* __restrict__ n_active, int* __restrict__ active, int* __restrict__ seg_start,
                                                               int* __restrict__ seg_count, unsigned* __restrict__ tickets, int n_tickets) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ int s_sum[8];
  const int i = blockIdx.x, tid = threadIdx.x;
  const int e = topk_i[(size_t)i * id_step] - expert_offset;
  const bool mine = e >= 0 && e < e_local;
  int before = 0;
  if (mine)
    for (int j = tid; j < entries; j += 256) {
      const int ej = topk_i[(size_t)j * id_step] - expert_offset;
      before += ej >= 0 && (ej < e || (ej == e && j < i));
    }
  before = __reduce_add_sync(0xffffffffu, before);
  if ((tid & 31) == 0) s_sum[tid >> 5] = before;
  __syncthreads();
  int row = 0;
  for (int w = 0; w < 8; ++w) row += s_sum[w];
  if (tid == 0) pos[i] = mine ? row : -1;
  if (mine) {
    const uint4* src = reinterpret_cast<const uint4*>(x + (size_t)(i / k) * H);
    uint4* dst = reinterpret_cast<uint4*>(xp + (size_t)row * H);
    const float w = scale_input ? topk_w[i] : 1.f;
    for (int v = tid; v < H / 8; v += 256) {
      uint4 q = ldg_act(src + v);
      if (scale_input)
        q = make_uint4(pack_bf16(bf16lo(q.x) * w, bf16hi(q.x) * w), pack_bf16(bf16lo(q.y) * w, bf16hi(q.y) * w),
                       pack_bf16(bf16lo(q.z) * w, bf16hi(q.z) * w), pack_bf16(bf16lo(q.w) * w, bf16hi(q.w) * w));
      dst[v] = q;
    }
  }
  if (i == 0) {
    __shared__ int s_cnt[512];
    for (int c = tid; c < e_local; c += 256) s_cnt[c] = 0;
    __syncthreads();
    for (int j = tid; j < entries; j += 256) {
      const int ej = topk_i[(size_t)j * id_step] - expert_offset;
      if (ej >= 0 && ej < e_local) atomicAdd(&s_cnt[ej], 1);
    }
    __syncthreads();
    if (tid < 32) {                       // exclusive scans of the counts and of the segments, 32 experts at a time
      int rows = 0, segs = 0;
      for (int c0 = 0; c0 < e_local; c0 += 32) {
        const int c = c0 + tid, n = c < e_local ? s_cnt[c] : 0;
        const int ns = (n + seg_rows - 1) / seg_rows;
        int incl = n, sincl = ns;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int t = __shfl_up_sync(0xffffffffu, incl, o), ts = __shfl_up_sync(0xffffffffu, sincl, o);
          if (tid >= o) {
            incl += t;
            sincl += ts;
          }
        }
        for (int j = 0, s = segs + sincl - ns; j < n; j += seg_rows, ++s) {
          active[s] = c;
          seg_start[s] = rows + incl - n + j;
          seg_count[s] = min(seg_rows, n - j);
        }
        rows += __shfl_sync(0xffffffffu, incl, 31);
        segs += __shfl_sync(0xffffffffu, sincl, 31);
      }
      if (tid == 0) *n_active = segs;
    }
    for (int t = tid; t < n_tickets; t += 256) tickets[t] = 0u;
  }
}

// out[token] = sum over slots of affinity * y[row of (token, slot)], fp32 rows, fixed slot order
__global__ void __launch_bounds__(256) moe_small_combine_kernel(const float* __restrict__ y, const float* __restrict__ topk_w, const int* __restrict__ pos,
                                                                __nv_bfloat16* __restrict__ out, int H, int k, int scale_input) {
  pdl_launch_dependents();
  pdl_wait();
  const int tok = blockIdx.y, v = blockIdx.x * 256 + threadIdx.x;
  if (v >= H / 4) return;
  float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int s = 0; s < k; ++s) {
    const int r = pos[tok * k + s];
    if (r < 0) continue;
    const float w = scale_input ? 1.f : topk_w[tok * k + s];
    const float4 q = __ldcg(reinterpret_cast<const float4*>(y + (size_t)r * H) + v);
    f.x += w * q.x; f.y += w * q.y; f.z += w * q.z; f.w += w * q.w;
  }
  *reinterpret_cast<uint2*>(out + (size_t)tok * H + v * 4) = make_uint2(pack_bf16(f.x, f.y), pack_bf16(f.z, f.w));
}

void moe_small_gather_launch(const void* x, const float* topk_w, const int* topk_i, int id_step, int entries, int k, int H, int expert_offset, int e_local,
                             int seg_rows, int scale_input, void* xp, int* pos, int* n_active, int* active, int* seg_start, int* seg_count, unsigned* tickets,
                             int n_tickets, cudaStream_t stream) {
  if (e_local > 512 || H % 8 != 0) throw std::runtime_error("moe (small step): at most 512 experts, hidden size % 8 == 0");
  launch_pdl(moe_small_gather_kernel, dim3(entries), dim3(256), 0, stream, reinterpret_cast<const __nv_bfloat16*>(x), topk_w, topk_i, id_step, entries, k, H,
             expert_offset, e_local, seg_rows, scale_input, reinterpret_cast<__nv_bfloat16*>(xp), pos, n_active, active, seg_start, seg_count, tickets, n_tickets);
}
void moe_small_combine_launch(const float* y, const float* topk_w, const int* pos, void* out, int N, int H, int k, int scale_input, cudaStream_t stream) {
  launch_pdl(moe_small_combine_kernel, dim3((H / 4 + 255) / 256, N), dim3(256), 0, stream, y, topk_w, pos, reinterpret_cast<__nv_bfloat16*>(out), H, k,
             scale_input);
}

}  // namespace nxdi
