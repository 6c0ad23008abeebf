// Flash attention over prompts on the 5th-generation tensor cores: S = Q K^T and O += P V are tcgen05.mma instructions whose accumulators
// AND whose probabilities live in TENSOR MEMORY; Q / K / V tiles arrive through TMA (SWIZZLE_128B); the softmax owns one query row per
// thread (tcgen05.ld of its TMEM lane), so no cross-thread reductions exist anywhere.
//
//   CTA = one or two 128-query tiles of one batch row (NX; the rule stands at fa_go).  Two tiles read the same keys: the same queries of two neighbouring
//   q heads of a kv head (grouped heads), or 256 consecutive queries of one head.  Per tile four softmax warps, then an MMA warp, a TMA warp, a warp
//   that zeroes the value rows past the end of a paged row (see below).
//   per 128-key tile j and query tile x:
//     S_x = Q_x K_j^T     D/16 x UMMA 128x128x16 (shared-memory operands)                      -> TMEM cols [128 x, 128 x + 128)
//     P_x = exp2(S_x c - m)   registers -> bf16 -> TMEM, over the first half of S_x (a thread has read its whole row before)
//     O_x += P_x V_j      8 x UMMA 128xDx16 with A = P_x from TMEM, B = V_j in its natural [key][d] layout = MN-major
//   Query tiles take turns: while one is in its softmax the tensor pipe works on P V and the next Q K^T of the other.  P is handed over in two
//   64-key halves: P V of the first runs while the second is exponentiated.
//   What bounds it: per pair of tiles (head size 128) the tensor pipe, the exponentials (16 per clock and SM) and shared memory each need
//   about 2048 clocks; measured about 3100: the chain scores -> maximum (450) -> exponentials (1500) -> second half of P V and Q K^T (900) of a tile, with
//   200 clocks for each hand-over.  One 8192-token prompt, 32 / 8 heads x 128: 0.44 ms alone (1.25 PFLOP/s).  Before: 0.495 ms; of that, 28 us from
//   the MMA warp's code (fa_umma), 27 us from the halves of P, 7 us from the mixed-type sums (fa_add_bf16x2), 20 us from masks outside the tiles
//   that need none.  3 x 1000 tokens of head size 64, window 128: 24 us, 30 before.
//   A soft cap (tanh) needs nine more fp32 pair operations per pair of scores; they run beside the exponentials, the maximum is taken before the cap and capped
//   alone.  Three portions with cap, gate and window: 208 us in a graph (254 before the gate came
//   through shared memory; 193 with a shorter polynomial up to half the cap, but 290 .. 340 for scores between that and the cap, which then take both).
//   Tried and slower: 64-key tiles with two score buffers per query tile (478 us: both tiles' softmax phases fall together, and a hand-over costs as
//   much per 64 keys); sixteen softmax warps with half a row per thread (482 us); a share of the exponentials as polynomials on the FMA pipe (2 of 16: no
//   gain, 4 of 16: 1 % slower: the fp32 pair operations cost more clocks than the exponentials they replace); the maximum beside the exponentials of
//   the maximum before (493 us); four hand-overs of P (439 us).
//   O and l are rescaled by the softmax warps themselves, decided per warp: S_j was issued after P V_{j-1}, so "S_j is complete" says that O
//   is quiescent.  Contiguous rows of head size 128 move their maximum only when it grows by more than 2^8; the others move it at once, as the
//   mma.sync kernels did that they ran on: then a row's largest probability is exactly 1 and takes no rounding (error against 64 bits of the mixed
//   portions below 2.249e-3, with the lazy maximum 2.337e-3, mma.sync 2.248e-3; 3 x 1000 tokens of head size 64 2.088e-3, 2.143e-3, and 2.059e-3
//   with that kernel's four maxima per row).  It costs 4 of 83 us at two portions of up to 969 tokens over contexts up to 2556 without a cap.
//
// Keys come from contiguous [B, T, Hkv, D] tensors or from a PAGED cache [blocks, page, Hkv, D] (page a power of two >= 8: a 128-key tile is
// 128 / page boxes, whose 1024-byte swizzle atoms line up).  Pages past the last visible key are not fetched, and the rows after it in the
// last tile are zeroed in shared memory before P V: probability 0 times whatever an unwritten cache row holds must stay 0.
// Masks are arguments: causal or bidirectional, sliding window with kept first tokens, chunks, per-head sink logit, tanh soft cap.
// reference kernel contract: attention_cte / flash_fwd (modules/attention/attention_base.py:603-630,722-744).
#include <algorithm>
#include <cfloat>
#include <stdexcept>
#include <string>
#include <type_traits>

#include "api.h"
#include "common.cuh"
#include "mbar_wait.cuh"
#include "seqmix.h"

namespace nxdi {

constexpr int FA_ROWS = 128;                   // queries per tile = keys per tile
constexpr int FA_SHORT = 6;                    // key tiles of a CTA that does not wait for the large code of a tile (capped_tile)
constexpr float FA_LOG2E = 1.4426950408889634f;

struct FaParams {
  CUtensorMap tm_q, tm_k, tm_v, tm_o;   // q / o (and contiguous k / v): 4-D {D, heads, T, B}; paged k / v: 3-D {D, kv heads, slots}; boxes of 64 columns
  CUtensorMap tm_g;                     // the gate, like q (gate_tma)
  const float* sinks;                   // [Hq] or null
  const float* head_scale;              // [Hq] or null: a further factor of the scores of a head
  const __nv_bfloat16* gate;            // [B, T, Hq * D] (or [B, T, Hq] with gate_per_head) with the strides below, or null
  long long g_sb, g_st;
  __nv_bfloat16* out;                   // [B, T, Hq, D]
  const int *ctx_len, *q_len, *block_table;   // paged rows
  int max_blocks, page_shift;
  int gate_per_head, gate_tma;
  int B, T, Hq, Hkv, causal, window, keep, chunk, pair_heads;
  float scale, softcap;
  unsigned* wait_word;                  // mbar_wait.cuh
};

__device__ __forceinline__ void fa_tma_4d(void* dst, const CUtensorMap* tm, int c0, int c1, int c2, int c3, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(mbar_s32(dst)),
               "l"(tm), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(mbar_s32(bar)) : "memory");
}
__device__ __forceinline__ void fa_tma_3d(void* dst, const CUtensorMap* tm, int c0, int c1, int c2, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(mbar_s32(dst)),
               "l"(tm), "r"(c0), "r"(c1), "r"(c2), "r"(mbar_s32(bar)) : "memory");
}
__device__ __forceinline__ void fa_tma_store_4d(const CUtensorMap* tm, const void* src, int c0, int c1, int c2, int c3) {
  asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%1, %2, %3, %4}], [%5];" ::"l"(tm), "r"(c0), "r"(c1), "r"(c2), "r"(c3),
               "r"(mbar_s32(src)) : "memory");
}
// K-major operand tile [rows][64 cols] of 128-byte rows, SWIZZLE_128B: 8-row groups 1024 B apart
__device__ __forceinline__ uint64_t fa_desc_kmajor(const void* smem) {
  uint64_t d = 0;
  d |= (uint64_t)((mbar_s32(smem) & 0x3FFFF) >> 4);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
// MN-major operand (V in its natural [key][d] layout): canonical SW128 layout ((8,8,m),(8,k)) : ((1,8,LBO),(64,SBO)) in 16-byte
// units — a 128-byte row holds 64 contiguous MN (= d) elements of ONE k (= key); 8 keys form a 1024-byte group (SBO);
// the second 64-column half of the tile sits LBO = 16 KB further.
__device__ __forceinline__ uint64_t fa_desc_mnmajor(const void* smem) {
  uint64_t d = 0;
  d |= (uint64_t)((mbar_s32(smem) & 0x3FFFF) >> 4);
  d |= (uint64_t)((FA_ROWS * 128) >> 4) << 16;       // leading byte offset: next 64-element block along MN
  d |= (uint64_t)(1024 >> 4) << 32;                  // stride byte offset: next 8-row (key) group
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
// instruction descriptor: D = f32, A = B = bf16, M = 128; bit 16 = B is MN-major
__host__ __device__ constexpr uint32_t fa_idesc(int n, bool b_mn_major) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (b_mn_major ? (1u << 16) : 0u) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}
// Called by a whole warp, issued by the lane whose `on` is 1: in code that all lanes run the descriptors stay in uniform registers.  (A branch
// for one lane moves each of them there before every instruction: the issuing thread, not the tensor pipe, was what a key tile waited for.)
__device__ __forceinline__ void fa_umma(uint32_t on, uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc) {
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
               "l"(da), "l"(db), "r"(idesc), "r"(acc), "r"(on) : "memory");
}
__device__ __forceinline__ void fa_umma_ts(uint32_t on, uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t idesc, uint32_t acc) {
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
               "r"(tmem_a), "l"(db), "r"(idesc), "r"(acc), "r"(on) : "memory");
}
__device__ __forceinline__ void fa_commit(uint32_t on, uint64_t* bar) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(mbar_s32(bar)),
               "r"(on) : "memory");
}
__device__ __forceinline__ uint32_t fa_elect() {
  uint32_t r;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r));
  return r;
}
__device__ __forceinline__ void fa_tmem_ld32(uint32_t taddr, uint32_t* v) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
        "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]),
        "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]),
        "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(taddr));
}
__device__ __forceinline__ void fa_tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]),
                 "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]) : "r"(taddr));
}
__device__ __forceinline__ void fa_tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]),
               "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
               : "memory");
}
__device__ __forceinline__ void fa_tmem_st32(uint32_t taddr, const uint32_t* v) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]),
      "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]),
      "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]),
      "r"(v[31])
      : "memory");
}

__device__ __forceinline__ float fa_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// 1 / (1 + e^-g) without a division: its branch for the ends of the range keeps the compiler from running several of them side by side (200 clocks each, one
// after the other).  The reciprocal's last bit comes from a Newton step, except where 1 + e^-g is infinite or nearly so.
__device__ __forceinline__ float fa_sigmoid(float g) {
  const float x = 1.f + expf(-g);
  float r;
  asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  const float n = fmaf(r, fmaf(-x, r, 1.f), r);
  return x < 0x1p126f ? n : r;
}
// two fp32 operations per instruction
__device__ __forceinline__ uint64_t fa_pack2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(__float_as_uint(a)), "r"(__float_as_uint(b)));
  return r;
}
__device__ __forceinline__ void fa_unpack2(uint64_t v, float& a, float& b) {
  uint32_t x, y;
  asm("mov.b64 {%0, %1}, %2;" : "=r"(x), "=r"(y) : "l"(v));
  a = __uint_as_float(x);
  b = __uint_as_float(y);
}
__device__ __forceinline__ uint64_t fa_fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t fa_mul2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
// s_lo, s_hi += the two bf16 halves of w
__device__ __forceinline__ void fa_add_bf16x2(float& s_lo, float& s_hi, uint32_t w) {
  asm("{\n\t.reg .b16 l, h;\n\tmov.b32 {l, h}, %2;\n\tadd.rn.f32.bf16 %0, l, %0;\n\tadd.rn.f32.bf16 %1, h, %1;\n\t}" : "+f"(s_lo), "+f"(s_hi) : "r"(w));
}
// tanh on |x| <= 1: x times a polynomial in x^2 (weighted least squares on Chebyshev nodes, relative error 1.7e-7 with fp32 arithmetic)
__device__ __forceinline__ uint64_t fa_tanh2_unit(uint64_t x) {
  const float t[7] = {0.00104102155f, -0.00620337576f, 0.0202899761f, -0.0534570292f, 0.13325204f, -0.333328396f, 0.99999994f};
  const uint64_t u = fa_mul2(x, x);
  uint64_t r = fa_pack2(t[0], t[0]);
#pragma unroll
  for (int i = 1; i < 7; ++i) r = fa_fma2(r, u, fa_pack2(t[i], t[i]));
  return fa_mul2(x, r);
}
// tanh on |x| > 1: 1 - 2 / (1 + e^2|x|), without the branches of tanhf
__device__ __forceinline__ float fa_tanh_large(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.f + fa_ex2(fabsf(x) * (2.f * FA_LOG2E))));
  return copysignf(fmaf(-2.f, r, 1.f), x);
}

template <int D, int NX>
struct FaShape {
  static constexpr int THREADS = 128 * NX + 128;
  static constexpr int TILE = FA_ROWS * D * 2;           // bytes of a [128][D] tile: D / 64 blocks of [128 rows][128 bytes]
  static constexpr int SLOTS = NX == 2 ? (D == 128 ? 5 : 8) : D == 128 ? 2 : 5;     // K and V tiles share one ring: K0 V0 K1 V1 ...
  static constexpr int SMEM = (NX + SLOTS) * TILE + 256 + 1024;                     // NX == 1: two CTAs per SM
};

// NX: query tiles of a CTA
template <int D, int NX, bool PAGED, bool CAP>
__global__ void __launch_bounds__(FaShape<D, NX>::THREADS, 3 - NX) attention_prefill_tc_kernel(const __grid_constant__ FaParams p) {
  constexpr int TILE = FaShape<D, NX>::TILE, SLOTS = FaShape<D, NX>::SLOTS, THREADS = FaShape<D, NX>::THREADS;
  constexpr int HALF = FA_ROWS * 128;
  constexpr int W_MMA = 4 * NX, W_TMA = W_MMA + 1, W_CLEAN = W_MMA + 2;
  constexpr uint32_t T_COLS = 256 * NX, T_OUT = 128 * NX;     // TMEM: S (and P) of every tile, then O
  constexpr float SLACK = D == 128 && !PAGED ? 8.f : 0.f; // log2 of what a row's largest probability may exceed 1 by
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  uint8_t* smem = smem_raw + ((1024u - (mbar_s32(smem_raw) & 1023u)) & 1023u);
  uint8_t* sQ = smem;                                    // [NX]; the outputs are staged here at the end
  uint8_t* sKV = sQ + NX * TILE;                         // [SLOTS]
  uint64_t* bars = reinterpret_cast<uint64_t*>(sKV + SLOTS * TILE);
  uint64_t* q_full = bars;
  uint64_t* kv_full = bars + 1;                          // [SLOTS]
  uint64_t* kv_empty = kv_full + SLOTS;                  // [SLOTS]
  uint64_t* s_full = kv_empty + SLOTS;                   // [2] S_x complete (and P V of the tile before retired)
  uint64_t* p_half = s_full + 2;                         // [2] P_x of the first 64 keys written and O_x rescaled: four warps arrive
  uint64_t* p_full = p_half + 2;                         // [2] the rest of P_x
  uint64_t* o_full = p_full + 2;                         // [2]
  uint64_t* v_landed = o_full + 2;                       // the last value tile is there
  uint64_t* v_clean = v_landed + 1;                      // its rows past the end are zeroed
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(v_clean + 1);
  volatile int* stop = reinterpret_cast<volatile int*>(tmem_slot + 1);

  if (warp == W_TMA && lane == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&p.tm_q) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&p.tm_k) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&p.tm_v) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&p.tm_o) : "memory");
    if (p.gate_tma) asm volatile("prefetch.tensormap [%0];" ::"l"(&p.tm_g) : "memory");
    mbar_init(q_full, 1);
    for (int s = 0; s < SLOTS; ++s) {
      mbar_init(&kv_full[s], 1);
      mbar_init(&kv_empty[s], 1);
    }
    for (int x = 0; x < 2; ++x) {
      mbar_init(&s_full[x], 1);
      mbar_init(&p_half[x], 4);
      mbar_init(&p_full[x], 4);
      mbar_init(&o_full[x], 1);
    }
    mbar_init(v_landed, 1);
    mbar_init(v_clean, 1);
    *stop = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == W_MMA) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(mbar_s32(tmem_slot)), "n"(T_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  pdl_launch_dependents();
  pdl_wait();               // from here on: what earlier kernels wrote

  // ---- which queries: heavy (late) tiles first
  const bool pair = NX == 2 && p.pair_heads;
  const int n_hp = pair ? p.Hq / 2 : p.Hq;
  const int span = pair ? FA_ROWS : NX * FA_ROWS;
  const int n_qt = (p.T + span - 1) / span;
  const int per_qt = p.B * n_hp;
  const int qt = n_qt - 1 - (int)(blockIdx.x / per_qt);
  const int bh = blockIdx.x % per_qt, b = bh / n_hp, hp = bh % n_hp;
  const int q0 = qt * span;
  const int qn = PAGED ? min(p.q_len[b], p.T) : p.T, ctx = PAGED ? p.ctx_len[b] : 0;
  if (PAGED && q0 >= qn) {                               // padding queries: zeros
    const int rows = min(span, p.T - q0), heads = pair ? 2 : 1, h0 = hp * heads;
    for (int i = threadIdx.x; i < rows * heads * (D / 8); i += THREADS) {
      const int r = i / (heads * (D / 8)), c = i % (heads * (D / 8));
      *reinterpret_cast<uint4*>(p.out + (((long long)b * p.T + q0 + r) * p.Hq + h0) * D + c * 8) = make_uint4(0u, 0u, 0u, 0u);
    }
    if (warp == W_MMA) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(T_COLS));
    return;
  }
  const int h_first = pair ? 2 * hp : hp, hk = h_first / (p.Hq / p.Hkv);
  // ---- which keys: the kept first tokens below the window's reach (whole tiles), then [lo, hi]
  const int p_first = ctx + q0, p_last = ctx + min(q0 + span, qn) - 1;
  const int hi = p.causal ? p_last : qn - 1, end = hi + 1;
  const int lo = p.window > 0 ? max(p_first - p.window + 1, 0) : p.chunk > 0 ? p_first / p.chunk * p.chunk : 0;
  const int keep = p.window > 0 ? p.keep : 0;
  const int t_lo = lo / FA_ROWS, nA = min((keep + FA_ROWS - 1) / FA_ROWS, t_lo);
  const int n_tiles = nA + hi / FA_ROWS - t_lo + 1;
  auto key_at = [&](int i) { return (i < nA ? i : t_lo + i - nA) * FA_ROWS; };
  const bool dirty_end = PAGED && (end & (FA_ROWS - 1)) != 0;

  if (warp >= W_MMA) {
    // registers: 384 threads x 168 at launch = 256 x 208 + 128 x 88; 256 x 128 = 128 x 200 + 128 x 56
    if constexpr (NX == 2) asm volatile("setmaxnreg.dec.sync.aligned.u32 88;");
    else asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    if (warp == W_TMA) {
      // ================= TMA producer =================
      const int pieces = PAGED ? max(1, FA_ROWS >> p.page_shift) : 1;    // boxes per 64-column block
      const int piece_rows = FA_ROWS / pieces;
      const int* table = PAGED ? p.block_table + (long long)b * p.max_blocks : nullptr;
      auto slot_at = [&](int key0) {                     // lane l: cache slot of the first key of piece l
        const int k = key0 + lane * piece_rows;
        if (!PAGED || lane >= pieces || k >= end) return 0;
        const int pi = min(k >> p.page_shift, p.max_blocks - 1);
        return (table[pi] << p.page_shift) + (k & ((1 << p.page_shift) - 1));
      };
      if (lane == 0) {
        mbar_expect(q_full, NX * TILE);
        for (int x = 0; x < NX; ++x)
          for (int c = 0; c < D / 64; ++c)
            fa_tma_4d(sQ + x * TILE + c * HALF, &p.tm_q, c * 64, pair ? h_first + x : h_first, pair ? q0 : q0 + x * FA_ROWS, b, q_full);
      }
      int next = slot_at(key_at(0));
      bool go = true;
      for (int i = 0; i < n_tiles && go; ++i) {
        const int key0 = key_at(i), cur = next;
        if (i + 1 < n_tiles) next = slot_at(key_at(i + 1));
        const int live = PAGED ? min(pieces, (end - key0 + piece_rows - 1) / piece_rows) : 1;
        for (int v = 0; v < 2 && go; ++v) {
          const int it = 2 * i + v, s = it % SLOTS;
          go = mbar_wait_warp(&kv_empty[s], (uint32_t)((it / SLOTS) & 1) ^ 1u, stop, p.wait_word);
          if (!go) break;
          uint8_t* dst = sKV + s * TILE;
          const CUtensorMap* tm = v ? &p.tm_v : &p.tm_k;
          if (lane == 0) mbar_expect(&kv_full[s], (uint32_t)(live * piece_rows * D * 2));
          if (PAGED) {
            for (int u = 0; u < live; ++u) {
              const int row = __shfl_sync(0xffffffffu, cur, u);
              if (lane == 0)
                for (int c = 0; c < D / 64; ++c) fa_tma_3d(dst + c * HALF + u * piece_rows * 128, tm, c * 64, hk, row, &kv_full[s]);
            }
          } else if (lane == 0) {
            for (int c = 0; c < D / 64; ++c) fa_tma_4d(dst + c * HALF, tm, c * 64, hk, key0, b, &kv_full[s]);
          }
        }
      }
      // the gate's tiles follow the last values through the ring: they are there when the epilogue starts
      for (int x = 0; x < NX && go && p.gate_tma; ++x) {
        const int it = 2 * n_tiles + x, s = it % SLOTS;
        go = mbar_wait_warp(&kv_empty[s], (uint32_t)((it / SLOTS) & 1) ^ 1u, stop, p.wait_word);
        if (!go || lane != 0) continue;
        mbar_expect(&kv_full[s], TILE);
        for (int c = 0; c < D / 64; ++c) fa_tma_4d(sKV + s * TILE + c * HALF, &p.tm_g, c * 64, pair ? h_first + x : h_first, pair ? q0 : q0 + x * FA_ROWS, b, &kv_full[s]);
      }
    } else if (warp == W_MMA) {
      // ================= MMA issuer =================
      constexpr uint32_t idesc_qk = fa_idesc(128, false), idesc_pv = fa_idesc(D, true);
      const uint32_t on = fa_elect();
      const uint64_t dq0 = fa_desc_kmajor(sQ), dk0 = fa_desc_kmajor(sKV), dv0 = fa_desc_mnmajor(sKV);
      int slot = 0;                                      // the ring's next tile
      uint32_t par = 0;
      auto full = [&] { return mbar_wait_warp(&kv_full[slot], par, stop, p.wait_word); };
      auto pop = [&] {
        if (++slot == SLOTS) {
          slot = 0;
          par ^= 1u;
        }
      };
      auto issue_s = [&](int x) {                        // S_x = Q_x K^T with the keys at `slot`
        const uint64_t dq = dq0 + (uint64_t)(x * (TILE >> 4)), dk = dk0 + (uint64_t)(slot * (TILE >> 4));
#pragma unroll
        for (int c = 0; c < D / 16; ++c) {
          // 16 d = 32 bytes inside the 128-byte swizzle atom; the second 64-d half is a separate 16 KB block
          const uint64_t off = (uint64_t)((c >> 2) * (HALF >> 4) + (c & 3) * 2);
          fa_umma(on, tmem + 128 * x, dq + off, dk + off, idesc_qk, c != 0 ? 1u : 0u);
        }
        fa_commit(on, &s_full[x]);
        if (x == NX - 1) fa_commit(on, &kv_empty[slot]);
      };
      bool go = mbar_wait_warp(q_full, 0, stop, p.wait_word) && full();
      if (go) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int x = 0; x < NX; ++x) issue_s(x);
        pop();
      }
      for (int i = 0; i < n_tiles && go; ++i) {
        const bool more = i + 1 < n_tiles;
        go = full();
        const int sv = slot;
        pop();
        if (go && dirty_end && !more) {
          if (lane == 0) mbar_arrive(v_landed);
          go = mbar_wait_warp(v_clean, 0, stop, p.wait_word);
        }
        const uint64_t dv = dv0 + (uint64_t)(sv * (TILE >> 4));
#pragma unroll
        for (int x = 0; x < NX; ++x) {
          // O_x += P_x V: A = P: 16 keys = 8 TMEM columns; B = V (MN-major): 16 keys = 16 rows of 128 bytes further in all blocks
          if (go) go = mbar_wait_warp(&p_half[x], (uint32_t)(i & 1), stop, p.wait_word);       // first half of P_x in TMEM, O_x rescaled, S_x fully read
          if (!go) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
          for (int c = 0; c < FA_ROWS / 32; ++c)
            fa_umma_ts(on, tmem + T_OUT + 128 * x, tmem + 128 * x + 8 * c, dv + (uint64_t)(c * 128), idesc_pv, (i | c) != 0 ? 1u : 0u);
          go = mbar_wait_warp(&p_full[x], (uint32_t)(i & 1), stop, p.wait_word);
          if (!go) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
          for (int c = FA_ROWS / 32; c < FA_ROWS / 16; ++c)
            fa_umma_ts(on, tmem + T_OUT + 128 * x, tmem + 128 * x + 8 * c, dv + (uint64_t)(c * 128), idesc_pv, 1u);
          if (x == NX - 1) fa_commit(on, &kv_empty[sv]);
          if (more) {
            if (x == 0) go = full();
            if (!go) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            issue_s(x);
            if (x == NX - 1) pop();
          } else {
            fa_commit(on, &o_full[x]);
          }
        }
      }
    } else if (warp == W_CLEAN && dirty_end) {
      // ================= value rows past the last key of the last tile =================
      const int valid = end - key_at(n_tiles - 1);
      if (mbar_wait_warp(v_landed, 0, stop, p.wait_word)) {
        uint8_t* v = sKV + ((2 * n_tiles - 1) % SLOTS) * TILE;
        for (int c = lane; c < (FA_ROWS - valid) * 8; c += 32)
#pragma unroll
          for (int hf = 0; hf < D / 64; ++hf) *reinterpret_cast<uint4*>(v + hf * HALF + valid * 128 + c * 16) = make_uint4(0u, 0u, 0u, 0u);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(v_clean);
      }
    }
  } else {
    // ================= softmax / rescale / epilogue: one query row per thread =================
    if constexpr (NX == 2) asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");
    else asm volatile("setmaxnreg.inc.sync.aligned.u32 200;");
    const int x = warp >> 2, qd = warp & 3;
    const int r = qd * 32 + lane;                        // row inside the tile = TMEM lane
    const int t_tile = pair ? q0 : q0 + x * FA_ROWS;
    const int h = pair ? h_first + x : h_first;
    const int t = t_tile + r, pos = ctx + t;             // token of the batch row, position in the sequence
    const uint32_t lanes = (uint32_t)(qd * 32) << 16;
    const uint32_t tS = tmem + 128 * x + lanes, tO = tmem + T_OUT + 128 * x + lanes;
    const int up = p.causal ? min(pos, end - 1) : end - 1;
    auto reach = [&](int at) { return p.window > 0 ? at - p.window + 1 : p.chunk > 0 ? at / p.chunk * p.chunk : 0; };
    const int lb = reach(pos);                           // a row sees [lb, up] and the first `keep` keys
    // bounds over the rows of this warp
    const int w_pos = ctx + t_tile + 32 * qd;
    const int up_min = p.causal ? min(w_pos, end - 1) : end - 1, up_max = p.causal ? min(w_pos + 31, end - 1) : end - 1;
    const int lb_min = reach(w_pos), lb_max = reach(w_pos + 31);
    const float hs = p.head_scale ? p.scale * p.head_scale[h] : p.scale;
    float m_run = -INFINITY, l_run = 0.f;
    // O = alpha O: P V of the tile before has retired
    auto rescale = [&](auto cols, float alpha) {
      constexpr int C = decltype(cols)::value;
#pragma unroll 1
      for (int c0 = 0; c0 < D; c0 += C) {
        uint32_t o[C];
#pragma unroll
        for (int c = 0; c < C; c += 32) fa_tmem_ld32(tO + c0 + c, o + c);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int e = 0; e < C; e += 2) {
          float a, d;
          fa_unpack2(fa_mul2(fa_pack2(__uint_as_float(o[e]), __uint_as_float(o[e + 1])), fa_pack2(alpha, alpha)), a, d);
          o[e] = __float_as_uint(a);
          o[e + 1] = __float_as_uint(d);
        }
#pragma unroll
        for (int c = 0; c < C; c += 32) fa_tmem_st32(tO + c0 + c, o + c);
      }
    };
    const float to_cap = CAP ? hs / p.softcap : 0.f;     // scores -> what the soft cap takes the tanh of
    const uint64_t tc2 = fa_pack2(to_cap, to_cap);
    auto tile = [&](auto masked, int i, int key0) {      // false: nothing done, scores beyond the cap
      constexpr bool MASKED = decltype(masked)::value;
      uint32_t v[128];
#pragma unroll
      for (int c = 0; c < 4; ++c) fa_tmem_ld32(tS + 32 * c, v + 32 * c);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      float scl = hs * FA_LOG2E;                         // scores -> log2 domain
      // halves of 64 keys that no row of the warp sees: probability 0 without looking at the scores
      bool dead[2] = {false, false};
      if constexpr (MASKED) {
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int k0 = key0 + 64 * c;
          dead[c] = k0 > up_max || (k0 + 63 < lb_min && k0 >= keep);
        }
      }
      if constexpr (CAP) {
        // v = score / cap from here on; the cap itself is taken beside the exponentials, the maximum's alone before them (it is increasing)
        float big[2] = {0.f, 0.f};
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          if (dead[c]) continue;
#pragma unroll
          for (int e = 64 * c; e < 64 * c + 64; e += 2) {
            float a, d;
            fa_unpack2(fa_mul2(fa_pack2(__uint_as_float(v[e]), __uint_as_float(v[e + 1])), tc2), a, d);
            v[e] = __float_as_uint(a);
            v[e + 1] = __float_as_uint(d);
            big[c] = fmaxf(big[c], fmaxf(fabsf(a), fabsf(d)));
          }
        }
        // Looked for over scores that the row does not see too (later keys, rows of pages that were not fetched, whatever shared memory held): both ways give a
        // score the same bits.
        if (__any_sync(0xffffffffu, !(fmaxf(big[0], big[1]) <= 1.f))) return false;
        scl = p.softcap * FA_LOG2E;
      } else if (!(scl > 0.f)) {                         // a head's factor may be zero or negative: the maximum below needs a positive scale
#pragma unroll
        for (int e = 0; e < 128; ++e) v[e] = __float_as_uint(__uint_as_float(v[e]) * scl);
        scl = 1.f;
      }
      uint32_t see[4] = {~0u, ~0u, ~0u, ~0u};
      if constexpr (MASKED) {
        // masks only where 32 keys are visible to some rows of the warp and not to others (a tile on the diagonal: one of four)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const int k0 = key0 + 32 * c;
          if (!(k0 + 31 <= up_min && (k0 >= lb_max || k0 + 31 < keep)) && !dead[c >> 1]) {
            const int e_hi = up - k0, e_lo = lb - k0, e_keep = keep - k0;
            const uint32_t m_hi = e_hi >= 31 ? ~0u : e_hi < 0 ? 0u : (2u << e_hi) - 1u;
            const uint32_t m_lo = e_lo <= 0 ? ~0u : e_lo > 31 ? 0u : ~0u << e_lo;
            const uint32_t m_keep = e_keep > 31 ? ~0u : e_keep <= 0 ? 0u : (1u << e_keep) - 1u;
            see[c] = m_hi & (m_lo | m_keep);
#pragma unroll
            for (int e = 0; e < 32; ++e)
              if (!(see[c] & (1u << e))) v[32 * c + e] = 0xff800000u;      // -inf
          }
        }
      }
      // row maximum in the domain of v (its scale is positive), four independent chains
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int c0 = 0; c0 < 128; c0 += 64) {
        if (dead[c0 >> 6]) continue;
#pragma unroll
        for (int e = c0; e < c0 + 64; e += 8)
#pragma unroll
          for (int c = 0; c < 4; ++c) mx4[c] = fmaxf(mx4[c], fmaxf(__uint_as_float(v[e + 2 * c]), __uint_as_float(v[e + 2 * c + 1])));
      }
      const float mx_raw = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
      float mx = (mx_raw == -INFINITY) ? -INFINITY : mx_raw * scl;
      if (CAP && mx_raw > -INFINITY) {
        float t, unused;
        fa_unpack2(fa_tanh2_unit(fa_pack2(mx_raw, mx_raw)), t, unused);
        mx = t * scl;
      }
      const bool grow = mx > m_run + SLACK || (m_run == -INFINITY && mx > -INFINITY);
      const float m_new = grow ? mx : m_run;
      const float alpha = (m_run == -INFINITY) ? 0.f : fa_ex2(m_run - m_new);
      const bool move = i > 0 && __any_sync(0xffffffffu, grow);

      m_run = m_new;
      if (SLACK > 0.f && move) rescale(std::integral_constant<int, 32>{}, alpha);       // seldom: in few registers, beside the scores
      // ---- P = exp2(v * scl - m) -> bf16 -> TMEM, over the scores, 64 keys at a time: their P V runs while the next are exponentiated
      const float neg_m = (m_run == -INFINITY) ? 0.f : -m_run;
      const uint64_t scl2 = fa_pack2(scl, scl), neg2 = fa_pack2(neg_m, neg_m);
      float ls[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t pk[32];
        if (dead[c]) {
#pragma unroll
          for (int e = 0; e < 32; ++e) pk[e] = 0u;
        } else {
#pragma unroll
          for (int e = 0; e < 64; e += 2) {
            const uint64_t v2 = fa_pack2(__uint_as_float(v[64 * c + e]), __uint_as_float(v[64 * c + e + 1]));
            float a, bb;
            fa_unpack2(fa_fma2(CAP ? fa_tanh2_unit(v2) : v2, scl2, neg2), a, bb);
            if (CAP && MASKED) {                         // the cap of a masked score is no -inf
              if (!(see[2 * c + (e >> 5)] & (1u << (e & 31)))) a = -INFINITY;
              if (!(see[2 * c + (e >> 5)] & (2u << (e & 31)))) bb = -INFINITY;
            }
            const uint32_t w = pack_bf16(fa_ex2(a), fa_ex2(bb));          // -inf -> 0
            // the sum uses the bf16-rounded probabilities, exactly what the tensor core multiplies
            fa_add_bf16x2(ls[e & 2], ls[(e & 2) + 1], w);
            pk[e >> 1] = w;
          }
        }
        fa_tmem_st32(tS + 32 * c, pk);
        if (SLACK == 0.f && c == 0 && move) rescale(std::integral_constant<int, 64>{}, alpha);      // often: in the registers of the first scores
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(c == 0 ? &p_half[x] : &p_full[x]);
      }
      l_run = fmaf(l_run, alpha, (ls[0] + ls[2]) + (ls[1] + ls[3]));
      return true;
    };
    // Soft cap, tiles with scores beyond the cap and CTAs of few key tiles: 64 or 32 keys at a time, the scores read from TMEM twice, in loops that are not unrolled
    // (the same bits).  Slower per tile once `tile` is in the instruction cache (254 against 207 us for the three portions named above), but a tenth of its code: four
    // portions of up to 287 tokens with a window of 500 38 us, 44 with `tile`; where an SM has one CTA alone (20 tokens: 16 CTAs) 27 and 25.  A window of up to a tile
    // leaves a warp two of six halves that it sees, and `tile` skips the others: 4 x 1024 tokens of head size 64, window 128, 45 us, 52 here (192: 59 and 57).
    // Scores up to twice the cap: 323 us, 1156 with a tanhf behind a branch for each of them in `tile`.
    auto capped_tile = [&](int i, int key0) {
      const float scl = p.softcap * FA_LOG2E;
      auto visible = [&](int k0) {                       // which of 32 keys this row sees
        const int e_hi = up - k0, e_lo = lb - k0, e_keep = keep - k0;
        const uint32_t m_hi = e_hi >= 31 ? ~0u : e_hi < 0 ? 0u : (2u << e_hi) - 1u;
        const uint32_t m_lo = e_lo <= 0 ? ~0u : e_lo > 31 ? 0u : ~0u << e_lo;
        const uint32_t m_keep = e_keep > 31 ? ~0u : e_keep <= 0 ? 0u : (1u << e_keep) - 1u;
        return m_hi & (m_lo | m_keep);
      };
      float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
      uint32_t any = 0u;
#pragma unroll 1
      for (int c = 0; c < 2; ++c) {
        const uint32_t see[2] = {visible(key0 + 64 * c), visible(key0 + 64 * c + 32)};
        any |= see[0] | see[1];
        uint32_t v[64];
        fa_tmem_ld32(tS + 64 * c, v);
        fa_tmem_ld32(tS + 64 * c + 32, v + 32);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int e = 0; e < 64; ++e) v[e] = __float_as_uint(__uint_as_float(v[e]) * to_cap);
        if (__any_sync(0xffffffffu, (see[0] & see[1]) != ~0u)) {
#pragma unroll
          for (int e = 0; e < 64; ++e)
            if (!(see[e >> 5] & (1u << (e & 31)))) v[e] = 0xff800000u;      // -inf
        }
#pragma unroll
        for (int e = 0; e < 64; e += 8)
#pragma unroll
          for (int k = 0; k < 4; ++k) m4[k] = fmaxf(m4[k], fmaxf(__uint_as_float(v[e + 2 * k]), __uint_as_float(v[e + 2 * k + 1])));
      }
      const float mx_raw = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3]));
      // the cap is increasing: the maximum alone is capped.  A row that sees keys has one, of scores below fp32's range too: -cap
      float mx;
      {
        float a, unused;
        fa_unpack2(fa_tanh2_unit(fa_pack2(mx_raw, mx_raw)), a, unused);
        mx = any != 0u ? (fabsf(mx_raw) <= 1.f ? a : fa_tanh_large(mx_raw)) * scl : -INFINITY;
      }
      const bool grow = mx > m_run + SLACK || (m_run == -INFINITY && mx > -INFINITY);
      const float m_new = grow ? mx : m_run;
      const float alpha = (m_run == -INFINITY) ? 0.f : fa_ex2(m_run - m_new);
      if (i > 0 && __any_sync(0xffffffffu, grow)) rescale(std::integral_constant<int, 32>{}, alpha);

      m_run = m_new;
      const float neg_m = (m_run == -INFINITY) ? 0.f : -m_run;
      const uint64_t scl2 = fa_pack2(scl, scl), neg2 = fa_pack2(neg_m, neg_m);
      float ls[4] = {0.f, 0.f, 0.f, 0.f};
      uint32_t v[32];
      fa_tmem_ld32(tS, v);
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        const uint32_t see = visible(key0 + 32 * c);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        float t[32], big = 0.f;
#pragma unroll
        for (int e = 0; e < 32; e += 2) {
          float a, d;
          const uint64_t y = fa_mul2(fa_pack2(__uint_as_float(v[e]), __uint_as_float(v[e + 1])), tc2);
          fa_unpack2(y, a, d);
          fa_unpack2(fa_tanh2_unit(y), t[e], t[e + 1]);
          big = fmaxf(big, fmaxf(fabsf(a), fabsf(d)));
        }
        if (__any_sync(0xffffffffu, !(big <= 1.f))) {
#pragma unroll
          for (int e = 0; e < 32; ++e) {
            const float a = __uint_as_float(v[e]) * to_cap, la = fa_tanh_large(a);
            t[e] = fabsf(a) <= 1.f ? t[e] : la;
          }
        }
        if (c < 3) fa_tmem_ld32(tS + 32 * c + 32, v);      // the next scores, beside the exponentials
        if (__any_sync(0xffffffffu, see != ~0u)) {
#pragma unroll
          for (int e = 0; e < 32; ++e)
            if (!(see & (1u << e))) t[e] = -INFINITY;
        }
        uint32_t pk[16];
#pragma unroll
        for (int e = 0; e < 32; e += 2) {
          float a, d;
          fa_unpack2(fa_fma2(fa_pack2(t[e], t[e + 1]), scl2, neg2), a, d);
          const uint32_t w = pack_bf16(fa_ex2(a), fa_ex2(d));          // -inf -> 0
          fa_add_bf16x2(ls[e & 2], ls[(e & 2) + 1], w);
          pk[e >> 1] = w;
        }
        fa_tmem_st16(tS + 16 * c, pk);
        if (c & 1) {
          asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(c == 1 ? &p_half[x] : &p_full[x]);
        }
      }
      l_run = fmaf(l_run, alpha, (ls[0] + ls[2]) + (ls[1] + ls[3]));
    };
    // (a choice for the whole launch, but for the row's number of tiles: CTAs of both kinds on an SM fetch both codes)
    bool large = n_tiles <= FA_SHORT && !(p.window > 0 && p.window <= FA_ROWS) && gridDim.x > kNumSMs;      // or a tile of this warp had scores beyond the cap: no more tries
    for (int i = 0; i < n_tiles; ++i) {
      const int key0 = key_at(i);
      if (!mbar_wait_warp(&s_full[x], (uint32_t)(i & 1), stop, p.wait_word)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      // masks only in a tile that has keys which some row of the warp does not see
      const bool plain = key0 + FA_ROWS - 1 <= up_min && (key0 >= lb_max || key0 + FA_ROWS <= keep);
      if constexpr (CAP) {
        if (!large) large = !(plain ? tile(std::false_type{}, i, key0) : tile(std::true_type{}, i, key0));
        if (large) capped_tile(i, key0);
      } else if (plain) {
        tile(std::false_type{}, i, key0);
      } else {
        tile(std::true_type{}, i, key0);
      }
    }
    // ---- epilogue: O / l (times the gate) -> bf16 -> shared memory -> TMA store (rows past T are clipped, padding rows are zeros)
    bool done = mbar_wait_warp(&o_full[x], 0, stop, p.wait_word);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    float l = l_run;
    if (p.sinks != nullptr) l = (m_run == -INFINITY) ? 1.f : l + fa_ex2(p.sinks[h] * FA_LOG2E - m_run);
    float inv = (m_run == -INFINITY || l == 0.f) ? 0.f : 1.f / l;
    const bool live_row = t < qn;
    const uint32_t live_mask = live_row ? ~0u : 0u;
    uint8_t* so = sQ + x * TILE + r * 128;
    auto put = [&](int col, const float (&f)[8]) {       // 16-byte chunk of the 128-byte row, XOR-swizzled like TMA does
      // (the choice is made on the packed words: one per element puts each sigmoid behind a branch of its own)
      *reinterpret_cast<uint4*>(so + (col >> 6) * HALF + ((((col & 63) >> 3) ^ (r & 7)) << 4)) =
          make_uint4(pack_bf16(f[0], f[1]) & live_mask, pack_bf16(f[2], f[3]) & live_mask, pack_bf16(f[4], f[5]) & live_mask, pack_bf16(f[6], f[7]) & live_mask);
    };
    const __nv_bfloat16* gp = nullptr;
    if (p.gate != nullptr && live_row) {
      gp = p.gate + (long long)b * p.g_sb + (long long)t * p.g_st + (p.gate_per_head ? h : h * D);
      if (p.gate_per_head) inv *= 1.f / (1.f + expf(-__bfloat162float(*gp)));
    }
    if (p.gate != nullptr && !p.gate_per_head) {
      // The gate's tile is in shared memory, and the sigmoids of 16 columns run side by side; read from global memory where it is used, with a branch per
      // element (for the division and for padding rows), the gate took 13 us of a CTA's last 16 (now 4.5; no gate: 0.9).
      const int it = 2 * n_tiles + x;
      const uint8_t* sg = sKV + (it % SLOTS) * TILE + r * 128;
      if (p.gate_tma) done = mbar_wait_warp(&kv_full[it % SLOTS], (uint32_t)((it / SLOTS) & 1), stop, p.wait_word) && done;
#pragma unroll 1
      for (int c0 = 0; c0 < D; c0 += 16) {
        uint32_t o[16], w[8];
        fa_tmem_ld16(tO + c0, o);
        if (p.gate_tma) {
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const uint4 q = *reinterpret_cast<const uint4*>(sg + (c0 >> 6) * HALF + (((((c0 & 63) >> 3) + k) ^ (r & 7)) << 4));
            w[4 * k] = q.x; w[4 * k + 1] = q.y; w[4 * k + 2] = q.z; w[4 * k + 3] = q.w;
          }
        } else {
#pragma unroll
          for (int k = 0; k < 8; ++k) w[k] = live_row ? ldg_act_u16(gp + c0 + 2 * k) | ldg_act_u16(gp + c0 + 2 * k + 1) << 16 : 0u;
        }
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int k = 0; k < 16; k += 8) {
          float f[8];
#pragma unroll
          for (int e = 0; e < 8; e += 2) {
            f[e] = __uint_as_float(o[k + e]) * inv * fa_sigmoid(bf16lo(w[(k + e) >> 1]));
            f[e + 1] = __uint_as_float(o[k + e + 1]) * inv * fa_sigmoid(bf16hi(w[(k + e) >> 1]));
          }
          put(c0 + k, f);
        }
      }
    } else {
#pragma unroll 1
      for (int c0 = 0; c0 < D; c0 += 32) {
        uint32_t o[32];
        fa_tmem_ld32(tO + c0, o);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int e = 0; e < 32; e += 8) {
          float f[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) f[k] = __uint_as_float(o[e + k]) * inv;
          put(c0 + e, f);
        }
      }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("bar.sync %0, 128;" ::"r"(1 + x) : "memory");
    if (r == 0 && done && t_tile < p.T) {
      for (int c = 0; c < D / 64; ++c) fa_tma_store_4d(&p.tm_o, sQ + x * TILE + c * HALF, c * 64, h, t_tile, b);
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    }
  }
  if (*stop) __nanosleep(1000000);        // gave up: let copies in flight land before the shared memory goes away
  __syncthreads();
  if (warp == W_MMA) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(T_COLS));
  }
}

typedef CUresult (*FaEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                               const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static FaEncodeFn fa_encode_fn() {
  static FaEncodeFn fn = [] {
    void* q = nullptr;
    cudaDriverEntryPointQueryResult r;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &q, cudaEnableDefault, &r) != cudaSuccess || q == nullptr)
      throw std::runtime_error("cuTensorMapEncodeTiled not available");
    return reinterpret_cast<FaEncodeFn>(q);
  }();
  return fn;
}
// dims / strides in elements of bf16, innermost first (its stride is 1); boxes of 64 columns x `rows` entries of dimension 2
static void fa_make_map(CUtensorMap* tm, const void* ptr, int rank, const long long* dims, const long long* strides, int rows) {
  cuuint64_t gdim[4], gstride[3];
  cuuint32_t box[4] = {64, 1, (cuuint32_t)rows, 1}, estr[4] = {1, 1, 1, 1};
  for (int i = 0; i < rank; ++i) gdim[i] = (cuuint64_t)dims[i];
  for (int i = 1; i < rank; ++i) gstride[i - 1] = (cuuint64_t)strides[i] * 2;
  CUresult r = fa_encode_fn()(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (cuuint32_t)rank, const_cast<void*>(ptr), gdim, gstride, box, estr,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) throw std::runtime_error("cuTensorMapEncodeTiled (attention) failed: " + std::to_string((int)r));
}
static void fa_map_rows(CUtensorMap* tm, const void* ptr, int B, int T, int H, int D) {      // [B, T, H, D]
  const long long dims[4] = {D, H, T, B}, strides[4] = {1, D, (long long)H * D, (long long)T * H * D};
  fa_make_map(tm, ptr, 4, dims, strides, FA_ROWS);
}

template <int D, int NX, bool PAGED, bool CAP>
static void fa_run(FaParams& p, cudaStream_t stream) {
  using Shape = FaShape<D, NX>;
  auto kernel = attention_prefill_tc_kernel<D, NX, PAGED, CAP>;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Shape::SMEM) != cudaSuccess)
    throw std::runtime_error("attention (tensor cores): shared memory size refused");
  check_waits();
  p.wait_word = wait_word(WAIT_ATTENTION);
  count_launch(COUNT_ATTENTION);
  if (NX == 2) count_launch(COUNT_ATTENTION_TWO);
  // grouped heads share their keys two by two; a head of its own takes 256 queries instead
  p.pair_heads = (p.Hq / p.Hkv) % 2 == 0 ? 1 : 0;
  const bool pair = NX == 2 && p.pair_heads;
  const int span = pair ? FA_ROWS : NX * FA_ROWS;
  const long long blocks = (long long)((p.T + span - 1) / span) * p.B * (pair ? p.Hq / 2 : p.Hq);
  launch_pdl(kernel, dim3((unsigned)blocks), dim3(Shape::THREADS), Shape::SMEM, stream, p);
}
// One query tile per CTA and two CTAs per SM where a tile reads few keys (a CTA's first loads, its epilogue and its masks then overlap the other's
// work), or where pairs of tiles would not fill the SMs; two tiles per CTA, which share the keys they load, for long rows.  us, two tiles / one, 32 / 8
// heads x 128, causal: 512 tokens 15.0 / 13.3, 4 x 1024 57.4 / 53.1, 2048 41.3 / 42.4, 8192 444 / 481; 2 x 3000 with a window of 128 67.8 / 59.9, 8192 with
// 1024 161 / 160; 8 / 1 heads, 4096: 63.1 / 58.4 (128 CTAs of two tiles).  Head size 64: 13.1 / 11.5, 48.0 / 45.2, 36.5 / 38.3; 49.5 / 43.7, 143 / 138.
template <int D, bool PAGED, bool CAP>
static void fa_go(FaParams& p, long long keys, cudaStream_t stream) {
  if (p.window > 0) keys = std::min(keys, (long long)p.window + p.keep + FA_ROWS);
  else if (p.chunk > 0) keys = std::min(keys, (long long)p.chunk + FA_ROWS);
  const bool pair = (p.Hq / p.Hkv) % 2 == 0;
  const long long blocks = pair ? (long long)((p.T + FA_ROWS - 1) / FA_ROWS) * p.B * (p.Hq / 2) : (long long)((p.T + 2 * FA_ROWS - 1) / (2 * FA_ROWS)) * p.B * p.Hq;
  if (keys <= 9 * FA_ROWS || blocks < kNumSMs) fa_run<D, 1, PAGED, CAP>(p, stream);
  else fa_run<D, 2, PAGED, CAP>(p, stream);
}

// q [B,T,Hq,D], k / v [B,T,Hkv,D] bf16 contiguous, D = 128, or 64 without a soft cap -> out [B,T,Hq,D]
void attention_prefill_tc_launch(const void* q, const void* k, const void* v, void* out, const float* sinks, int B, int T, int Hq, int Hkv, int D,
                                 float scale, int causal, int window, float softcap, cudaStream_t stream) {
  if (B <= 0 || T <= 0) return;
  FaParams p{};
  fa_map_rows(&p.tm_q, q, B, T, Hq, D);
  fa_map_rows(&p.tm_k, k, B, T, Hkv, D);
  fa_map_rows(&p.tm_v, v, B, T, Hkv, D);
  fa_map_rows(&p.tm_o, out, B, T, Hq, D);
  p.out = reinterpret_cast<__nv_bfloat16*>(out);
  p.sinks = sinks;
  p.B = B; p.T = T; p.Hq = Hq; p.Hkv = Hkv; p.causal = causal; p.window = window;
  p.scale = scale; p.softcap = softcap;
  if (D == 128 && softcap > 0.f) fa_go<128, false, true>(p, T, stream);
  else if (D == 128) fa_go<128, false, false>(p, T, stream);
  else if (D == 64 && softcap <= 0.f) fa_go<64, false, false>(p, T, stream);
  else throw std::runtime_error("attention (tensor cores): head size 128, or 64 without a soft cap");
}

// Prompt portions over a paged cache.  Sizes this kernel takes: keys and values of one size, 64 or 128, rows on 16-byte boundaries, pages of
// 2^k >= 8 tokens (smaller ones would break the 8-row swizzle atoms), no distance term; the rest is paged_window_attention_mma_kernel's.
// 3 rows of up to 1024 tokens over contexts up to 3000, 32 / 8 heads x 128, window 2048, cap, gate: 0.21 ms, mma.sync kernel 0.89 ms.
bool paged_attention_tc_supported(const WindowAttnParams& p, bool lp) {
  return lp && p.T >= 16 && p.maps != 2 && p.slopes == nullptr && p.D == p.Dv && (p.D == 64 || p.D == 128) && (p.v_rs * 2) % 16 == 0 && p.page >= 8 &&
         (p.page & (p.page - 1)) == 0 && (long long)p.B * p.Hq * ((p.T + FA_ROWS - 1) / FA_ROWS) <= 0x7fffffffLL &&
         (reinterpret_cast<uintptr_t>(p.q) | reinterpret_cast<uintptr_t>(p.k_cache) | reinterpret_cast<uintptr_t>(p.v_cache)) % 16 == 0;
}
void paged_attention_tc_launch(const WindowAttnParams& w, long long slots, cudaStream_t stream) {
  FaParams p{};
  fa_map_rows(&p.tm_q, w.q, w.B, w.T, w.Hq, w.D);
  fa_map_rows(&p.tm_o, w.out, w.B, w.T, w.Hq, w.D);
  const long long kd[3] = {w.D, w.G, slots}, ks[3] = {1, w.D, (long long)w.G * w.D}, vs[3] = {1, w.v_rs, w.G * w.v_rs};
  fa_make_map(&p.tm_k, w.k_cache, 3, kd, ks, std::min(w.page, FA_ROWS));
  fa_make_map(&p.tm_v, w.v_cache, 3, kd, vs, std::min(w.page, FA_ROWS));
  p.out = reinterpret_cast<__nv_bfloat16*>(w.out);
  p.sinks = w.sinks; p.head_scale = w.head_scale;
  p.gate = reinterpret_cast<const __nv_bfloat16*>(w.gate); p.g_sb = w.g_sb; p.g_st = w.g_st; p.gate_per_head = w.gate_per_head;
  const long long g_sb = w.B == 1 ? w.T * w.g_st : w.g_sb;
  p.gate_tma = w.gate != nullptr && !w.gate_per_head && reinterpret_cast<uintptr_t>(w.gate) % 16 == 0 && g_sb > 0 && g_sb % 8 == 0 && w.g_st > 0 && w.g_st % 8 == 0 ? 1 : 0;
  if (p.gate_tma) {
    const long long gd[4] = {w.D, w.Hq, w.T, w.B}, gs[4] = {1, w.D, w.g_st, g_sb};
    fa_make_map(&p.tm_g, w.gate, 4, gd, gs, FA_ROWS);
  }
  p.ctx_len = w.ctx_len; p.q_len = w.q_len; p.block_table = w.block_table; p.max_blocks = w.max_blocks;
  while ((1 << p.page_shift) < w.page) ++p.page_shift;
  p.B = w.B; p.T = w.T; p.Hq = w.Hq; p.Hkv = w.G; p.causal = 1; p.window = w.window; p.keep = w.keep_first; p.chunk = w.chunk;
  p.scale = w.scale; p.softcap = w.softcap;
  const bool cap = w.softcap > 0.f;
  const long long keys = (long long)w.max_blocks * w.page;       // contexts are known on the device alone
  if (w.D == 128) { if (cap) fa_go<128, true, true>(p, keys, stream); else fa_go<128, true, false>(p, keys, stream); }
  else { if (cap) fa_go<64, true, true>(p, keys, stream); else fa_go<64, true, false>(p, keys, stream); }
}

}  // namespace nxdi
