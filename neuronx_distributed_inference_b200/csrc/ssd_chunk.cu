// Mamba-2 recurrence over prompts in chunks of 64 tokens on tcgen05 (state size 128, head size 64, heads of a group in pairs); the step-by-step
// kernels of seqmix.cu keep every other shape, short rows and decode.  With cs the running sum of log2(decay) inside a chunk, dt the step sizes, S the state:
//
//   y_t   = 2^cs_t S^T C_t  +  sum_{s <= t} (C_t . B_s) 2^(cs_t - cs_s) dt_s x_s  +  D x_t,  times silu(z_t)
//   S'    = 2^cs_end S  +  sum_s dt_s 2^(cs_end - cs_s) B_s x_s^T
//
// Precision is that of fp32: every operand of a product is an exact sum of three bf16 parts (8 + 8 + 8 bits), six of the nine part products are taken
// (the three left out are below 2^-24 of a term), small ones first, sums in the fp32 accumulators over at most 128 terms; decays, the state and everything
// around the products stay fp32, the running sum of the exponents is taken in 64 bits (a chunk's exponents reach -200, neighbours differ by 1e-2).
//
//   prepare  (chunk, group, row): the parts of B and C as images of their shared-memory tiles, G = C B^T in fp32 on the CUDA cores, and the largest |G|, infinite
//            where a value of B or C is large or no number (64 heads share them)
//   scan     CTA = two heads of a row, the longest rows first, chunks in order.  128 rows of the products = (head, channel) = TMEM lanes:
//              update  W[(h,p)][n]  = X~^T B      A = the parts of dt 2^(cs_end - cs) x in TMEM, B image MN-major           K = 64
//              inter   I[(h,p)][t]  = S^T C^T     A = the parts of the state in TMEM, C image K-major                       K = 128
//              intra   W[(h,p)][(h,t)] = X^T M^T  A = the parts of x in shared memory, MN-major, M = masked G 2^.. dt + D of both heads as 128 columns  K = 64
//            8 warps hold the state (64 values a thread) and form its parts and those of x~, 4 warps form M and the parts of x, 8 warps finish the outputs,
//            one warp issues the MMAs, one the copies, two (one per head) the step sizes and exponents.
//   What bounds it: the chain of a chunk, about 9000 clocks: update (1500 and a hand-over), the state's parts (2500), inter and intra (3100), outputs (1400); the
//   96 MMAs alone are 4600.  us, here / step by step: 64 heads, state 128, 4 rows of up to 1024 tokens 107 / 423, one row of 1024 89 / 254, of 128 27 / 41,
//   4 rows of 64 23.5 / 37.5, one of 48 23 / 22 (the host); 128 heads in 8 groups, 4 rows of up to 1024 207 / 734.  Error against 64 bits, 4 rows of up to
//   1024: 1.0e-7, step by step 1.1e-7.  Tried: everything unrolled 217 us (2.3 warps waiting for instructions at every issue); four warps for
//   the outputs 142; conditional loads of x, z 136 and more (the compiler waits for each).
//   Rows of few tokens (a serving step puts one token of every running request beside a prompt portion) run step by step (ssd_steps.cuh), four groups of 128 threads
//   per CTA, and the longest rows start first.  us, here / all rows in chunks, in their order / all step by step, 64 heads, one-token rows beside a portion:
//     32 and 48 tokens 90 / 106 / 82     32 and 128 96 / 119 / 119     32 and 256 104 / 137 / 174     64 and 48 151 / 184 / 139     64 and 512 209 / 295 / 414
//     8 and 256 49 / 59 / 121            12 rows of 48 to 1024 160 / 201 / 666.   128 heads in 8 groups: 32 and 48 154 / 193 / 141, 64 and 512 405 / 549 / 588
//   Bound by the state's bytes (32 KB a head, in and out) and a CTA's start; the next row's state comes to the L2 meanwhile (4 to 8 us of the 151).  The code of these
//   rows stands behind that of the chunks: in front of it, every first launch fetched it from memory (4 us).
//   A chunk runs step by step in the state's warps where x, dt x, B, C, the state or a bound of M (largest |G| times dt, and D) is 1e18 or more or no number: a product
//   with 0 must not spread what is not finite to earlier tokens, and products that the recurrence does not form (C B^T before it meets x, S^T C before S has
//   decayed) must not leave fp32's range where its own values do not.
// The chunked form: Dao and Gu, "Transformers are SSMs" (2024), section 6.
#include <cuda_bf16.h>
#include <math.h>

#include <algorithm>
#include <stdexcept>
#include <string>

#include "api.h"
#include "common.cuh"
#include "mbar_wait.cuh"
#include "seqmix.h"
#include "ssd_steps.cuh"

namespace nxdi {
namespace {

constexpr int SQ = 64, SN = 128, SP = 64;                 // tokens of a chunk, state size, head size
constexpr int S_IMG = 3 * SQ * SN * 2, S_PART = SQ * SN * 2, S_BLK = SQ * 128;      // image of B or C; of one part; of 64 columns of a part
constexpr int S_G = SQ * SQ * 4;
constexpr int S_WS = 2 * S_IMG + S_G;                     // workspace of a (row, chunk, group): B, C, G
constexpr int SC_THREADS = 768;
constexpr int W_M = 8, W_OUT = 12, W_MMA = 20, W_COPY = 21, W_STEP = 22;             // first warps of the roles; the state's are 0 .. 7
constexpr uint32_t TM_I = 0, TM_W = 64, TM_S = 192, TM_X = 384;      // TMEM columns: inter, update / intra, state parts, x~ parts
constexpr float S_LARGE = 1e18f;                          // 128 products of two values below it stay in fp32's range

// two values -> their three bf16 parts.  w - v of a bf16 w and a fp32 v is one mixed-type instruction; it is the negative of what is left, so the
// middle part comes out negated
__device__ __forceinline__ void parts2(float a, float b, uint32_t& w0, uint32_t& w1, uint32_t& w2) {
  auto left = [](uint32_t w, float& x, float& y) {
    asm("{\n\t.reg .b16 l, h;\n\tmov.b32 {l, h}, %2;\n\tsub.rn.f32.bf16 %0, l, %0;\n\tsub.rn.f32.bf16 %1, h, %1;\n\t}" : "+f"(x), "+f"(y) : "r"(w));
  };
  w0 = pack_bf16(a, b);
  left(w0, a, b);
  const uint32_t m = pack_bf16(a, b);
  left(m, a, b);
  w1 = m ^ 0x80008000u;
  w2 = pack_bf16(a, b);
}
// eight values of a row -> 16 bytes in each of the three part tiles
__device__ __forceinline__ void store_parts(uint8_t* dst, int part, const float (&v)[8]) {
  uint32_t w[3][4];
#pragma unroll
  for (int k = 0; k < 4; ++k) parts2(v[2 * k], v[2 * k + 1], w[0][k], w[1][k], w[2][k]);
#pragma unroll
  for (int q = 0; q < 3; ++q) *reinterpret_cast<uint4*>(dst + q * part) = make_uint4(w[q][0], w[q][1], w[q][2], w[q][3]);
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// z / (1 + e^-z), the reciprocal with one step of Newton's method.  For |z| <= 80 e^-z = 2^t (1 + rest ln 2), t and rest the parts of -z log2(e), which is rounded
// to two fp32 terms (Cody and Waite's reduction)
constexpr float SILU_FAST = 80.f;
__device__ __forceinline__ float silu_fast(float z) {
  const float t = z * -1.44269502f, rest = fmaf(z, -1.44269502f, -t) + z * -1.92596303e-8f;
  const float d = 1.f + ex2(t) * fmaf(rest, 0.69314718f, 1.f);
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  r = fmaf(fmaf(-d, r, 1.f), r, r);
  return z * r;
}
// any z, from e^-|z|: nothing leaves the range on the way to the definition's values (-inf: not a number)
__device__ __forceinline__ float silu_any(float z) {
  const float q = expf(-fabsf(z)), d = 1.f + q;
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  r = fmaf(fmaf(-d, r, 1.f), r, r);
  return fabsf(z) <= SILU_FAST ? silu_fast(z) : (z < 0.f ? z * q : z) * r;
}
// byte of a 16-byte piece in a tile of 128-byte rows, SWIZZLE_128B
__device__ __forceinline__ uint32_t swz(int row, int piece) { return (uint32_t)(row * 128 + ((piece ^ (row & 7)) << 4)); }

// ---- prepare ---------------------------------------------------------------------------------------------------------------------
constexpr int SP_THREADS = 512;
// {row, tokens of this window, state line, earlier context} of all rows, the longest first, by one block.  The window is `most` tokens after the first `done`
__device__ __forceinline__ void order_rows(const SsdScanParams& p, int4* __restrict__ order, int* len, int done, int most) {
  for (int i = threadIdx.x; i < p.B; i += SP_THREADS) len[i] = p.q_len[i];
  __syncthreads();
  for (int i = threadIdx.x; i < p.B; i += SP_THREADS) {
    const int4 row = make_int4(i, min(min(p.q_len[i], p.T) - done, most), p.lines[i], done > 0 ? 1 : p.ctx_len[i]);
    const int own = len[i];
    int at = 0;
#pragma unroll 4
    for (int j = 0; j < p.B; ++j) at += len[j] > own || (len[j] == own && j < i);
    order[at] = row;
  }
}
__global__ void __launch_bounds__(SP_THREADS) ssd_prepare_kernel(SsdScanParams p, uint8_t* __restrict__ ws, float* __restrict__ most_g, int4* __restrict__ order,
                                                                 int chunks, int min_tokens, int done) {
  extern __shared__ __align__(16) float pm[];              // B, C [64][132]
  __shared__ unsigned most;                                // as bits (of positive numbers: in order)
  constexpr int LD = SN + 4;
  const int c = blockIdx.x, g = blockIdx.y, b = (int)blockIdx.z - 1, tid = threadIdx.x;
  pdl_launch_dependents();
  if (b < 0) {
    if (c == 0 && g == 0) order_rows(p, order, reinterpret_cast<int*>(pm), done, chunks * SQ);
    return;
  }
  const int n_tok = min(min(p.q_len[b], p.T) - done, chunks * SQ), n = min(n_tok - c * SQ, SQ);
  if (n_tok < min_tokens || n <= 0) return;
  const long long slot = ((long long)b * chunks + c) * p.G + g;
  uint8_t* img = ws + slot * S_WS;
  const int inner = p.nh * SP, Cd = inner + 2 * p.G * SN;
  const float* src = p.xBC + ((long long)b * p.T + c * SQ) * Cd + inner + g * SN;
  if (tid == 0) most = 0u;
  bool bad = false;
#pragma unroll                                             // (by a factor, the compiler settles for 40 registers: 11.1 us instead of 10.5)
  for (int i = tid; i < 2 * SQ * SN / 8; i += SP_THREADS) {       // 8 columns of a token
    const int which = i >> 10, t = (i >> 4) & 63, n0 = (i & 15) * 8;
    float v[8] = {};
    if (t < n) {
      const float4* q = reinterpret_cast<const float4*>(src + (long long)t * Cd + which * p.G * SN + n0);
      const float4 u = q[0], w = q[1];
      v[0] = u.x; v[1] = u.y; v[2] = u.z; v[3] = u.w; v[4] = w.x; v[5] = w.y; v[6] = w.z; v[7] = w.w;
    }
    float* row = pm + (which * SQ + t) * LD + n0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      bad |= !(fabsf(v[k]) < S_LARGE);
      row[k] = v[k];
    }
    store_parts(img + which * S_IMG + (n0 >> 6) * S_BLK + swz(t, (n0 & 63) >> 3), S_PART, v);
  }
  __syncthreads();
  // G[t][s], stored [s / 4][t][4]; 2 x 4 outputs of a thread (lanes along t: their rows of C miss each other's banks), sums over 16 columns added up in order
  const float *Bs = pm, *Cs = pm + SQ * LD;
  const int t0 = tid & 31, s0 = (tid >> 5) * 4;
  float tot[2][4] = {};
#pragma unroll 1
  for (int n0 = 0; n0 < SN; n0 += 16) {
    float acc[2][4] = {};
#pragma unroll
    for (int k = 0; k < 16; k += 4) {
      float4 bv[4], cv[2];
#pragma unroll
      for (int j = 0; j < 4; ++j) bv[j] = *reinterpret_cast<const float4*>(Bs + (s0 + j) * LD + n0 + k);
#pragma unroll
      for (int i = 0; i < 2; ++i) cv[i] = *reinterpret_cast<const float4*>(Cs + (t0 + 32 * i) * LD + n0 + k);
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          acc[i][j] = fmaf(cv[i].w, bv[j].w, fmaf(cv[i].z, bv[j].z, fmaf(cv[i].y, bv[j].y, fmaf(cv[i].x, bv[j].x, acc[i][j]))));
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) tot[i][j] += acc[i][j];
  }
  float big = 0.f;
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) big = fmaxf(big, fabsf(tot[i][j]));
  const unsigned m = __reduce_max_sync(0xffffffffu, bad ? 0x7f800000u : __float_as_uint(big));
  if ((tid & 31) == 0) atomicMax(&most, m);
  float4* G = reinterpret_cast<float4*>(img + 2 * S_IMG);
#pragma unroll
  for (int i = 0; i < 2; ++i) G[(s0 >> 2) * SQ + t0 + 32 * i] = make_float4(tot[i][0], tot[i][1], tot[i][2], tot[i][3]);
  __syncthreads();
  if (tid == 0) most_g[slot] = __uint_as_float(most);
}

// ---- scan ------------------------------------------------------------------------------------------------------------------------
struct ScanArgs {
  SsdScanParams p;
  const uint8_t* ws;
  const float* most_g;
  const int4* order;
  int chunks, min_tokens, pad;
  unsigned* wait_word;
};
// what a chunk's step sizes give, per head; two chunks in flight
struct ChunkSteps {
  float hi[2][SQ], lo[2][SQ];     // cs = hi + lo
  float dt[2][SQ];
  float e[2][SQ];                 // 2^cs
  float w[2][SQ];                 // dt 2^(cs_end - cs)
  float dA[2];                    // 2^cs_end
  float pad[2];
};
struct ScanShared {
  ChunkSteps st[2];
  float part[128];                // half of an output (step by step)
  uint64_t b_full, c_full, g_full, upd_done, inter_done, intra_done, xt_ready, s_ready, ds_read, mx_ready, y_read[2], dt_ready[2], part_full[4], part_free[4];
  uint32_t tmem;
  int stop;
  int odd_chunk[2];               // chunk + 1 when it runs step by step
};
static_assert(4 * SC2_FLOATS * sizeof(float) <= 4 * S_IMG + S_G && SC2_FLOATS % 4 == 0, "four groups of steps in the tiles");
constexpr int SC_SMEM = 4 * S_IMG + S_G + (int)sizeof(ScanShared) + 1024;

__device__ __forceinline__ uint64_t sc_desc(const void* smem, uint32_t lbo) {       // SWIZZLE_128B, 8-row groups 1024 bytes apart
  uint64_t d = 0;
  d |= (uint64_t)((mbar_s32(smem) & 0x3FFFF) >> 4);
  d |= (uint64_t)(lbo >> 4) << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
// D = f32, A = B = bf16, M = 128; bits 15 / 16: A / B are MN-major
__host__ __device__ constexpr uint32_t sc_idesc(int n, bool a_mn, bool b_mn) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (a_mn ? (1u << 15) : 0u) | (b_mn ? (1u << 16) : 0u) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}
// called by a whole warp, issued by the lane whose `on` is 1
__device__ __forceinline__ void sc_mma(uint32_t on, uint32_t d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc) {
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
               "l"(da), "l"(db), "r"(idesc), "r"(acc), "r"(on) : "memory");
}
__device__ __forceinline__ void sc_mma_ts(uint32_t on, uint32_t d, uint32_t a, uint64_t db, uint32_t idesc, uint32_t acc) {
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d),
               "r"(a), "l"(db), "r"(idesc), "r"(acc), "r"(on) : "memory");
}
__device__ __forceinline__ void sc_commit(uint32_t on, uint64_t* bar) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(mbar_s32(bar)),
               "r"(on) : "memory");
}
__device__ __forceinline__ void sc_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]),
                 "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
               : "r"(taddr));
}
__device__ __forceinline__ void sc_ld8(uint32_t taddr, uint32_t (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]) : "r"(taddr));
}
__device__ __forceinline__ void sc_st4(uint32_t taddr, const uint32_t* v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
}
// loads that stay where they are written, for values that are used much later; 0 where they are not `on` (as a conditional expression the compiler
// waits for every load to choose between it and the 0)
__device__ __forceinline__ float ld_ahead(const float* p, bool on) {
  float v = 0.f;
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\t@q ld.global.nc.f32 %0, [%1];\n\t}" : "+f"(v) : "l"(p), "r"((int)on));
  return v;
}
__device__ __forceinline__ float ld_ahead(const __nv_bfloat16* p, bool on) {
  unsigned short v = 0;
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\t@q ld.global.nc.u16 %0, [%1];\n\t}" : "+h"(v) : "l"(p), "r"((int)on));
  return __uint_as_float((uint32_t)v << 16);
}
__device__ __forceinline__ float4 ld_ahead4(const float4* p, bool on) {
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %5, 0;\n\t@q ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];\n\t}" : "+f"(v.x), "+f"(v.y), "+f"(v.z), "+f"(v.w)
               : "l"(p), "r"((int)on));
  return v;
}
// the parts of 8 neighbouring values of the K axis -> 4 columns in each of the three part regions, `stride` columns apart
__device__ __forceinline__ void put_parts(uint32_t taddr, uint32_t stride, const float (&v)[8]) {
  uint32_t w[3][4];
#pragma unroll
  for (int k = 0; k < 4; ++k) parts2(v[2 * k], v[2 * k + 1], w[0][k], w[1][k], w[2][k]);
#pragma unroll
  for (int q = 0; q < 3; ++q) sc_st4(taddr + q * stride, w[q]);
}
__device__ __forceinline__ void sc_bulk(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(mbar_s32(dst)), "l"(src), "r"(bytes),
               "r"(mbar_s32(bar)) : "memory");
}

template <typename T>
__global__ void __launch_bounds__(SC_THREADS, 1) ssd_chunk_kernel(const __grid_constant__ ScanArgs a) {
  extern __shared__ __align__(1024) uint8_t sc_raw[];
  uint8_t* smem = sc_raw + ((1024u - (mbar_s32(sc_raw) & 1023u)) & 1023u);
  uint8_t *sB = smem, *sC = sB + S_IMG, *sX = sC + S_IMG, *sM = sX + S_IMG, *sG = sM + S_IMG;
  ScanShared& sh = *reinterpret_cast<ScanShared*>(sG + S_G);
  const SsdScanParams& p = a.p;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int h0 = blockIdx.x * 2, g = h0 / (p.nh / p.G);
  volatile int* stop = &sh.stop;

  if (threadIdx.x == 0) {
    mbar_init(&sh.b_full, 1); mbar_init(&sh.c_full, 1); mbar_init(&sh.g_full, 1);
    mbar_init(&sh.upd_done, 1); mbar_init(&sh.inter_done, 1); mbar_init(&sh.intra_done, 1);
    mbar_init(&sh.xt_ready, 8); mbar_init(&sh.s_ready, 8); mbar_init(&sh.ds_read, 8); mbar_init(&sh.mx_ready, 4);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&sh.y_read[i], 8);
      mbar_init(&sh.dt_ready[i], 2);
      sh.odd_chunk[i] = 0;
    }
    for (int i = 0; i < 4; ++i) {
      mbar_init(&sh.part_full[i], 1);
      mbar_init(&sh.part_free[i], 1);
    }
    sh.stop = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == W_MMA) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(mbar_s32(&sh.tmem)), "n"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = sh.tmem;
  pdl_wait();
  const int4 row = a.order[blockIdx.y];
  const int b = row.x, n_tok = row.y, nc = (n_tok + SQ - 1) / SQ;
  const int inner = p.nh * SP, Cd = inner + 2 * p.G * SN;
  const float* xrow = p.xBC + (long long)b * p.T * Cd + h0 * SP;
  float* yrow = p.y + (long long)b * p.T * inner + h0 * SP;
  auto pad = [&](int tid, int threads) {                   // padding tokens: zeros
    for (int i = tid; i < (p.T - max(n_tok, 0)) * 32 * a.pad; i += threads)
      *reinterpret_cast<float4*>(yrow + (long long)(max(n_tok, 0) + (i >> 5)) * inner + (i & 31) * 4) = make_float4(0.f, 0.f, 0.f, 0.f);
  };
  if (n_tok >= a.min_tokens) {
    pad(threadIdx.x, SC_THREADS);
    auto wait = [&](uint64_t* bar, int phase) { return mbar_wait_warp(bar, (uint32_t)(phase & 1), stop, a.wait_word); };
    auto arrive = [&](uint64_t* bar) {
      __syncwarp();
      if (lane == 0) mbar_arrive(bar);
    };
    auto is_odd = [&](int c) { return *const_cast<volatile int*>(&sh.odd_chunk[c & 1]) == c + 1; };

    // registers: 768 threads x 80 at launch = 256 x 128 + 128 x 80 + 256 x 56 + 128 x 32
    if (warp < W_M) {
      // ================= the state: thread = (head, channel) row x half of the state axis =================
      asm volatile("setmaxnreg.inc.sync.aligned.u32 128;");
      const int hf = warp >> 2, r = (warp & 3) * 32 + lane, h = h0 + (r >> 6), hl = r >> 6;
      const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
      float* Sg = p.state + (((long long)row.z * p.nh + h) * SN + hf * 64) * SP + (r & 63);
      const bool ctx = row.w > 0;
      float S[64];
#pragma unroll
      for (int i = 0; i < 64; ++i) S[i] = ctx ? Sg[i * SP] : 0.f;
      auto put_state = [&](int c) {                          // the state's parts, for chunk c
        bool bad = false;
#pragma unroll
        for (int i0 = 0; i0 < 64; i0 += 8) {
          float v[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            v[i] = S[i0 + i];
            bad |= !(fabsf(v[i]) < S_LARGE);
          }
          put_parts(tmem + lanes + TM_S + hf * 32 + i0 / 2, 64, v);
        }
        if (bad) *const_cast<volatile int*>(&sh.odd_chunk[c & 1]) = c + 1;
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        arrive(&sh.s_ready);
      };
      float x[32];                                           // this thread's channel, tokens 32 hf .. 32 hf + 31 of the next chunk
      auto fetch_x = [&](int c) {
        const float* xs = xrow + (long long)(c * SQ + hf * 32) * Cd + r;
        const int n = n_tok - c * SQ - hf * 32;
        if (n >= 32) {                                       // (predicates cost the state's warps registers)
#pragma unroll
          for (int t = 0; t < 32; ++t) {
            x[t] = __ldg(xs);
            xs += Cd;
          }
        } else {
#pragma unroll
          for (int t = 0; t < 32; ++t) {
            x[t] = ld_ahead(xs, t < n);
            xs += Cd;
          }
        }
      };
      auto put_x = [&](int c) {                              // the parts of x~ of chunk c
        if (!wait(&sh.dt_ready[c & 1], c >> 1)) return false;
        const ChunkSteps& st = sh.st[c & 1];
        bool bad = false;
#pragma unroll
        for (int t0 = 0; t0 < 32; t0 += 8) {
          float v[8];
#pragma unroll
          for (int t = 0; t < 8; ++t) {
            v[t] = x[t0 + t] * st.w[hl][hf * 32 + t0 + t];
            bad |= !(fabsf(x[t0 + t]) < S_LARGE && fabsf(v[t]) < S_LARGE);
          }
          put_parts(tmem + lanes + TM_X + hf * 16 + t0 / 2, 32, v);
        }
        if (bad) *const_cast<volatile int*>(&sh.odd_chunk[c & 1]) = c + 1;
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        arrive(&sh.xt_ready);
        return true;
      };
      bool go = true;
      if (nc > 0) {
        fetch_x(0);
        put_state(0);
        go = put_x(0);
      }
      int c = 0, steps = 0;                                  // steps: tokens that ran step by step so far
      for (; c < nc && go; ++c) {
        const ChunkSteps& st = sh.st[c & 1];
        const int n = min(SQ, n_tok - c * SQ);
        const float dA = st.dA[hl];
        if (c + 1 < nc) fetch_x(c + 1);                      // in flight while the state is updated
        if (!wait(&sh.upd_done, c)) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (!is_odd(c)) {
#pragma unroll
          for (int i0 = 0; i0 < 64; i0 += 8) {
            uint32_t d[8];
            sc_ld8(tmem + lanes + TM_W + hf * 64 + i0, d);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int i = 0; i < 8; ++i) S[i0 + i] = fmaf(dA, S[i0 + i], __uint_as_float(d[i]));
          }
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        } else {
          // step by step, as ssd_scan_kernel (seqmix.cu)
          const float negA = -expf(p.A_log[h]), Dh = p.D_skip[h];
          const T* zp = (const T*)p.z + (long long)b * p.z_sb + h * SP + (r & 63);
          const int q = warp & 3;
#pragma unroll 1
          for (int t = 0; t < n; ++t, ++steps) {
            const long long at = (long long)c * SQ + t;
            const float* row = xrow + at * Cd;
            const float *Bt = row - h0 * SP + inner + g * SN + hf * 64, *Ct = Bt + p.G * SN;
            const float dt = st.dt[hl][t], dAt = expf(negA * dt), xt = row[r], dx = dt * xt;
            float y = 0.f;
#pragma unroll
            for (int i = 0; i < 64; ++i) {
              S[i] = fmaf(dAt, S[i], dx * __ldg(Bt + i));
              y = fmaf(S[i], __ldg(Ct + i), y);
            }
            if (hf == 1) {
              if (steps > 0 && !wait(&sh.part_free[q], steps - 1)) break;
              sh.part[r] = y;
              arrive(&sh.part_full[q]);
            } else {
              if (!wait(&sh.part_full[q], steps)) break;
              const float z = ldf(zp + at * p.z_st);
              yrow[at * inner + r] = ((y + sh.part[r]) + Dh * xt) * (z * (1.f / (1.f + expf(-z))));
              arrive(&sh.part_free[q]);
            }
          }
        }
        arrive(&sh.ds_read);
        if (c + 1 < nc) {
          if (!put_x(c + 1) || !wait(&sh.inter_done, c)) break;
          put_state(c + 1);
        }
      }
      if (nc > 0 && c == nc) {
#pragma unroll
        for (int i = 0; i < 64; ++i) Sg[i * SP] = S[i];
      }
    } else if (warp < W_OUT) {
      // ================= M and the parts of x =================
      asm volatile("setmaxnreg.inc.sync.aligned.u32 80;");
      // M is a triangle: rows 0 .. 31 of a head have 4 pieces of 8 columns, rows 32 .. 63 have 8; the two warps of a head take 6 each (lane = row)
      const int m = threadIdx.x - 32 * W_M, hl = m >> 6, second = (m >> 5) & 1;
      const float Dh = p.D_skip[h0 + hl];
      if (second == 0) {                                           // the other 4 pieces of rows 0 .. 31 stay 0
#pragma unroll 1
        for (int j = 4; j < 8; ++j)
#pragma unroll
          for (int q = 0; q < 3; ++q) *reinterpret_cast<uint4*>(sM + q * S_PART + swz(hl * 64 + lane, j)) = make_uint4(0u, 0u, 0u, 0u);
      }
      for (int c = 0; c < nc; ++c) {
        const int n = min(SQ, n_tok - c * SQ);
        const int ch = m & 15, row = m >> 4;                       // 8 channels of tokens row, row + 8, ..
        const float4* xq = reinterpret_cast<const float4*>(xrow + (long long)(c * SQ + row) * Cd + ch * 8);
        float4 u[8][2];                                            // in flight during the waits
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          u[i][0] = ld_ahead4(xq, row + 8 * i < n);
          u[i][1] = ld_ahead4(xq + 1, row + 8 * i < n);
          xq += 2LL * Cd;
        }
        if (c > 0 && !wait(&sh.intra_done, c - 1)) break;          // the tiles of the chunk before are read
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float v[8] = {u[i][0].x, u[i][0].y, u[i][0].z, u[i][0].w, u[i][1].x, u[i][1].y, u[i][1].z, u[i][1].w};
          store_parts(sX + (ch >> 3) * S_BLK + swz(row + 8 * i, ch & 7), S_PART, v);
        }
        if (!wait(&sh.g_full, c) || !wait(&sh.dt_ready[c & 1], c >> 1)) break;
        const ChunkSteps& st = sh.st[c & 1];
        const float4* G = reinterpret_cast<const float4*>(sG);
        // loops stay rolled here and in the other roles where they can: with everything unrolled the warps waited for instructions, not for data
#pragma unroll 2
        for (int i = 0; i < 6; ++i) {                              // 8 columns of row (head, t)
          const int j = second ? i + 2 : i & 3, t = lane + (second || i >= 4 ? 32 : 0);
          const float hi = st.hi[hl][t], lo = st.lo[hl][t];
          const float4 g0 = G[2 * j * SQ + t], g1 = G[(2 * j + 1) * SQ + t];
          float v[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
          float sh_[8], sl[8], sd[8];
          auto eight = [&](float* to, const float* from) {
            const float4 p0 = *reinterpret_cast<const float4*>(from), p1 = *reinterpret_cast<const float4*>(from + 4);
            to[0] = p0.x; to[1] = p0.y; to[2] = p0.z; to[3] = p0.w; to[4] = p1.x; to[5] = p1.y; to[6] = p1.z; to[7] = p1.w;
          };
          eight(sh_, st.hi[hl] + 8 * j);
          eight(sl, st.lo[hl] + 8 * j);
          eight(sd, st.dt[hl] + 8 * j);
          const int own = t - 8 * j;                               // the diagonal
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            v[k] = k <= own ? v[k] * (sd[k] * ex2((hi - sh_[k]) + (lo - sl[k]))) : 0.f;
            if (k == own) v[k] += Dh;                              // the skip rides on it
          }
          store_parts(sM + swz(hl * 64 + t, j), S_PART, v);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        arrive(&sh.mx_ready);
      }
    } else if (warp < W_MMA) {
      // ================= outputs: thread = (head, channel) x half of the tokens =================
      asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
      const int hf = (warp - W_OUT) >> 2, r = (warp & 3) * 32 + lane, hl = r >> 6, h = h0 + hl;
      const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
      const T* zp = (const T*)p.z + (long long)b * p.z_sb + h * SP + (r & 63);
      for (int c = 0; c < nc; ++c) {
        const long long at = (long long)c * SQ + hf * 32;
        const int n = (int)min(32LL, n_tok - at);
        float s[32];                                               // silu(z), while the products run
        const T* zt = zp + at * p.z_st;
        float* yt = yrow + at * inner + r;
#pragma unroll
        for (int t = 0; t < 32; ++t) {
          s[t] = ld_ahead(zt, t < n);
          zt += p.z_st;
        }
        float big = 0.f;
#pragma unroll
        for (int t = 0; t < 32; ++t) big = fmaxf(big, fabsf(s[t]));
        if (__any_sync(0xffffffffu, big > SILU_FAST)) {
#pragma unroll
          for (int t = 0; t < 32; ++t) s[t] = silu_any(s[t]);
        } else {
#pragma unroll
          for (int t = 0; t < 32; ++t) s[t] = silu_fast(s[t]);
        }
        if (!wait(&sh.intra_done, c)) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const bool mine = !is_odd(c);
        if (mine) {
          const ChunkSteps& st = sh.st[c & 1];
#pragma unroll
          for (int t0 = 0; t0 < 32; t0 += 8) {
            uint32_t u[8], w[8];
            sc_ld8(tmem + lanes + TM_I + hf * 32 + t0, u);
            sc_ld8(tmem + lanes + TM_W + hl * 64 + hf * 32 + t0, w);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int t = 0; t < 8; ++t) s[t0 + t] *= fmaf(st.e[hl][hf * 32 + t0 + t], __uint_as_float(u[t]), __uint_as_float(w[t]));
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        arrive(&sh.y_read[c & 1]);                                 // the next chunk's products may start
        if (mine) {
#pragma unroll
          for (int t = 0; t < 32; ++t) {
            if (t < n) *yt = s[t];
            yt += inner;
          }
        }
      }
    } else {
      asm volatile("setmaxnreg.dec.sync.aligned.u32 32;");
      if (warp == W_MMA) {
        // ================= MMAs =================
        uint32_t on;
        asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(on));
        constexpr uint32_t id_upd = sc_idesc(128, false, true), id_inter = sc_idesc(64, false, false), id_intra = sc_idesc(128, true, false);
        const uint64_t dB = sc_desc(sB, S_BLK), dC = sc_desc(sC, 16), dX = sc_desc(sX, S_BLK), dM = sc_desc(sM, 16);
        for (int c = 0; c < nc; ++c) {
          if (!wait(&sh.b_full, c) || !wait(&sh.xt_ready, c) || !wait(&sh.s_ready, c) || (c > 0 && !wait(&sh.y_read[(c - 1) & 1], (c - 1) >> 1))) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const bool run = !is_odd(c);
          // part products, the smallest first: 2 0, 1 1, 0 2, 1 0, 0 1, 0 0
          if (run) {
#pragma unroll 1
            for (int q = 0; q < 6; ++q) {
              const int i = (0x001012 >> (4 * q)) & 3, j = (0x010210 >> (4 * q)) & 3;
#pragma unroll
              for (int k = 0; k < 4; ++k)       // 16 tokens: 8 columns of A, 16 rows of B
                sc_mma_ts(on, tmem + TM_W, tmem + TM_X + 32 * i + 8 * k, dB + (uint64_t)(j * (S_PART >> 4) + k * 128), id_upd, (q | k) != 0 ? 1u : 0u);
            }
          }
          sc_commit(on, &sh.upd_done);
          if (!wait(&sh.c_full, c)) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          if (run) {
#pragma unroll 1
            for (int q = 0; q < 6; ++q) {
              const int i = (0x001012 >> (4 * q)) & 3, j = (0x010210 >> (4 * q)) & 3;
#pragma unroll
              for (int k = 0; k < 8; ++k)       // 16 state columns: 8 columns of A, 32 bytes of the rows of C
                sc_mma_ts(on, tmem + TM_I, tmem + TM_S + 64 * i + 8 * k, dC + (uint64_t)(j * (S_PART >> 4) + (k >> 2) * (S_BLK >> 4) + (k & 3) * 2), id_inter,
                          (q | k) != 0 ? 1u : 0u);
            }
          }
          sc_commit(on, &sh.inter_done);
          if (!wait(&sh.ds_read, c) || !wait(&sh.mx_ready, c)) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          if (run) {
#pragma unroll 1
            for (int q = 0; q < 6; ++q) {
              const int i = (0x001012 >> (4 * q)) & 3, j = (0x010210 >> (4 * q)) & 3;
#pragma unroll
              for (int k = 0; k < 4; ++k)       // 16 tokens s: 16 rows of A, 32 bytes of the rows of M
                sc_mma(on, tmem + TM_W, dX + (uint64_t)(i * (S_PART >> 4) + k * 128), dM + (uint64_t)(j * (S_PART >> 4) + k * 2), id_intra, (q | k) != 0 ? 1u : 0u);
            }
          }
          sc_commit(on, &sh.intra_done);
        }
      } else if (warp == W_COPY) {
        // ================= copies of the B, C and G images =================
        const uint8_t* img = a.ws + ((long long)b * a.chunks * p.G + g) * S_WS;
        for (int c = 0; c < nc; ++c) {
          const uint8_t* src = img + (long long)c * p.G * S_WS;
          if (c > 0 && !wait(&sh.upd_done, c - 1)) break;
          if (lane == 0) {
            mbar_expect(&sh.b_full, S_IMG);
            sc_bulk(sB, src, S_IMG, &sh.b_full);
          }
          if (c > 0 && !wait(&sh.inter_done, c - 1)) break;
          if (lane == 0) {
            mbar_expect(&sh.c_full, S_IMG);
            sc_bulk(sC, src + S_IMG, S_IMG, &sh.c_full);
          }
          if (c > 0 && !wait(&sh.mx_ready, c - 1)) break;
          if (lane == 0) {
            mbar_expect(&sh.g_full, S_G);
            sc_bulk(sG, src + 2 * S_IMG, S_G, &sh.g_full);
          }
        }
      } else {
        // ================= step sizes and exponents of one head: lane = two neighbouring tokens =================
        const int hl = warp - W_STEP, h = h0 + hl;
        const T* dtp = (const T*)p.dt_raw + (long long)b * p.dt_sb + h;
        const double negA = -(double)expf(p.A_log[h]) * 1.4426950408889634;      // to log2
        const float bias = p.dt_bias[h], Dh = fabsf(p.D_skip[h]);
        const float* most_g = a.most_g + (long long)b * a.chunks * p.G + g;
        for (int c = 0; c < nc; ++c) {
          const int n = min(SQ, n_tok - c * SQ);
          const float g_most = most_g[(long long)c * p.G];
          float dt[2];
          double cs[2];
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const int t = 2 * lane + k;
            dt[k] = 0.f;
            if (t < n) {
              const float v = ldf(dtp + (long long)(c * SQ + t) * p.dt_st) + bias;
              dt[k] = v > 20.f ? v : log1pf(expf(v));
            }
            cs[k] = negA * (double)dt[k];
          }
          cs[1] += cs[0];
          double incl = cs[1];
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const double v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
          }
          const double before = __shfl_up_sync(0xffffffffu, incl, 1), end = __shfl_sync(0xffffffffu, incl, 31);
          if (lane > 0) {
            cs[0] += before;
            cs[1] += before;
          }
          if (c > 1 && !wait(&sh.y_read[c & 1], (c - 2) >> 1)) break;             // everybody is done with the chunk before the last
          ChunkSteps& st = sh.st[c & 1];
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const int t = 2 * lane + k;
            const float hi = (float)cs[k], lo = (float)(cs[k] - (double)hi);
            st.hi[hl][t] = hi;
            st.lo[hl][t] = lo;
            st.dt[hl][t] = dt[k];
            st.e[hl][t] = exp2f(hi) * fmaf(lo, 0.69314718f, 1.f);
            st.w[hl][t] = dt[k] * exp2f((float)(end - cs[k]));
          }
          // |M| <= |G| dt + |D|
          if (!(fmaf(g_most, dt[0], Dh) < S_LARGE && fmaf(g_most, dt[1], Dh) < S_LARGE)) *const_cast<volatile int*>(&sh.odd_chunk[c & 1]) = c + 1;
          if (lane == 31) st.dA[hl] = exp2f((float)end) * fmaf((float)(end - (double)(float)end), 0.69314718f, 1.f);
          arrive(&sh.dt_ready[c & 1]);
        }
      }
    }
    if (*stop) __nanosleep(1000000);        // gave up: let copies in flight land before the shared memory goes away
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == W_MMA) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(512));
    }
    return;
  }
  // ================= a short row, step by step: four groups of 128 threads, one per head and half of its channels =================
  if (warp == W_MMA) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(512));
  // the state of the short row that starts when this one ends comes to the L2 meanwhile
  if (threadIdx.x == SC_THREADS - 1) {
    const int next = blockIdx.y * gridDim.x + blockIdx.x + kNumSMs;
    if (next < (int)(gridDim.x * gridDim.y)) {
      const int4 to = a.order[next / gridDim.x];
      if (to.y > 0 && to.w > 0 && to.y < a.min_tokens)
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p.state + ((long long)to.z * p.nh + next % gridDim.x * 2) * SN * SP), "r"(2 * SN * SP * 4) : "memory");
    }
  }
  __syncwarp();
  // registers: 768 threads x 80 at launch > 512 x 104 + 256 x 24
  if (warp < 16) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
    const int at = warp >> 2;
    if (n_tok > 0)
      ssd_steps<T>(p, reinterpret_cast<float*>(smem) + at * SC2_FLOATS, b, n_tok, row.z, row.w, h0 + (at >> 1), (at & 1) * SC2_PT, threadIdx.x & 127,
                   [&] { asm volatile("bar.sync %0, 128;" ::"r"(1 + at) : "memory"); });
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 24;");
    pad(threadIdx.x - 512, SC_THREADS - 512);
  }
}

}  // namespace

bool ssd_chunk_supported(const SsdScanParams& p) {
  return p.N == SN && p.P == SP && p.T >= SSD_CHUNK_MIN_T && p.G > 0 && (p.nh / p.G) % 2 == 0 && p.B <= 65535 && p.G <= 65535 &&
         (reinterpret_cast<uintptr_t>(p.xBC) | reinterpret_cast<uintptr_t>(p.state)) % 16 == 0;
}
// The images take 114.7 KB per (row, chunk of 64 tokens, group): 1.8 KB a token and group, padding included.  Calls that would take more than this run in windows of
// tokens, the state carried in its place, and where one chunk of all rows is more, in groups of rows (at least one chunk of one row).  A window ends with an
// emptying chip and costs the state's way through memory: with 128 MB, 16 rows of 1024 tokens (128 heads, 8 groups) ran in two windows, 971 us instead of 843.
constexpr long long S_WS_MOST = 512LL << 20;
static_assert(S_WS_MOST / S_WS <= 2 * SQ * (SN + 4), "a group's rows are ordered in the prepare kernel's shared memory");
static void ssd_window(const SsdScanParams& p, int& rows, int& chunks) {
  const long long per = (long long)p.G * S_WS;
  rows = (int)std::max(1LL, std::min((long long)p.B, S_WS_MOST / per));
  chunks = (int)std::max(1LL, std::min((long long)(p.T + SQ - 1) / SQ, S_WS_MOST / (per * rows)));
}
// images, order of the rows, largest |G| per (row, chunk, group)
long long ssd_chunk_workspace(const SsdScanParams& p) {
  int rows, chunks;
  ssd_window(p, rows, chunks);
  return (long long)rows * chunks * p.G * (S_WS + (long long)sizeof(float)) + rows * (long long)sizeof(int4);
}
bool ssd_chunk_pads(const SsdScanParams& p) {
  int rows, chunks;
  ssd_window(p, rows, chunks);
  return (long long)chunks * SQ >= p.T;
}
void ssd_chunk_launch(const SsdScanParams& all, void* workspace, bool lp, cudaStream_t st) {
  int rows, chunks;
  ssd_window(all, rows, chunks);
  ScanArgs a{};
  a.chunks = chunks;
  a.ws = static_cast<const uint8_t*>(workspace);
  a.order = reinterpret_cast<const int4*>(a.ws + (long long)rows * chunks * all.G * S_WS);
  a.most_g = reinterpret_cast<const float*>(a.order + rows);
  // tokens from which on a row takes chunks.  us, steps / chunks: one row of 16, 24 and 32 tokens 20.5 / 26.6, 24.6 / 26.6, 28.7 / 26.6; sixteen rows (several CTAs
  // per SM, one after the other) of 8 and 16 47 / 57, 61 / 59
  a.min_tokens = (long long)all.B * all.nh > 4 * kNumSMs ? 16 : 28;
  a.pad = ssd_chunk_pads(all) ? 1 : 0;
  check_waits();
  a.wait_word = wait_word(WAIT_SSD);
  count_launch(COUNT_SSD);
  constexpr int PREP_SMEM = 2 * SQ * (SN + 4) * (int)sizeof(float);
  const int esz = lp ? 2 : 4;
  const long long inner = (long long)all.nh * SP, Cd = inner + 2LL * all.G * SN;
  auto go = [&](auto kernel) {
    if (cudaFuncSetAttribute(ssd_prepare_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PREP_SMEM) != cudaSuccess ||
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SC_SMEM) != cudaSuccess)
      throw std::runtime_error("ssd scan: shared memory size refused");
    for (int b0 = 0; b0 < all.B; b0 += rows)
      for (int done = 0; done < all.T; done += chunks * SQ) {
        SsdScanParams& p = a.p;                            // the rows and tokens of this window; a row's stride stays T tokens
        p = all;
        p.B = std::min(rows, all.B - b0);
        const long long at = (long long)b0 * all.T + done;
        p.xBC += at * Cd;
        p.y += at * inner;
        p.dt_raw = static_cast<const char*>(all.dt_raw) + (b0 * all.dt_sb + done * all.dt_st) * esz;
        p.z = static_cast<const char*>(all.z) + (b0 * all.z_sb + done * all.z_st) * esz;
        p.lines += b0;
        p.ctx_len += b0;
        p.q_len += b0;
        ssd_prepare_kernel<<<dim3(chunks, p.G, p.B + 1), SP_THREADS, PREP_SMEM, st>>>(p, static_cast<uint8_t*>(workspace), const_cast<float*>(a.most_g),
                                                                                       const_cast<int4*>(a.order), chunks, a.min_tokens, done);
        launch_pdl(kernel, dim3(p.nh / 2, p.B), dim3(SC_THREADS), SC_SMEM, st, a);
      }
  };
  if (lp) go(ssd_chunk_kernel<__nv_bfloat16>); else go(ssd_chunk_kernel<float>);
}

}  // namespace nxdi
