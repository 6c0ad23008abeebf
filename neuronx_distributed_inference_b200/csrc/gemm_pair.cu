// Prompt-sized GEMM on CTA pairs:  C[M,N] = epilogue( A[M,K] · B[N,K]^T ), bf16 in, fp32 accumulators (tcgen05.mma.cta_group::2).
//
// What bounded the one-CTA kernel (gemm_tcgen05.cu, 128 x 256 tiles): 48 KB of operands per 64-deep k-block and SM from L2 (12 TB/s over the chip) and
// 96 B/clk of operand reads plus as much of TMA writes on a 128 B/clk shared memory.  Two SMs that work on ONE 256 x 256 tile need 32 KB each: a CTA
// holds 128 rows of A and half of B's rows, and the pair's MMA reads both halves.
//   * cluster of 2; the even CTA (leader) issues every MMA; TMEM of both holds 128 rows x 256 columns, double buffered (512 columns)
//   * warps 0 / 3: TMA producers of B / A, 6-stage ring of 32 KB; the copies of both CTAs complete on the leader's full barrier; the leader's commits
//     free the stages and hand over the accumulators in both CTAs (multicast arrive)
//   * warps 4..11: epilogue of the CTA's own 128 rows (two warps per 32 rows take turns at 64-column pieces: with four warps the gate products of
//     2048-deep tiles took longer than their MMAs); bias / residual / gate products; rows leave (and residual rows come) through shared memory as
//     whole 128-byte pieces
//   * grouped (mixture of experts): A holds tokens permuted by expert, one row per token and slot; tile_expert / tile_row give a row tile's expert, how many
//     rows it stores (a half without any is neither loaded nor stored) and its first row; an expert's last tile reads on into the rows behind its own.  Tiles are walked in bands of four row tiles, n-tile by n-tile
//     inside a band: the permuted rows and an expert's weights are read from HBM once (128 experts of 2048 x 768, 4096 tokens, 8 each, both GEMMs with
//     permutation: 456 us; bands of 32 row tiles 480, no bands 589; 8 experts of 4096 x 14336, 1024 tokens: 858, 951, 944).
// Measured (isolated, us, here / 128 x 256 tiles of one CTA): 4096 tokens 28672 x 4096 gate|up 624 / 725 (1.54 PFLOP/s, 94 % of the measured cuBLAS burst),
// 4096 x 14336 336 / 371, 16384 x 2048 gate|up 188 / 356 (290 with four epilogue warps).  256 x 128 tiles are slower wherever they were tried (960 us
// for the first): their operand traffic per flop is that of the one-CTA tiles again.
#include <algorithm>
#include <stdexcept>
#include <string>

#include "api.h"
#include "common.cuh"
#include "mbar_wait.cuh"

namespace nxdi {

constexpr int GP_BN = 256, GP_BK = 64, GP_STAGES = 6;
constexpr int GP_EPI_WARPS = 8, GP_THREADS = 128 + 32 * GP_EPI_WARPS;
constexpr int GP_A_BYTES = 128 * GP_BK * 2, GP_STAGE = GP_A_BYTES + GP_BN / 2 * GP_BK * 2;
constexpr int GP_SMEM = GP_STAGES * GP_STAGE + 256 + GP_EPI_WARPS * 4096 + 1024;

struct PairParams {
  CUtensorMap tma_a;              // A [M, K], box {64, 128}
  CUtensorMap tma_b;              // B [experts * N, K], box {64, BN / 2}
  const __nv_bfloat16* bias;      // [experts][N] or null
  const __nv_bfloat16* residual;  // [M, n_out] or null (act == 0)
  __nv_bfloat16* c;               // [M, n_out]
  int M, N, K, n_out, act;        // act: 0 none, 1 silu*up, 2 gelu_tanh*up, 3 gelu*up, 4 clamped gate product (n_out = N / 2)
  float limit, alpha;
  const float* scale;             // SCALED: of the sums, [N], or [1] (scale_one)
  int scale_one;
  int m_tiles, n_tiles, band;
  int w_fresh;                    // B was written by a kernel just before this one
  unsigned* wait_word;            // mbar_wait.cuh
  const int* tile_expert;         // grouped: [m_tiles] expert | rows << 10 of a row tile, < 0: not in use; null: one weight
  const int* tile_row;            // grouped: [m_tiles] first row of a row tile
};

// shared::cluster address of a local shared-memory object in the pair's leader
__device__ __forceinline__ uint32_t gp_leader(const void* p) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(mbar_s32(p)));
  return r;
}
__device__ __forceinline__ void gp_tma(void* dst, const CUtensorMap* tm, int c0, int c1, uint32_t leader_bar) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(mbar_s32(dst)),
               "l"(tm), "r"(c0), "r"(c1), "r"(leader_bar) : "memory");
}
__device__ __forceinline__ uint64_t gp_desc(const void* smem) {     // K-major, 128-byte rows, SWIZZLE_128B
  uint64_t d = 0;
  d |= (uint64_t)((mbar_s32(smem) & 0x3FFFF) >> 4);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
// Called by a whole warp, issued by the lane whose `on` is 1: in code that all lanes run the descriptors stay in uniform registers
__device__ __forceinline__ void gp_umma(uint32_t on, uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc) {
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d), "l"(da),
               "l"(db), "r"(idesc), "r"(acc), "r"(on) : "memory");
}
__device__ __forceinline__ void gp_commit_both(uint32_t on, uint64_t* bar) {      // arrives on the barrier at this offset in both CTAs
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\t@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}" ::"r"(mbar_s32(bar)),
               "h"((unsigned short)3), "r"(on) : "memory");
}
__device__ __forceinline__ uint32_t gp_elect() {
  uint32_t r;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r));
  return r;
}
__device__ __forceinline__ void gp_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void gp_ld32(uint32_t taddr, uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
        "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]),
        "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]),
        "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(taddr));
}
// tile number -> coordinates: band by band, inside a band n-tile by n-tile, m fastest
__device__ __forceinline__ void gp_tile(const PairParams& p, int t, int& mt, int& nt) {
  const int per = p.band * p.n_tiles, b = t / per, r = t - b * per, rows = min(p.band, p.m_tiles - b * p.band);
  mt = b * p.band + r % rows;
  nt = r / rows;
}

// SCALED: of a weight that was expanded from bytes without its scale
template <bool SCALED>
__global__ void __launch_bounds__(GP_THREADS, 1) gemm_pair_kernel(const __grid_constant__ PairParams p) {
  constexpr int BN = GP_BN, ST = GP_STAGES, STAGE = GP_STAGE;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (mbar_s32(smem_raw) & 1023u)) & 1023u);
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + ST * STAGE);    // the leader's are used
  uint64_t* empty_bar = full_bar + ST;
  uint64_t* tmem_full = empty_bar + ST;     // [2]
  uint64_t* tmem_empty = tmem_full + 2;     // [2] the leader's: the epilogue warps of the pair
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_empty + 2);
  volatile int* stop = reinterpret_cast<volatile int*>(tmem_slot + 1);
  uint8_t* staging = reinterpret_cast<uint8_t*>(smem + ST * STAGE + 256);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t rank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const bool glu = p.act != 0;
  const int nkb = p.K / GP_BK, total = p.m_tiles * p.n_tiles;
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const int tile_out = glu ? BN / 2 : BN;

  if (warp == 1 && lane == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&p.tma_a) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&p.tma_b) : "memory");
    for (int s = 0; s < ST; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tmem_full[b], 1);
      mbar_init(&tmem_empty[b], 2 * GP_EPI_WARPS);
    }
    *stop = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(mbar_s32(tmem_slot)), "n"(2 * BN));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  gp_cluster_sync();            // the peer's barriers exist
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  pdl_launch_dependents();
  // a weight that is a parameter does not depend on earlier kernels; everything else does
  bool early = warp == 0 && p.tile_expert == nullptr && !p.w_fresh;
  if (!early) pdl_wait();

  if (warp == 0 || warp == 3) {
    // ================= TMA producers: B (warp 0), A (warp 3) of this CTA =================
    if (lane == 0) {
      int s = 0;
      uint32_t phase = 0;
      bool go = true;
      for (int t = pair; t < total && go; t += pairs) {
        int mt, nt;
        gp_tile(p, t, mt, nt);
        int e = 0, m0 = mt * 256;
        bool second = true;              // the odd CTA's half has rows
        if (p.tile_expert != nullptr) {
          e = __ldg(p.tile_expert + mt);
          if (e < 0) continue;
          second = (e >> 10) > 128;
          e &= 1023;
          m0 = __ldg(p.tile_row + mt);
        }
        const int row_a = m0 + (int)rank * 128;
        const int row_b = e * p.N + (glu ? nt * (BN / 2) + (rank ? p.n_out : 0) : nt * BN + (int)rank * (BN / 2));
        for (int kb = 0; kb < nkb; ++kb) {
          if (early && phase != 0) {       // the ring is full: from here on a wait depends on the warps that wait for earlier kernels
            pdl_wait();
            early = false;
          }
          go = mbar_wait<true>(&empty_bar[s], phase ^ 1u, stop, p.wait_word);
          if (!go) break;
          uint8_t* st = smem + s * STAGE;
          const uint32_t bar = gp_leader(&full_bar[s]);
          if (warp == 0) {
            gp_tma(st + GP_A_BYTES, &p.tma_b, kb * GP_BK, row_b, bar);
          } else {
            if (rank == 0) mbar_expect(&full_bar[s], 2 * STAGE - (second ? 0 : GP_A_BYTES));       // everything that both CTAs copy for this stage
            if (rank == 0 || second) gp_tma(st, &p.tma_a, kb * GP_BK, row_a, bar);
          }
          if (++s == ST) {
            s = 0;
            phase ^= 1u;
          }
        }
      }
    }
  } else if (warp == 1) {
    // ================= MMA issuer: a warp of the leader =================
    if (rank == 0) {
      // D = f32, A = B = bf16, both K-major, M = 256, N = BN
      constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
      const uint32_t on = gp_elect();
      const uint64_t da0 = gp_desc(smem), db0 = gp_desc(smem + GP_A_BYTES);
      int tc = 0, s = 0;
      uint32_t phase = 0;
      bool go = true;
      for (int t = pair; t < total && go; t += pairs) {
        if (p.tile_expert != nullptr) {
          int mt, nt;
          gp_tile(p, t, mt, nt);
          if (__ldg(p.tile_expert + mt) < 0) continue;
        }
        const int buf = tc & 1;
        go = mbar_wait_warp<true>(&tmem_empty[buf], (uint32_t)((tc >> 1) & 1) ^ 1u, stop, p.wait_word);
        if (!go) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        for (int kb = 0; kb < nkb; ++kb) {
          go = mbar_wait_warp<true>(&full_bar[s], phase, stop, p.wait_word);
          if (!go) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint64_t da = da0 + (uint64_t)(s * (STAGE >> 4)), db = db0 + (uint64_t)(s * (STAGE >> 4));
#pragma unroll
          for (int k = 0; k < GP_BK / 16; ++k)       // 16 k = 32 bytes inside the swizzle atom
            gp_umma(on, tmem + (uint32_t)(buf * BN), da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), idesc, (kb | k) != 0 ? 1u : 0u);
          gp_commit_both(on, &empty_bar[s]);
          if (++s == ST) {
            s = 0;
            phase ^= 1u;
          }
        }
        if (go) gp_commit_both(on, &tmem_full[buf]);
        ++tc;
      }
    }
  } else if (warp >= 4) {
    // ================= epilogue of this CTA's 128 rows =================
    const int q = warp & 3;
    uint8_t* stg = staging + (warp - 4) * 4096;             // 32 rows x 64 columns, 16-byte chunks XOR-swizzled
    auto stg_at = [&](int r, int ch) { return reinterpret_cast<uint4*>(stg + r * 128 + ((ch ^ (r & 7)) << 4)); };
    // rows row0 .. row0 + 31, columns col0 .. col0 + 63, lanes along the rows: residual in, results out
    auto move_rows = [&](int row0, int row_end, int col0, bool in) {
      __syncwarp();
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = i * 4 + (lane >> 3), ch = lane & 7, row = row0 + r, col = col0 + ch * 8;
        if (row < row_end && col < p.n_out) {          // n_out % 8 == 0: a chunk is inside or outside as a whole
          if (in) *stg_at(r, ch) = ldg_act(p.residual + (size_t)row * p.n_out + col);
          else *reinterpret_cast<uint4*>(p.c + (size_t)row * p.n_out + col) = *stg_at(r, ch);
        }
      }
      __syncwarp();
    };
    int tc = 0;
    for (int t = pair; t < total; t += pairs) {
      int mt, nt;
      gp_tile(p, t, mt, nt);
      int eo = 0, m0 = mt * 256, row_end = p.M;
      if (p.tile_expert != nullptr) {
        const int e = __ldg(p.tile_expert + mt);
        if (e < 0) continue;
        eo = (e & 1023) * p.N;
        m0 = __ldg(p.tile_row + mt);
        row_end = m0 + (e >> 10);
      }
      const int buf = tc & 1, row0 = m0 + (int)rank * 128 + q * 32, col_t = nt * tile_out;
      if (!mbar_wait_warp<true>(&tmem_full[buf], (uint32_t)((tc >> 1) & 1), stop, p.wait_word)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t acc = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * BN);
#pragma unroll 1
      for (int c0 = warp >= 8 ? 64 : 0; c0 < tile_out && row0 < row_end; c0 += 128) {
        if (p.residual != nullptr) move_rows(row0, row_end, col_t + c0, true);
#pragma unroll 1
        for (int c = c0; c < c0 + 64; c += 32) {
          float sg[32], su[32];      // SCALED: loaded in front of the sums
          if (SCALED) {
            load_scales(p.scale, p.scale_one != 0, col_t + c, p.n_out, sg);
            if (glu) load_scales(p.scale + (p.scale_one ? 0 : p.n_out), p.scale_one != 0, col_t + c, p.n_out, su);
          }
          uint32_t vg[32], vu[32];
          gp_ld32(acc + c, vg);
          if (glu) gp_ld32(acc + BN / 2 + c, vu);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          const int col0 = col_t + c;
          if (col0 >= p.n_out) continue;
#pragma unroll
          for (int j = 0; j < 32; j += 8) {
            if (col0 + j >= p.n_out) break;
            float f[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) f[k] = __uint_as_float(vg[j + k]);
            if (SCALED) {
#pragma unroll
              for (int k = 0; k < 8; ++k) f[k] *= sg[j + k];
            }
            if (p.bias != nullptr) {
#pragma unroll
              for (int k = 0; k < 8; ++k) f[k] += __bfloat162float(p.bias[eo + col0 + j + k]);
            }
            if (glu) {
              float up[8];
#pragma unroll
              for (int k = 0; k < 8; ++k) up[k] = __uint_as_float(vu[j + k]);
              if (SCALED) {
#pragma unroll
                for (int k = 0; k < 8; ++k) up[k] *= su[j + k];
              }
              if (p.bias != nullptr) {
#pragma unroll
                for (int k = 0; k < 8; ++k) up[k] += __bfloat162float(p.bias[eo + p.n_out + col0 + j + k]);
              }
              // the activation is chosen once for eight values: chosen for each, they ran one after the other
              if (p.act == 1) {
#pragma unroll
                for (int k = 0; k < 8; ++k) f[k] = silu(f[k]) * up[k];
              } else if (p.act == 4) {     // (clamp(up, -limit, limit) + 1) * g * sigmoid(alpha g), g = min(gate, limit)
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                  const float g = fminf(f[k], p.limit), u = fminf(fmaxf(up[k], -p.limit), p.limit);
                  f[k] = (u + 1.f) * g * (1.f / (1.f + __expf(-p.alpha * g)));
                }
              } else {
#pragma unroll
                for (int k = 0; k < 8; ++k) f[k] = (p.act == 2 ? gelu_tanh(f[k]) : gelu_erf(f[k])) * up[k];
              }
            }
            uint4* at = stg_at(lane, (c - c0 + j) >> 3);
            if (p.residual != nullptr) {
              const uint4 r = *at;
              f[0] += bf16lo(r.x); f[1] += bf16hi(r.x); f[2] += bf16lo(r.y); f[3] += bf16hi(r.y);
              f[4] += bf16lo(r.z); f[5] += bf16hi(r.z); f[6] += bf16lo(r.w); f[7] += bf16hi(r.w);
            }
            *at = make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
          }
        }
        move_rows(row0, row_end, col_t + c0, false);
      }
      // this warp has read its lanes of the buffer: back to the pair's issuer
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0)
        asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(gp_leader(&tmem_empty[buf])) : "memory");
      ++tc;
    }
  }
  if (*stop) __nanosleep(1000000);        // gave up: let copies in flight land before the shared memory goes away
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  gp_cluster_sync();                      // the peer no longer reads this CTA's operands or arrives on its barriers
  if (warp == 2) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(2 * BN));
  }
}

typedef CUresult (*GpEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                               const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static void gp_map(CUtensorMap* tm, const void* ptr, long long rows, int K, long long ld, int box_rows) {
  static GpEncodeFn fn = [] {
    void* q = nullptr;
    cudaDriverEntryPointQueryResult r;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &q, cudaEnableDefault, &r) != cudaSuccess || q == nullptr)
      throw std::runtime_error("cuTensorMapEncodeTiled not available");
    return reinterpret_cast<GpEncodeFn>(q);
  }();
  cuuint64_t gdim[2] = {(cuuint64_t)K, (cuuint64_t)rows}, gstride[1] = {(cuuint64_t)ld * 2};
  cuuint32_t box[2] = {(cuuint32_t)GP_BK, (cuuint32_t)box_rows}, estr[2] = {1, 1};
  CUresult r = fn(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) throw std::runtime_error("cuTensorMapEncodeTiled (gemm pair) failed: " + std::to_string((int)r));
}

static int gp_sms() {
  static int n = [] {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    return v;
  }();
  return n;
}

// a [M, K] (row stride lda), b [experts * N, K], c [M, n_out]; tile_expert / tile_row (device, [m_tiles]) for the grouped flavour
void gemm_pair_launch(const void* a, long long lda, const void* b, const void* bias, const void* residual, void* c, int M, int N, int K, int act,
                      cudaStream_t stream, bool w_fresh, const int* tile_expert, const int* tile_row, int m_tiles, int experts, float limit, float alpha,
                      const float* scale, int scale_n) {
  if (K % GP_BK != 0 || M < 1) throw std::runtime_error("gemm pair: K must be a multiple of 64");
  PairParams p{};
  const bool glu = act != 0;
  p.bias = reinterpret_cast<const __nv_bfloat16*>(bias);
  p.residual = reinterpret_cast<const __nv_bfloat16*>(residual);
  p.c = reinterpret_cast<__nv_bfloat16*>(c);
  p.scale = scale; p.scale_one = scale_n == 1 ? 1 : 0;
  p.M = M; p.N = N; p.K = K; p.act = act; p.n_out = glu ? N / 2 : N; p.limit = limit; p.alpha = alpha;
  check_waits();
  p.wait_word = wait_word(WAIT_GEMM_PAIR);
  count_launch(COUNT_GEMM_PAIR);
  p.tile_expert = tile_expert; p.tile_row = tile_row; p.w_fresh = w_fresh ? 1 : 0;
  const int tile_out = glu ? GP_BN / 2 : GP_BN;
  p.m_tiles = tile_expert != nullptr ? m_tiles : (M + 255) / 256;
  p.n_tiles = (p.n_out + tile_out - 1) / tile_out;
  p.band = tile_expert == nullptr ? p.m_tiles : std::min(4, p.m_tiles);
  gp_map(&p.tma_a, a, M, K, lda, 128);
  gp_map(&p.tma_b, b, (long long)experts * N, K, K, GP_BN / 2);
  auto kernel = scale != nullptr ? gemm_pair_kernel<true> : gemm_pair_kernel<false>;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, GP_SMEM) != cudaSuccess)
    throw std::runtime_error("gemm pair: shared memory size refused");
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(2 * std::min(gp_sms() / 2, p.m_tiles * p.n_tiles));
  cfg.blockDim = dim3(GP_THREADS);
  cfg.dynamicSmemBytes = GP_SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, p);
  if (e != cudaSuccess) throw std::runtime_error(std::string("gemm pair launch failed: ") + cudaGetErrorString(e));
}

}  // namespace nxdi
