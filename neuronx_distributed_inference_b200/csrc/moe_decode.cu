// MoE token-generation kernels: the routed experts of a decode step (T <= 8 tokens, top-k experts each) as two batched
// weight-streaming launches over (token, slot) pairs — no host-side dispatch, no data-dependent shapes, CUDA-graph safe.
//   K1  u[p, :] = silu(x_t . Wg_e^T) * (x_t . Wu_e^T)        W_gate_up [E, 2I, H]  (rows [0,I) gate, [I,2I) up)
//   K2  y[p, :] = u[p, :] . Wd_e^T                           W_down    [E, H, I]
// with p = (t, j), e = topk_i[t, j] - expert_offset; pairs routed to an expert that lives on another EP rank produce zeros.
// The combine  out[t] = sum_j w[t, j] * y[(t, j)]  is fused into K2's epilogue through fp32 atomics on a zeroed [T, H] buffer.
// reference kernels replaced: K16 moe_token_gen_all_experts / fused MoE TKG kernels (moe_v2.py), K17 for T <= 8.
//
// Bound by the experts' bytes.  A warp has one unit: a gate row and its up row, four rows of the down product, or one of 2048 columns or more; its lanes stride the
// reduction dimension with eight 16-byte weight loads in flight each (a ragged end is zeros, not a loop of its own), over x / u staged in shared memory once per CTA.
// grid = (pairs, units / 8): CTAs with fewer rows than warps in their last round, or one CTA more than fits, cost as much as a whole round or wave, and short CTAs
// even out; the pairs are next to one another, so that when two tokens pick the same expert the second read of a row comes from L2.  K2 starts while K1 runs and
// requests its first weights before it waits for u.
// MoE layer with norm, router and residual, us in a graph, this / 148 x 4 CTAs of uneven rows after a fill kernel: 4 of 16 experts 6144 x 1344, 1 token
// 53 / 73, 2 tokens 78 / 104; 8 of 128 2048 x 768: 30 / 42, 42 / 54; 2 of 8 4096 x 14336, 1 token: 128 / 140.
#include <stdexcept>

#include "api.h"
#include "common.cuh"

namespace nxdi {

constexpr int MOE_THREADS = 256, MOE_CTAS = 4;

template <bool GLU, int S>   // S: weight rows of a warp's unit (gate and up; 4 rows of the down product, or 1 of 256 loads or more)
__global__ void __launch_bounds__(MOE_THREADS, MOE_CTAS) moe_rows_kernel(const __nv_bfloat16* __restrict__ xin,   // K1: x [T,K]; K2: u [P,K]
                                                                const __nv_bfloat16* __restrict__ W,     // [E, N_rows, K]
                                                                const int* __restrict__ topk_i, int id_step,   // [P]; 2: the low words of int64 ids
                                                                const float* __restrict__ topk_w,         // [P] (K2 only)
                                                                __nv_bfloat16* __restrict__ u_out,        // K1: [P, N]
                                                                float* __restrict__ y_acc,                // [T, n_y] fp32: K1 clears it, K2 adds (atomics)
                                                                int n_y, int K, int N, int topk, int E, int expert_offset, int act, float limit, float alpha) {
  constexpr int D = 8 / S;                                // 16-byte loads of each row in flight
  extern __shared__ __align__(16) uint8_t smem[];
  uint4* xs = reinterpret_cast<uint4*>(smem);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int p = blockIdx.x, t = p / topk;
  if (GLU) {
    pdl_wait();
    pdl_launch_dependents();     // after the wait: the ids are written when K2 starts, so it reads them, and its first weights, before its own wait
    for (int c = (blockIdx.y * gridDim.x + blockIdx.x) * MOE_THREADS + tid; c < n_y; c += gridDim.x * gridDim.y * MOE_THREADS) y_acc[c] = 0.f;
  }
  const int e = __ldcg(topk_i + (size_t)p * id_step) - expert_offset;
  const bool mine = e >= 0 && e < E;                      // else the expert is owned by another rank
  const int unit = blockIdx.y * (MOE_THREADS / 32) + warp;
  const bool work = unit < (GLU ? N : (N + S - 1) / S);
  if (!mine) {
    if (GLU && work && lane == 0) u_out[(size_t)p * N + unit] = __float2bfloat16(0.f);
    if (!GLU) pdl_wait();        // K2 must not be complete before K1, which clears y_acc for the kernel after
    return;
  }
  const int nvec = K >> 3;
  const __nv_bfloat16* We = W + (size_t)e * ((size_t)(GLU ? 2 : 1) * N) * K;
  uint4 w[S][D];
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  auto load = [&](int v) {
#pragma unroll
    for (int s = 0; s < S; ++s) {
      const int r = GLU ? unit + s * N : min(unit * S + s, N - 1);
      const uint4* wr = reinterpret_cast<const uint4*>(We + (size_t)r * K);
#pragma unroll
      for (int d = 0; d < D; ++d) w[s][d] = v + 32 * d < nvec ? ldg_stream(wr + v + 32 * d) : zero;
    }
  };
  if (work) load(lane);
  if (!GLU) {
    pdl_wait();
    pdl_launch_dependents();
  }
  const uint4* src = reinterpret_cast<const uint4*>(xin + (size_t)(GLU ? t : p) * K);
  for (int v = tid; v < nvec; v += MOE_THREADS) xs[v] = __ldcg(src + v);
  __syncthreads();
  auto dot8 = [](const uint4& a, const uint4& b) {
    return bf16lo(a.x) * bf16lo(b.x) + bf16hi(a.x) * bf16hi(b.x) + bf16lo(a.y) * bf16lo(b.y) + bf16hi(a.y) * bf16hi(b.y) +
           bf16lo(a.z) * bf16lo(b.z) + bf16hi(a.z) * bf16hi(b.z) + bf16lo(a.w) * bf16lo(b.w) + bf16hi(a.w) * bf16hi(b.w);
  };
  if (!work) return;
  float acc[S];
#pragma unroll
  for (int s = 0; s < S; ++s) acc[s] = 0.f;
  for (int v = lane; v < nvec; v += 32 * D) {
    if (v >= 32 * D) load(v);
    uint4 xv[D];
#pragma unroll
    for (int d = 0; d < D; ++d) xv[d] = v + 32 * d < nvec ? xs[v + 32 * d] : zero;
#pragma unroll
    for (int s = 0; s < S; ++s) {
      float sum = dot8(w[s][0], xv[0]);
#pragma unroll
      for (int d = 1; d < D; ++d) sum += dot8(w[s][d], xv[d]);
      acc[s] += sum;
    }
  }
#pragma unroll
  for (int s = 0; s < S; ++s) acc[s] = warp_sum(acc[s]);
  if (GLU) {
    if (lane == 0) {
      float u = silu(acc[0]) * acc[1];
      if (act == 4) {      // clamped, shifted gate product
        const float g = fminf(acc[0], limit);
        u = g / (1.f + __expf(-alpha * g)) * (fminf(fmaxf(acc[1], -limit), limit) + 1.f);
      }
      u_out[(size_t)p * N + unit] = __float2bfloat16(u);
    }
  } else {
#pragma unroll
    for (int s = 0; s < S; ++s)
      if (lane == s && unit * S + s < N) atomicAdd(y_acc + (size_t)t * N + unit * S + s, topk_w[p] * acc[s]);
  }
}

void moe_decode_launch(const void* x, const void* w_gate_up, const void* w_down, const float* topk_w, const int* topk_i, int id_step, void* u,
                       float* y_acc, int T, int topk, int H, int I, int E, int expert_offset, int act, float limit, float alpha,
                       cudaStream_t stream) {
  const int P = T * topk;
  if (H % 8 != 0 || I % 8 != 0) throw std::runtime_error("moe_decode: H and I must be multiples of 8");
  auto ctas = [](int units) { return (units + MOE_THREADS / 32 - 1) / (MOE_THREADS / 32); };
  const int down_rows = I >= 2048 ? 1 : 4;                // a row of 2048 columns is eight loads of a warp
  auto k1 = moe_rows_kernel<true, 2>;
  auto k2 = down_rows == 1 ? moe_rows_kernel<false, 1> : moe_rows_kernel<false, 4>;
  static bool configured = false;
  if (!configured) {
    cudaFuncSetAttribute(k1, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024);
    cudaFuncSetAttribute(moe_rows_kernel<false, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024);
    cudaFuncSetAttribute(moe_rows_kernel<false, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024);
    configured = true;
  }
  if ((size_t)H * 2 > 64 * 1024 || (size_t)I * 2 > 64 * 1024) throw std::runtime_error("moe_decode: row too wide for shared memory");
  launch_pdl(k1, dim3(P, ctas(I)), dim3(MOE_THREADS), (size_t)H * 2, stream, reinterpret_cast<const __nv_bfloat16*>(x),
             reinterpret_cast<const __nv_bfloat16*>(w_gate_up), topk_i, id_step, topk_w, reinterpret_cast<__nv_bfloat16*>(u),
             y_acc, T * H, H, I, topk, E, expert_offset, act, limit, alpha);
  launch_pdl(k2, dim3(P, ctas((H + down_rows - 1) / down_rows)), dim3(MOE_THREADS), (size_t)I * 2, stream, reinterpret_cast<const __nv_bfloat16*>(u),
             reinterpret_cast<const __nv_bfloat16*>(w_down), topk_i, id_step, topk_w, static_cast<__nv_bfloat16*>(nullptr), y_acc, 0, I, H, topk,
             E, expert_offset, act, limit, alpha);
}

}  // namespace nxdi
