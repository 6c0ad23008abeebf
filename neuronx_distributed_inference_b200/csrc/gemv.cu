// Launchers for the weight-streaming skinny GEMM (see gemv.cuh) and the stand-alone RMSNorm.
#include <algorithm>

#include "gemv.cuh"

namespace nxdi {

static int num_sms() {
  static int n = 0;
  if (n == 0) {
    int dev;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  }
  return n;
}

size_t gemv_smem_bytes(int T, int K, bool x_in_smem) {
  return (x_in_smem ? (size_t)T * (K * 2 + 64) : 0) + (2 * GEMV_WARPS * 128 + 64) * sizeof(float);
}

template <bool GLU>
static void launch_gemv(const GemvParams& p, cudaStream_t stream) {
  auto kern = gemv_kernel<GLU>;
  const size_t smem = gemv_smem_bytes(p.T, p.K, p.x_in_smem);
  static bool configured = false;
  if (!configured) {
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    configured = true;
  }
  const int n_tiles = GLU ? ((p.N / 2) + 7) / 8 : (p.N + 15) / 16;
  const int per_sm = smem <= 112 * 1024 ? 2 : 1;
  const int grid = std::min(n_tiles, per_sm * num_sms());
  launch_pdl(kern, dim3(grid), dim3(GEMV_THREADS), smem, stream, p);
}

void gemv_launch(const GemvParams& p, int mode, cudaStream_t stream) {
  const bool glu = p.act != ACT_NONE;
  if (mode != 0) throw std::runtime_error("gemv v1: the fused all-reduce lives in gemv2 (activations must fit shared memory)");
  if (glu) launch_gemv<true>(p, stream);
  else launch_gemv<false>(p, stream);
}

// rmsnorm kernel (also used to pre-normalise x when T*K does not fit the GEMV's shared memory)
// CLEAR: words that the kernel behind this one counts in are set to zero on the way.  CTAS: blocks per SM, two with 94 registers or three with 80; three where that
// saves a wave.  us in a graph, three / two: 296 rows of 8192 3.2 / 2.8, 350 3.1 / 4.4, 512 4.9 / 4.7, 740 5.2 / 5.9, 1023 6.4 / 7.1; 4096 of 16384 52 / 61.
template <bool CLEAR, int CTAS>
__global__ void __launch_bounds__(256, CTAS) rmsnorm_kernel(const __nv_bfloat16* __restrict__ x,
                                                      const __nv_bfloat16* __restrict__ res_in,
                                                      const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ y,
                                                      __nv_bfloat16* __restrict__ res_out, int H, float eps, float offset,
                                                      unsigned* __restrict__ clear, int n_clear) {
  __shared__ float sred[8];
  pdl_launch_dependents();
  pdl_wait();
  if (CLEAR && blockIdx.x == 0)
    for (int i = threadIdx.x; i < n_clear; i += 256) clear[i] = 0u;
  const int row = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint4* xr = reinterpret_cast<const uint4*>(x + (size_t)row * H);
  const uint4* rr = res_in ? reinterpret_cast<const uint4*>(res_in + (size_t)row * H) : nullptr;
  uint4* ro = res_out ? reinterpret_cast<uint4*>(res_out + (size_t)row * H) : nullptr;
  const int nvec = H >> 3;
  constexpr int MAXV = 8;  // up to H = 16384 in registers
  float v[MAXV][8];
  float acc = 0.f;
#pragma unroll
  for (int i = 0; i < MAXV; ++i) {
    const int idx = tid + i * 256;
    if (idx < nvec) {
      uint4 q = xr[idx];
      float f[8] = {bf16lo(q.x), bf16hi(q.x), bf16lo(q.y), bf16hi(q.y), bf16lo(q.z), bf16hi(q.z), bf16lo(q.w), bf16hi(q.w)};
      if (rr) {
        uint4 r = rr[idx];
        float g[8] = {bf16lo(r.x), bf16hi(r.x), bf16lo(r.y), bf16hi(r.y), bf16lo(r.z), bf16hi(r.z), bf16lo(r.w), bf16hi(r.w)};
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] = __bfloat162float(__float2bfloat16(f[j] + g[j]));  // residual stream is bf16
        if (ro) ro[idx] = make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        v[i][j] = f[j];
        acc += f[j] * f[j];
      }
    }
  }
  acc = warp_sum(acc);
  if (lane == 0) sred[warp] = acc;
  __syncthreads();
  float tot = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) tot += sred[i];
  const float rstd = rsqrtf(tot / (float)H + eps);
  const uint4* wr = reinterpret_cast<const uint4*>(w);
  uint4* yr = reinterpret_cast<uint4*>(y + (size_t)row * H);
#pragma unroll
  for (int i = 0; i < MAXV; ++i) {
    const int idx = tid + i * 256;
    if (idx < nvec) {
      uint4 g = wr[idx];
      float gm[8] = {bf16lo(g.x), bf16hi(g.x), bf16lo(g.y), bf16hi(g.y), bf16lo(g.z), bf16hi(g.z), bf16lo(g.w), bf16hi(g.w)};
      float o[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = v[i][j] * rstd * (gm[j] + offset);
      yr[idx] = make_uint4(pack_bf16(o[0], o[1]), pack_bf16(o[2], o[3]), pack_bf16(o[4], o[5]), pack_bf16(o[6], o[7]));
    }
  }
}

// Many rows: WR warps per row, the row in registers as it came, eight 16-byte pieces a lane, so that an SM has 128 KB of reads in flight (one block per
// row: 32 KB).  Bound by HBM and a load's latency; us, here / one block per row, inputs larger than L2, launches one after the other: 4096 x 4096 15.2 / 26.0,
// 4096 x 2048 8.1 / 21.1, 2048 x 6144 12.0 / 16.0, 1024 x 4096 6.8 / 8.3 (0.1 to 0.6 of that for the sums in the other kernel's order); a warp per row with 16
// or 32 pieces a lane: 23.1 and 19.9 for the first and the third.
template <int WR>
__global__ void __launch_bounds__(256, 4) rmsnorm_rows_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ res_in, const __nv_bfloat16* __restrict__ w,
                                                              __nv_bfloat16* __restrict__ y, __nv_bfloat16* __restrict__ res_out, int rows, int H, float eps,
                                                              float offset) {
  constexpr int NV = 8;
  __shared__ float part[8 / WR][8];
  pdl_launch_dependents();
  pdl_wait();
  const int warp = threadIdx.x >> 5, row = blockIdx.x * (8 / WR) + warp / WR, i0 = (warp % WR) * 32 + (threadIdx.x & 31);
  const int nvec = row < rows ? H >> 3 : 0;
  const uint4* xr = reinterpret_cast<const uint4*>(x + (size_t)row * H);
  uint4 v[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) v[i] = i0 + i * 32 * WR < nvec ? xr[i0 + i * 32 * WR] : make_uint4(0u, 0u, 0u, 0u);
  if (res_in) {
    const uint4* rr = reinterpret_cast<const uint4*>(res_in + (size_t)row * H);
    uint4* ro = res_out ? reinterpret_cast<uint4*>(res_out + (size_t)row * H) : nullptr;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int idx = i0 + i * 32 * WR;
      if (idx >= nvec) continue;
      const uint4 r = rr[idx], q = v[i];          // residual stream is bf16
      v[i] = make_uint4(pack_bf16(bf16lo(q.x) + bf16lo(r.x), bf16hi(q.x) + bf16hi(r.x)), pack_bf16(bf16lo(q.y) + bf16lo(r.y), bf16hi(q.y) + bf16hi(r.y)),
                        pack_bf16(bf16lo(q.z) + bf16lo(r.z), bf16hi(q.z) + bf16hi(r.z)), pack_bf16(bf16lo(q.w) + bf16lo(r.w), bf16hi(q.w) + bf16hi(r.w)));
      if (ro) ro[idx] = v[i];
    }
  }
  // The sums of rmsnorm_kernel, in its order, so that a row has the same bits however many rows a call has: piece i of this lane belongs to that kernel's
  // thread (i0 + 32 WR i) mod 256, whose warp is warp % WR + WR (i mod NS).
  constexpr int NS = NV / WR;
  float s[NS] = {};
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const float f[8] = {bf16lo(v[i].x), bf16hi(v[i].x), bf16lo(v[i].y), bf16hi(v[i].y), bf16lo(v[i].z), bf16hi(v[i].z), bf16lo(v[i].w), bf16hi(v[i].w)};
#pragma unroll
    for (int j = 0; j < 8; ++j) s[i % NS] += f[j] * f[j];
  }
#pragma unroll
  for (int i = 0; i < NS; ++i) s[i] = warp_sum(s[i]);
  float acc = 0.f;
  if (WR == 1) {
#pragma unroll
    for (int i = 0; i < NS; ++i) acc += s[i];
  } else {
    if ((threadIdx.x & 31) == 0)
#pragma unroll
      for (int i = 0; i < NS; ++i) part[warp / WR][warp % WR + WR * i] = s[i];
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 8; ++i) acc += part[warp / WR][i];
  }
  const float rstd = rsqrtf(acc / (float)H + eps);
  const uint4* wr = reinterpret_cast<const uint4*>(w);
  uint4* yr = reinterpret_cast<uint4*>(y + (size_t)row * H);
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int idx = i0 + i * 32 * WR;
    if (idx >= nvec) continue;
    const uint4 g = __ldg(wr + idx);
    const uint32_t a[4] = {v[i].x, v[i].y, v[i].z, v[i].w}, b[4] = {g.x, g.y, g.z, g.w};
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) o[j] = pack_bf16(bf16lo(a[j]) * rstd * (bf16lo(b[j]) + offset), bf16hi(a[j]) * rstd * (bf16hi(b[j]) + offset));
    yr[idx] = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

void rmsnorm_launch(const void* x, const void* res_in, const void* w, void* y, void* res_out, int rows, int H, float eps,
                    float offset, cudaStream_t stream, unsigned* clear, int n_clear) {
  if (n_clear > 0 && rows >= 1024) throw std::runtime_error("rmsnorm: words are cleared beside fewer than 1024 rows");
  // enough rows to fill the SMs that way; fewer, where a row's latency counts: a block per row
  if (rows >= 1024 && H <= 8192) {
    auto go = [&](auto kernel, int per_block) {
      launch_pdl(kernel, dim3((rows + per_block - 1) / per_block), dim3(256), 0, stream, reinterpret_cast<const __nv_bfloat16*>(x),
                 reinterpret_cast<const __nv_bfloat16*>(res_in), reinterpret_cast<const __nv_bfloat16*>(w), reinterpret_cast<__nv_bfloat16*>(y),
                 reinterpret_cast<__nv_bfloat16*>(res_out), rows, H, eps, offset);
    };
    if (H <= 2048) go(rmsnorm_rows_kernel<1>, 8);
    else if (H <= 4096) go(rmsnorm_rows_kernel<2>, 4);
    else go(rmsnorm_rows_kernel<4>, 2);
    return;
  }
  auto waves = [&](int ctas) { return (rows + ctas * kNumSMs - 1) / (ctas * kNumSMs); };
  const bool three = waves(3) < waves(2);
  launch_pdl(n_clear > 0 ? (three ? rmsnorm_kernel<true, 3> : rmsnorm_kernel<true, 2>) : three ? rmsnorm_kernel<false, 3> : rmsnorm_kernel<false, 2>, dim3(rows), dim3(256), 0, stream, reinterpret_cast<const __nv_bfloat16*>(x),
             reinterpret_cast<const __nv_bfloat16*>(res_in), reinterpret_cast<const __nv_bfloat16*>(w),
             reinterpret_cast<__nv_bfloat16*>(y), reinterpret_cast<__nv_bfloat16*>(res_out), H, eps, offset, clear, n_clear);
}

}  // namespace nxdi
