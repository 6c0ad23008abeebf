// pybind11 surface of the sm_100a extension (neuronx_distributed_inference_b200._C).  Compiled by the host
// compiler; the CUDA translation units expose raw-pointer launchers (api.h).
#include <limits>
#include <torch/extension.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <cuda_runtime.h>

#include "api.h"

namespace nxdi {

#define NXDI_CUDA_OK(call)                                                        \
  do {                                                                            \
    cudaError_t e__ = (call);                                                     \
    TORCH_CHECK(e__ == cudaSuccess, #call, " failed: ", cudaGetErrorString(e__)); \
  } while (0)

static inline cudaStream_t cur_stream() { return at::cuda::getCurrentCUDAStream(); }
static inline const void* optr(const c10::optional<at::Tensor>& t) { return t.has_value() ? t->data_ptr() : nullptr; }
static inline bool is_bf16(const at::Tensor& t) { return t.scalar_type() == at::kBFloat16; }

// ---- rmsnorm ------------------------------------------------------------------------------------------
constexpr int64_t RMSNORM_MAX_H = 16384;
// the kernels read a norm's weight as K bf16 values side by side
static void check_norm_weight(const at::Tensor& w, int64_t K) {
  TORCH_CHECK(w.is_cuda() && is_bf16(w) && w.numel() == K && w.is_contiguous(), "norm weight: ", K, " contiguous bf16 values on the GPU expected");
}
// x [.., H], a residual like it; clear: words set to zero on the way (the tickets of the GEMM that follows)
static at::Tensor rmsnorm_rows(const at::Tensor& x, const at::Tensor& w, double eps, double offset, const at::Tensor* residual, at::Tensor* res_out,
                               unsigned* clear = nullptr, int n_clear = 0) {
  TORCH_CHECK(x.is_cuda() && is_bf16(x) && x.is_contiguous());
  const int64_t H = x.size(-1), rows = H ? x.numel() / H : 0;
  check_norm_weight(w, H);
  TORCH_CHECK(H % 8 == 0 && H <= RMSNORM_MAX_H, "rmsnorm: hidden must be a multiple of 8 and <= 16384");
  c10::cuda::CUDAGuard guard(x.device());
  auto y = at::empty_like(x);
  if (residual != nullptr) {
    TORCH_CHECK(residual->is_contiguous() && residual->numel() == x.numel() && residual->size(-1) == H && is_bf16(*residual));
    *res_out = at::empty_like(x);
  }
  rmsnorm_launch(x.data_ptr(), residual != nullptr ? residual->data_ptr() : nullptr, w.data_ptr(), y.data_ptr(), residual != nullptr ? res_out->data_ptr() : nullptr,
                 (int)rows, (int)H, (float)eps, (float)offset, cur_stream(), clear, n_clear);
  return y;
}
std::tuple<at::Tensor, at::Tensor> rmsnorm(const at::Tensor& x, const at::Tensor& w, double eps, double offset, const c10::optional<at::Tensor>& residual) {
  TORCH_CHECK(x.dim() >= 1);
  const auto xc = x.contiguous(), wc = w.contiguous();          // (a slice of a wider projection arrives strided)
  if (!residual.has_value()) {
    auto y = rmsnorm_rows(xc, wc, eps, offset, nullptr, nullptr);
    return {y, y};
  }
  at::Tensor r;
  const auto rc = residual->contiguous();
  auto y = rmsnorm_rows(xc, wc, eps, offset, &rc, &r);
  return {y, r};
}

static void run_gemv(GemvParams& p, int mode) {
  const int wt = p.scale != nullptr ? p.wdtype : 0;
  if (gemv2_supported(p.T, p.K, wt) && p.x_in_smem) {
    const bool glu = p.act != 0;
    const int n_tiles = gemv2_ntiles(p.N, glu);
    const auto ws = workspace(cur_stream(), (int64_t)n_tiles * gemv2_pmax(p.N, p.K, glu, wt) * 128, 0, n_tiles);
    gemv2_launch(p, mode, ws.f, ws.tickets, cur_stream());
  } else {
    TORCH_CHECK(wt == 0, "gemv: 8-bit weights need the TMA streaming kernel");
    TORCH_CHECK(p.K % 256 == 0, "gemv: K must be a multiple of 256 on the wide-activation fallback");
    gemv_launch(p, mode, cur_stream());
  }
}

// ---- skinny GEMM ----------------------------------------------------------------------------------------
static void fill_params(GemvParams& p, const at::Tensor& x, const at::Tensor& w, const c10::optional<at::Tensor>& bias,
                        const c10::optional<at::Tensor>& norm_w, double eps, double offset, int act,
                        const c10::optional<at::Tensor>& residual, const c10::optional<at::Tensor>& scale, at::Tensor& y,
                        bool x_in_smem) {
  p.x = x.data_ptr();
  p.w = w.data_ptr();
  p.bias = optr(bias);
  p.norm_w = x_in_smem ? optr(norm_w) : nullptr;
  p.residual = optr(residual);
  p.scale = scale.has_value() ? scale->data_ptr<float>() : nullptr;
  p.scale_n = scale.has_value() ? (int)scale->numel() : 0;
  p.y = y.data_ptr();
  p.T = x.size(0);
  p.K = x.size(1);
  p.N = w.size(0);
  p.ldx = x.stride(0);
  p.ldy = y.stride(0);
  p.eps = (float)eps;
  p.norm_offset = (float)offset;
  p.act = act;
  p.x_in_smem = x_in_smem ? 1 : 0;
  p.wdtype = w.scalar_type() == at::kBFloat16 ? 0 : (w.scalar_type() == at::kChar ? 1 : 2);
}

static at::Tensor prenorm_if_needed(const at::Tensor& x, const c10::optional<at::Tensor>& norm_w, double eps, double offset,
                                    bool& x_in_smem) {
  x_in_smem = gemv_smem_bytes(x.size(0), x.size(1), true) <= 220 * 1024;
  if (!x_in_smem && norm_w.has_value()) return rmsnorm_rows(x.contiguous(), *norm_w, eps, offset, nullptr, nullptr);
  return x;
}

static void check_gemv_inputs(const at::Tensor& x, const at::Tensor& w) {
  TORCH_CHECK(x.is_cuda() && w.is_cuda() && x.dim() == 2 && w.dim() == 2 && x.size(1) == w.size(1));
  TORCH_CHECK(is_bf16(x) && is_bf16(w), "gemv: bf16 activations and weights");
  TORCH_CHECK(x.size(0) >= 1 && x.size(0) <= GEMV_MAX_T, "gemv: 1..8 tokens");
  TORCH_CHECK(x.size(1) % 64 == 0 && x.stride(1) == 1 && x.stride(0) % 8 == 0 && w.is_contiguous());
}

// Where the swapped, evenly split GEMM (skinny_gemm.cu) beats the 128-row token tiles of gemm_tcgen05.cu (us in a graph, skinny / tiles; 16, 32, 48, 64 and 128 tokens):
//   gate|up 28672 x 4096: 42 / 44, 44 / 44, 47 / 45, 49 / 45, 57 / 45     17280 x 3200: 24 / 24, 26 / 24, 29 / 24, 30 / 24, 37 / 25
//           16384 x 4096: 27 / 28, 29 / 29, 32 / 29, 33 / 29, 41 / 30     16384 x 2048: 16 / 25, 18 / 16, 20 / 16, 21 / 16, 28 / 16
//           12288 x 4096: 22 / 26, 24 / 27, 26 / 27, 28 / 27, 34 / 27     10240 x 5120: 24 / 30, 26 / 30, 28 / 30, 30 / 31, 37 / 31
//   plain 4096 x 14336:   25 / 50, 26 / 50, 28 / 51, 29 / 51, 35 / 52     12288 x 4096: 21 / 28, 22 / 29, 26 / 29, 27 / 29, 33 / 30 (80 tokens 29 / 30, 96 31 / 30)
//          4096 x 4096:   12 / 21, 13 / 21, 15 / 21, 15 / 21, 20 / 22      6144 x 4096: 14 / 21, 15 / 22, 17 / 22, 17 / 22, 22 / 22
//          2048 x 2048:    8 / 15,  8 / 14, 10 / 14, 10 / 14, 14 / 14      4096 x 1024:  8 / 8,   8 / 8,  10 / 8,  10 / 7,  13 / 8
//   at 65, 80 and 128:    8192 x 2048: 15 / 12, 15 / 12, 17 / 12    17280 x 3200: 28 / 24, 28 / 24, ..    3200 x 3200: 14 / 17, 15 / 17, 19 / 17
//   gate|up at 33 and 64: 2048 x 4096: 18 / 16, 22 / 16    1024 x 7168: 23 / 18, 28 / 18    2048 x 5120: 21 / 17, 25 / 17
// A feature's tokens are in one lane, so its epilogue and the fix-up of the cut tiles grow with the tokens, twice as fast with a gate product, while the tile kernel's
// time does not change up to 128; deep K leaves the tile kernel few tiles.  Between other kernels it gains what it prefetches: a whole gated MLP takes 75.0 / 74.9 us at 33
// tokens, 75.9 / 75.2 at 40 with 28672 x 4096 and 62.8 / 63.9, 63.2 / 64.1 with 22016 x 4096.  The line at 40 tokens is the break-even of these two.  Gate products of
// 16384 x 4096 stay here up to 64 tokens, where the tiles have been ahead since their MMA warp issues from uniform code (31 / 29 at 33, 33 / 29 at 64).
static bool skinny_pays(int M, int rows, int K, bool glu) {
  const long long size = (long long)rows * K;
  if (glu) return M <= 32 || (M <= 40 && size >= (64LL << 20)) || (M <= 64 && rows <= 16384 && K >= (rows >= 4096 ? 4096 : 8192));
  return M <= 64 || (M <= SKINNY_MAX_T && (K >= 2 * rows || (K >= 4096 && size >= (8LL << 20) && (M <= 80 || size < (32LL << 20))) || (K >= 3072 && rows <= 8192 && M <= 80)));
}

// norm_w: x is normalised first; its kernel clears the GEMM's tickets, which else takes a launch of its own (1.5 us in the stream)
static void run_skinny(at::Tensor x, const at::Tensor& w, const c10::optional<at::Tensor>& bias, int act, const c10::optional<at::Tensor>& residual,
                       at::Tensor& y, bool fresh_weight, const c10::optional<at::Tensor>& norm_w = c10::nullopt, double eps = 0., double offset = 0.,
                       const at::Tensor* scale = nullptr) {
  const int M = x.size(0);
  const int64_t nt = skinny_gemm_tickets(), nf = skinny_gemm_ws_floats(scale != nullptr ? skinny_gemm8_block(M) : M, act != 0);
  auto ws = at::empty({nf + nt}, x.options().dtype(at::kFloat));              // one per call: safe on any stream and inside captured graphs
  SkinnyGemm a{};
  a.ws = ws.data_ptr<float>();
  a.tickets = reinterpret_cast<unsigned*>(ws.data_ptr<float>() + nf);
  if (norm_w.has_value()) x = rmsnorm_rows(x.contiguous(), *norm_w, eps, offset, nullptr, nullptr, a.tickets, (int)nt);
  else skinny_clear_launch(a.tickets, (int)nt, cur_stream());
  a.x = x.data_ptr(); a.x_rows = M; a.ldx = x.stride(0); a.w = w.data_ptr(); a.bias = optr(bias); a.residual = optr(residual); a.y = y.data_ptr();
  a.experts = 1; a.tokens = M; a.n_out = y.size(1); a.K = x.size(1); a.act = act; a.limit = 7.f; a.alpha = 1.702f;
  a.w_fresh = fresh_weight ? 1 : 0;
  if (scale != nullptr) {
    a.wt = w.scalar_type() == at::kChar ? 1 : 2;
    a.scale = scale->data_ptr<float>();
    a.scale_n = (int)scale->numel();
  }
  skinny_gemm_launch(a, cur_stream());
}

at::Tensor gemv(const at::Tensor& x, const at::Tensor& w, const c10::optional<at::Tensor>& bias,
                const c10::optional<at::Tensor>& norm_w, double eps, double offset, int64_t act,
                const c10::optional<at::Tensor>& scale, const c10::optional<at::Tensor>& residual) {
  if (norm_w.has_value()) check_norm_weight(*norm_w, x.size(-1));
  if (scale.has_value()) {
    // weight-only quantised path (int8 / fp8-e4m3, per-channel or per-tensor scale)
    TORCH_CHECK(x.is_cuda() && w.is_cuda() && x.dim() == 2 && w.dim() == 2 && x.size(1) == w.size(1) && is_bf16(x));
    TORCH_CHECK(w.is_contiguous() && x.stride(1) == 1 && x.size(0) >= 1 && x.size(0) <= GEMV_MAX_T && x.size(1) % 16 == 0);
    const bool i8 = w.scalar_type() == at::kChar, f8 = w.scalar_type() == at::kFloat8_e4m3fn;
    TORCH_CHECK(i8 || f8, "qgemv: int8 or float8_e4m3fn weights");
    TORCH_CHECK(scale->scalar_type() == at::kFloat && scale->is_contiguous() && (scale->numel() == 1 || scale->numel() == w.size(0)));
    c10::cuda::CUDAGuard guard(x.device());
    const int N = w.size(0);
    const bool glu = act != 0;
    auto y = at::empty({x.size(0), glu ? N / 2 : N}, x.options());
    if (residual.has_value()) TORCH_CHECK(!glu && residual->is_contiguous() && residual->size(1) == N && is_bf16(*residual));
    // the TMA-streamed kernel (same ring as bf16, bytes expanded in registers) whenever the shapes allow it
    static const bool q2 = []() { const char* e = getenv("NXDI_B200_QGEMV2"); return e == nullptr || atoi(e) != 0; }();
    if (q2 && gemv2_supported((int)x.size(0), (int)x.size(1), i8 ? 1 : 2) && x.stride(0) % 8 == 0 && (!glu || N % 2 == 0)) {
      GemvParams p{};
      fill_params(p, x, w, bias, norm_w, eps, offset, (int)act, residual, scale, y, true);
      run_gemv(p, 0);
      return y;
    }
    // rows too wide for its shared memory (from 8 tokens of 11008, 7 of 14336): bytes expanded on the way to the tensor cores.  us in a graph, fp8 / one warp per
    // few weight rows: 4096 x 11008 at 8 tokens 16.6 / 98, 4096 x 14336 at 7 19.3 / 112, 1024 x 16384 at 6 12.3 / 59, 256 x 28672 at 4 14.1 / 64; int8 alike.  Both
    // keep products and sums in fp32 (errors against 64 bits are the same).  A norm stays with the warps, which scale the fp32 sums by 1 / rms instead of the rows.
    if (q2 && !norm_w.has_value() && x.stride(0) % 8 == 0 && y.size(1) % 8 == 0 && (!glu || N % 2 == 0) && skinny_gemm8_supported((int)x.size(0), (int)x.size(1), glu)) {
      run_skinny(x.contiguous(), w, bias, (int)act, residual, y, false, c10::nullopt, 0., 0., &*scale);
      return y;
    }
    static int n_sms = 0;
    if (n_sms == 0) n_sms = at::cuda::getCurrentDeviceProperties()->multiProcessorCount;
    qgemv_launch(x.data_ptr(), w.data_ptr(), scale->data_ptr<float>(), (int)scale->numel(), optr(bias), optr(norm_w), optr(residual),
                 y.data_ptr(), x.size(0), N, x.size(1), x.stride(0), y.stride(0), (int)act, i8 ? 1 : 2, (float)eps, (float)offset,
                 n_sms, cur_stream());
    return y;
  }
  check_gemv_inputs(x, w);
  c10::cuda::CUDAGuard guard(x.device());
  const int N = w.size(0);
  const bool glu = act != 0;
  if (glu) TORCH_CHECK(N % 2 == 0);
  auto y = at::empty({x.size(0), glu ? N / 2 : N}, x.options());
  if (residual.has_value())
    TORCH_CHECK(!glu && residual->is_contiguous() && residual->size(0) == x.size(0) && residual->size(1) == N && is_bf16(*residual));
  // rows too wide for the streaming kernel's shared memory (from 7 tokens of 14336, 8 of 11008).  us, here / one warp per weight row: 4096 x 14336 at 7 tokens
  // 26 / 57, at 8 26 / 36; 4096 x 11008 at 8 21 / 39.  With a norm, rows wider than its kernel takes stay with the kernel that normalises them itself
  if (!gemv2_supported(x.size(0), x.size(1), 0) && (glu ? N / 2 : N) % 8 == 0 && (!norm_w.has_value() || x.size(1) <= RMSNORM_MAX_H)) {
    run_skinny(x, w, bias, (int)act, residual, y, false, norm_w, eps, offset);
    return y;
  }
  bool x_in_smem;
  at::Tensor xn = prenorm_if_needed(x, norm_w, eps, offset, x_in_smem);
  GemvParams p{};
  fill_params(p, xn, w, bias, norm_w, eps, offset, (int)act, residual, scale, y, x_in_smem);
  run_gemv(p, 0);
  return y;
}

// Where 256 x 256 tiles on CTA pairs (gemm_pair.cu) beat the one-CTA tiles (us in a graph, pairs / one CTA, at 256, 384, 512 and 768 tokens):
//   gate|up 28672 x 4096: 57 / 64, 91 / 86, 95 / 111, 124 / 140     17280 x 3200: 28 / 32, 43 / 48, 43 / 50, 61 / 68     16384 x 2048: 20 / 23, 31 / 35, 29 / 33, 40 / 45
//           22016 x 4096: 51 / 60, 70 / 63, 73 / 88, 98 / 110
//   plain 12288 x 4096:   31 / 39, 47 / 40, 49 / 63, 58 / 68        6144 x 4096: 26 / 26, 28 / 26, 28 / 35, 31 / 36      4096 x 4096: 26 / 22, 27 / 25, 27 / 25, 28 / 33
//         4096 x 14336:   74 / 54, 75 / 75, 73 / 74, 78 / 91        2048 x 8192: 43 / 35, 44 / 35, 44 / 35, 44 / 53
// Up to 512 tokens the one-CTA kernel has smaller tiles and split-K to fill the chip; with 40 pair tiles or more (of 74 pairs) they are not needed, except up to 384
// tokens, a quarter of whose pair tiles is padding, where the last wave of pairs is short too.
static bool pair_pays(int M, int n_out, bool glu) {
  const int tiles = ((M + 255) / 256) * ((n_out + (glu ? 127 : 255)) / (glu ? 128 : 256)), waves = (tiles + 73) / 74;
  return M > 512 || (M > 128 && tiles >= 40 && (M <= 256 || M > 384 || 5 * tiles >= 4 * 74 * waves));
}


// fresh_weight: w was written by a kernel enqueued just before (an expanded 8-bit weight).  The kernels fetch a parameter's first tiles before the
// kernels in front of them have finished; such a weight has to be waited for.
// w_scale: of the sums, per output channel or one (a weight expanded from bytes; not in the kernel of few tokens).
// tcgen05 GEMM for T > 8 tokens (prefill, long speculation windows)
static at::Tensor gemm_rows(at::Tensor x, const at::Tensor& w, const c10::optional<at::Tensor>& bias, int64_t act,
                const c10::optional<at::Tensor>& residual, const c10::optional<at::Tensor>& out, bool fresh_weight, const c10::optional<at::Tensor>& norm_w, double eps,
                double offset, const at::Tensor* w_scale = nullptr) {
  TORCH_CHECK(x.is_cuda() && w.is_cuda() && x.dim() == 2 && w.dim() == 2 && x.size(1) == w.size(1));
  TORCH_CHECK(is_bf16(x) && is_bf16(w) && x.stride(1) == 1 && w.is_contiguous());
  const int M = x.size(0), K = x.size(1), N = w.size(0);
  TORCH_CHECK(K % 64 == 0 && x.stride(0) % 8 == 0, "gemm: K must be a multiple of 64");
  const bool glu = act != 0;
  const int n_out = glu ? N / 2 : N;
  TORCH_CHECK(n_out % 8 == 0 && (!glu || N % 2 == 0));
  c10::cuda::CUDAGuard guard(x.device());
  if (out.has_value())
    TORCH_CHECK(out->is_cuda() && is_bf16(*out) && out->dim() == 2 && out->size(0) == M && out->size(1) == n_out && out->is_contiguous());
  auto y = out.has_value() ? *out : at::empty({M, n_out}, x.options());
  if (residual.has_value())
    TORCH_CHECK(!glu && residual->is_contiguous() && residual->size(0) == M && residual->size(1) == n_out && is_bf16(*residual));
  const float* ws = w_scale != nullptr ? w_scale->data_ptr<float>() : nullptr;
  const int ws_n = w_scale != nullptr ? (int)w_scale->numel() : 0;
  if (ws == nullptr && skinny_pays(M, N, K, glu)) {
    run_skinny(x, w, bias, (int)act, residual, y, fresh_weight, norm_w, eps, offset);
    return y;
  }
  if (norm_w.has_value()) x = rmsnorm_rows(x.contiguous(), *norm_w, eps, offset, nullptr, nullptr);
  if (pair_pays(M, n_out, glu)) {
    gemm_pair_launch(x.data_ptr(), x.stride(0), w.data_ptr(), optr(bias), optr(residual), y.data_ptr(), M, N, K, (int)act, cur_stream(),
                     fresh_weight, nullptr, nullptr, 0, 1, 7.f, 1.702f, ws, ws_n);
    return y;
  }
  gemm_tcgen05_launch(x.data_ptr(), (int)x.stride(0), w.data_ptr(), optr(bias), optr(residual), y.data_ptr(), n_out, M, N, K,
                      (int)act, cur_stream(), nullptr, fresh_weight, ws, ws_n);
  return y;
}

at::Tensor gemm(const at::Tensor& x, const at::Tensor& w, const c10::optional<at::Tensor>& bias, int64_t act, const c10::optional<at::Tensor>& residual,
                const c10::optional<at::Tensor>& out, bool fresh_weight) {
  return gemm_rows(x, w, bias, act, residual, out, fresh_weight, c10::nullopt, 0., 0.);
}

static at::Tensor expand_bf16(const at::Tensor& w, const at::Tensor* scale);
at::Tensor dequant_bf16(const at::Tensor& w, const at::Tensor& scale);

// Whether 8-bit weights of 9 .. 512 tokens (64 with a gate product) are read as bytes (linear8_few) or expanded to bf16 in front of a tile GEMM.  Bytes cost their
// stream, once, and an epilogue that grows with the tokens of a block; the expansion costs a launch and two passes over bf16 weights, the tile GEMM behind it the
// same whatever the tokens of a tile.  us in a graph, bytes / expanded (fp8):
//   1024 x 1024: 16.3 / 13.5 at 128 tokens, 15.4 / 9.6 at 320      4096 x 1024: 16.7 / 12.0 at 128, 14.7 / 12.1 at 192, 19.7 / 14.3 at 512
//   2048 x 1024: 12.4 / 14.8 at 65                                 8192 x 1024: 19.9 / 16.4 at 256, 26.5 / 18.9 at 512
//   4096 x 512:  9.0 / 10.0 at 129, 10.6 / 11.7 at 320             8192 x 512:  9.3 / 12.5 at 129, 11.5 / 12.6 at 256, 20.9 / 14.5 at 320
//   2048 x 2048: 18.7 / 15.1 at 256, 21.8 / 15.5 at 512            8192 x 2048: 25.8 / 28.3 at 257, 33.3 / 28.9 at 512
//   512 x 2048:  14.8 / 18.6 at 257                                2048 x 3072: 16.9 / 18.6 at 129
//   gate products: 512 x 512 8.6 / 7.3 at 33, 2048 x 1024 12.7 / 14.3 at 48, 4096 x 1024 14.2 / 12.1 at 64
static bool linear8_bytes_pay(int64_t T, int64_t N, int64_t K, bool glu) {
  if (K < 512) return T <= 32;
  if (glu) return T <= 32 || K >= 2048 || (K >= 1024 ? T <= 48 || N >= 8192 : N >= 4096);
  if (T <= 64 || K >= 4096) return true;
  const int64_t b = (T + 127) / 128;
  const bool low = (T + b - 1) / b <= 96;        // tokens of a block
  if (K >= 2048) return b == 1 || (b == 2 && (low || N <= 1024)) || N <= 512 || (N >= 8192 && (b <= 3 || N * K >= (24LL << 20)));
  if (K >= 1024) return b <= 2 && ((N >= 8192 && (b == 1 || low)) || (N <= (b == 1 ? 2048 : 1024) && low));
  return N >= 4096 && N * T <= (2LL << 20);
}

// int8 / fp8 weights and 9 .. 512 tokens (64 with a gate product): the bytes are read once, by blocks of up to 128 tokens at the same time.  The weight is not rounded:
// the scale is applied to the fp32 sum.
static at::Tensor linear8_few(const at::Tensor& x, const at::Tensor& w, const c10::optional<at::Tensor>& bias, int64_t act, const at::Tensor& scale,
                              const c10::optional<at::Tensor>& residual, const c10::optional<at::Tensor>& norm_w, double eps, double offset) {
  const int64_t M = x.size(0), N = w.size(0), n_out = act != 0 ? N / 2 : N;
  TORCH_CHECK(x.size(1) == w.size(1) && w.is_cuda() && (act == 0 || N % 2 == 0) && (scale.numel() == 1 || scale.numel() == N));
  c10::cuda::CUDAGuard guard(x.device());
  auto y = at::empty({M, n_out}, x.options());
  if (residual.has_value())
    TORCH_CHECK(act == 0 && residual->is_contiguous() && residual->size(0) == M && residual->size(1) == n_out && is_bf16(*residual));
  run_skinny(x.contiguous(), w, bias, (int)act, residual, y, false, norm_w, eps, offset, &scale);
  return y;
}

// y = act(rmsnorm(x) w^T + bias) (+ residual) of rows x [.., K]: the choice between the kernels, made here because in Python it cost more than a launch.
// -> result and what ran (the bits below), or none where no kernel takes the call (the caller's library path) or the norm's weight is of another type (LINEAR_NORM
// alone: the caller normalises first).  bf16 x; w bf16, or int8 / fp8 with a scale per channel or one.
enum { LINEAR_QGEMV = 1, LINEAR_GEMV = 2, LINEAR_DEQUANT = 4, LINEAR_GEMM = 8, LINEAR_NORM = 16 };
std::tuple<c10::optional<at::Tensor>, int64_t> linear(const at::Tensor& x, const at::Tensor& w, const c10::optional<at::Tensor>& bias_in,
                                                      const c10::optional<at::Tensor>& norm_in, double eps, double offset, int64_t act,
                                                      const c10::optional<at::Tensor>& scale, const c10::optional<at::Tensor>& residual,
                                                      const c10::optional<at::Tensor>& out, bool tensor_cores) {
  const auto none = std::make_tuple(c10::optional<at::Tensor>(), (int64_t)0);
  const bool wq = w.scalar_type() == at::kChar || w.scalar_type() == at::kFloat8_e4m3fn;
  const bool plain = is_bf16(w) && !scale.has_value();
  if (!is_bf16(x) || x.dim() < 1 || x.size(-1) == 0 || w.dim() != 2 || !w.is_contiguous() || !(plain || (wq && scale.has_value() && scale->dim() == 1))) return none;
  const int64_t K = x.size(-1), T = x.numel() / K, N = w.size(0), n_out = act != 0 ? N / 2 : N;
  const bool few = T <= GEMV_MAX_T, few8 = wq && !out.has_value() && skinny_gemm8_supported((int)std::min<int64_t>(T, SKINNY8_MAX_T + 1), (int)K, act != 0);
  int64_t ran = 0;
  if (few && wq && K % 16 == 0) ran = LINEAR_QGEMV;
  else if (few && plain && K % 64 == 0 && (K % 256 == 0 || gemv2_supported((int)T, (int)K, 0))) ran = LINEAR_GEMV;
  else if (!few && K % 64 == 0 && n_out % 8 == 0 && tensor_cores) ran = LINEAR_GEMM | (wq && !(few8 && linear8_bytes_pay(T, N, K, act != 0)) ? LINEAR_DEQUANT : 0);
  else return none;
  c10::optional<at::Tensor> norm_w;
  if (norm_in.has_value()) {
    if (!is_bf16(*norm_in)) return std::make_tuple(c10::optional<at::Tensor>(), (int64_t)LINEAR_NORM);
    norm_w = norm_in->contiguous();
    if (ran & LINEAR_GEMM) ran |= LINEAR_NORM;
  }
  c10::optional<at::Tensor> bias;
  if (bias_in.has_value()) {
    TORCH_CHECK(bias_in->is_cuda() && is_bf16(*bias_in) && bias_in->numel() == N, "linear: a bias of ", N, " bf16 values on the GPU expected");
    bias = bias_in->contiguous();
  }
  if (scale.has_value()) TORCH_CHECK(scale->is_cuda() && (scale->numel() == 1 || scale->numel() == N), "linear: scales on the GPU, one or ", N, " expected");
  const auto x2 = x.reshape({T, K});
  c10::optional<at::Tensor> r2, scale_f;
  if (residual.has_value() && act == 0) r2 = wq && few ? residual->reshape({T, -1}).contiguous() : residual->reshape({T, -1});
  if (scale.has_value()) {
    scale_f = scale->to(at::kFloat).contiguous();
    if (reinterpret_cast<uintptr_t>(scale_f->data_ptr()) % 16 != 0) scale_f = scale_f->clone();      // (a slice; the tile kernels load four at a time)
  }
  at::Tensor y;
  if (ran & (LINEAR_QGEMV | LINEAR_GEMV)) {
    y = gemv(x2, w, bias, norm_w, eps, offset, act, scale_f, r2);
  } else {
    c10::optional<at::Tensor> o2;
    if (out.has_value()) o2 = out->view({T, -1});
    // weight-only 8-bit layers: few tokens read the bytes (linear8_few) where that pays; else one expansion pass to bf16 (stays in L2), then the bf16 GEMM, which waits
    // for it.  Up to 512 tokens (64 with a gate product) the weight is not rounded either way: its scale goes to the fp32 sum
    if (few8 && linear8_bytes_pay(T, N, K, act != 0)) y = linear8_few(x2, w, bias, act, *scale_f, r2, norm_w, eps, offset);
    else if (few8) y = gemm_rows(x2.contiguous(), expand_bf16(w, nullptr), bias, act, r2, o2, true, norm_w, eps, offset, &*scale_f);
    else y = gemm_rows(x2.contiguous(), wq ? dequant_bf16(w, *scale_f) : w, bias, act, r2, o2, wq, norm_w, eps, offset);
  }
  if ((ran & LINEAR_GEMM) && out.has_value()) {
    y = *out;
  } else {
    auto shape = x.sizes().vec();
    shape.back() = y.size(1);
    y = y.view(shape);
  }
  if (residual.has_value() && !r2.has_value()) y = y + *residual;
  return std::make_tuple(c10::optional<at::Tensor>(y), ran);
}

// Row-parallel GEMV -> one-shot all-reduce over NVLink peer buffers -> +bias +residual.  ONE kernel.
at::Tensor gemv_allreduce(const at::Tensor& x, const at::Tensor& w, const c10::optional<at::Tensor>& bias,
                          const c10::optional<at::Tensor>& residual, const std::vector<int64_t>& recv_ptrs,
                          const at::Tensor& step, int64_t rank, int64_t parity, int64_t call, int64_t n_max,
                          const c10::optional<at::Tensor>& scale) {
  int wt = 0;
  if (scale.has_value()) {   // weight-only int8 / fp8 row-parallel layer
    TORCH_CHECK(x.is_cuda() && w.is_cuda() && x.dim() == 2 && w.dim() == 2 && x.size(1) == w.size(1) && is_bf16(x) && w.is_contiguous());
    TORCH_CHECK(x.size(0) >= 1 && x.size(0) <= GEMV_MAX_T && x.stride(1) == 1 && x.stride(0) % 8 == 0);
    wt = w.scalar_type() == at::kChar ? 1 : 2;
    TORCH_CHECK(wt == 1 || w.scalar_type() == at::kFloat8_e4m3fn, "gemv_allreduce: int8 or float8_e4m3fn weights");
    TORCH_CHECK(scale->scalar_type() == at::kFloat && scale->is_contiguous() && (scale->numel() == 1 || scale->numel() == w.size(0)));
  } else {
    check_gemv_inputs(x, w);
  }
  const int world = recv_ptrs.size();
  TORCH_CHECK(world >= 2 && world <= SYMM_MAX_RANKS);
  TORCH_CHECK(step.is_cuda() && step.scalar_type() == at::kInt && step.numel() >= 1, "gemv_allreduce: step counter must be a CUDA int32 tensor");
  TORCH_CHECK(gemv2_supported(x.size(0), x.size(1), wt), "gemv_allreduce: activations too wide for shared memory");
  const int N = w.size(0);
  TORCH_CHECK(N <= n_max && (N + 15) / 16 <= SYMM_MAX_TILES, "gemv_allreduce: output too wide for the workspace");
  c10::cuda::CUDAGuard guard(x.device());
  bool x_in_smem;
  at::Tensor xn = prenorm_if_needed(x, c10::nullopt, 0, 0, x_in_smem);
  auto y = at::empty({x.size(0), N}, x.options());
  if (residual.has_value())
    TORCH_CHECK(residual->is_contiguous() && residual->size(0) == x.size(0) && residual->size(1) == N && is_bf16(*residual));
  GemvParams p{};
  fill_params(p, xn, w, bias, c10::nullopt, 0, 0, 0, residual, scale, y, x_in_smem);
  for (int i = 0; i < world; ++i) p.symm.recv[i] = reinterpret_cast<float*>(recv_ptrs[i]);
  p.symm.step = reinterpret_cast<const uint32_t*>(step.data_ptr<int>());
  p.symm.rank = rank;
  p.symm.world = world;
  p.symm.parity = parity;
  p.symm.call = call;
  p.symm.n_max = n_max;
  run_gemv(p, 1);
  return y;
}

// Expert ids come as int32, or as int64 from torch.topk and renormalised softmax routers: the kernels read the low words
static bool is_ids(const at::Tensor& t) { return t.scalar_type() == at::kInt || t.scalar_type() == at::kLong; }
static int id_step(const at::Tensor& t) { return t.scalar_type() == at::kLong ? 2 : 1; }
static const int* id_ptr(const at::Tensor& t) { return reinterpret_cast<const int*>(t.data_ptr()); }

// Routed experts of a decode step: x [T,H], w_gate_up [E,2I,H], w_down [E,H,I], topk_w/topk_i [T,k] -> [T,H] (local experts only;
// the caller all-reduces across EP/TP ranks).
at::Tensor moe_decode(const at::Tensor& x, const at::Tensor& w_gate_up, const at::Tensor& w_down, const at::Tensor& topk_w,
                      const at::Tensor& topk_i, int64_t expert_offset, int64_t act, double limit, double alpha) {
  TORCH_CHECK(act == 1 || act == 4, "moe_decode: SiLU or clamped gate product");
  TORCH_CHECK(x.is_cuda() && x.dim() == 2 && x.is_contiguous() && is_bf16(x) && is_bf16(w_gate_up) && is_bf16(w_down));
  TORCH_CHECK(w_gate_up.dim() == 3 && w_down.dim() == 3 && w_gate_up.is_contiguous() && w_down.is_contiguous());
  const int T = x.size(0), H = x.size(1), E = w_gate_up.size(0), I = w_gate_up.size(1) / 2, k = topk_i.size(1);
  TORCH_CHECK(w_gate_up.size(2) == H && w_down.size(0) == E && w_down.size(1) == H && w_down.size(2) == I);
  TORCH_CHECK(topk_w.scalar_type() == at::kFloat && is_ids(topk_i) && topk_w.is_contiguous() &&
              topk_i.is_contiguous() && topk_w.numel() == (int64_t)T * k && topk_i.size(0) == T);
  c10::cuda::CUDAGuard guard(x.device());
  auto u = at::empty({(int64_t)T * k, I}, x.options());
  auto y = at::empty({T, H}, x.options().dtype(at::kFloat));     // cleared by the first kernel
  moe_decode_launch(x.data_ptr(), w_gate_up.data_ptr(), w_down.data_ptr(), topk_w.data_ptr<float>(), id_ptr(topk_i), id_step(topk_i),
                    u.data_ptr(), y.data_ptr<float>(), T, k, H, I, E, (int)expert_offset, (int)act, (float)limit, (float)alpha, cur_stream());
  return y.to(x.scalar_type());
}

constexpr int64_t MOE_SMALL_ENTRIES = 2560;       // (token, slot) pairs that moe_small_gather_kernel counts by comparing each with all
// Routed experts of a step of up to 128 tokens, or of a few hundred: every expert's weights are streamed once for up to 128 of its tokens (bf16; act and biases as
// moe_grouped)
at::Tensor moe_small(const at::Tensor& x, const at::Tensor& w_gate_up, const at::Tensor& w_down, const at::Tensor& topk_w, const at::Tensor& topk_i,
                     int64_t expert_offset, int64_t act, bool scale_input, const c10::optional<at::Tensor>& gate_up_bias,
                     const c10::optional<at::Tensor>& down_bias, double limit, double alpha) {
  TORCH_CHECK(x.is_cuda() && x.dim() == 2 && x.is_contiguous() && is_bf16(x) && is_bf16(w_gate_up) && is_bf16(w_down));
  TORCH_CHECK(w_gate_up.dim() == 3 && w_down.dim() == 3 && w_gate_up.is_contiguous() && w_down.is_contiguous() && act >= 1 && act <= 4);
  const int N = x.size(0), H = x.size(1), E = w_gate_up.size(0), I = w_gate_up.size(1) / 2, k = topk_i.size(1);
  TORCH_CHECK(w_gate_up.size(1) == 2 * I && w_gate_up.size(2) == H && w_down.size(0) == E && w_down.size(1) == H && w_down.size(2) == I);
  const int most = std::min(N, SKINNY_MAX_T);                      // rows of a segment
  TORCH_CHECK(N >= 1 && (N <= SKINNY_MAX_T || (int64_t)N * k <= MOE_SMALL_ENTRIES) && H % 64 == 0 && I % 64 == 0 && E <= 512,
              "moe_small: 1 .. 128 tokens (or 2560 entries), sizes in multiples of 64, <= 512 experts");
  TORCH_CHECK(topk_w.scalar_type() == at::kFloat && is_ids(topk_i) && topk_w.is_contiguous() && topk_i.is_contiguous() &&
              topk_w.numel() == (int64_t)N * k && topk_i.size(0) == N);
  if (gate_up_bias) TORCH_CHECK(is_bf16(*gate_up_bias) && gate_up_bias->is_contiguous() && gate_up_bias->numel() == (int64_t)E * 2 * I);
  if (down_bias) TORCH_CHECK(is_bf16(*down_bias) && down_bias->is_contiguous() && down_bias->numel() == (int64_t)E * H);
  c10::cuda::CUDAGuard guard(x.device());
  const int64_t R = (int64_t)N * k, nt = skinny_gemm_tickets();
  auto iopt = x.options().dtype(at::kInt), fopt = x.options().dtype(at::kFloat);
  auto xp = at::empty({R, H}, x.options()), h = at::empty({R, I}, x.options()), out = at::empty({N, H}, x.options());
  auto y = at::empty({R, H}, fopt);
  // an expert has at most N entries when every token names it once, but nothing forbids a token to name it again (k times N): its rows are cut into
  // segments of what the GEMM's token tile holds
  const int seg_rows = skinny_gemm_rows(most);
  const int64_t segs = std::min<int64_t>(E, R) + R / seg_rows;
  auto meta = at::empty({R + 1 + 3 * segs + 2 * nt}, iopt);       // pos | n_active | active | seg_start | seg_count | tickets of both GEMMs
  auto ws = at::empty({std::max(skinny_gemm_ws_floats(most, true), skinny_gemm_ws_floats(most, false))}, fopt);
  int* pos = meta.data_ptr<int>();
  int *n_active = pos + R, *active = n_active + 1, *seg_start = active + segs, *seg_count = seg_start + segs;
  unsigned* tickets = reinterpret_cast<unsigned*>(seg_count + segs);
  auto st = cur_stream();
  moe_small_gather_launch(x.data_ptr(), topk_w.data_ptr<float>(), id_ptr(topk_i), id_step(topk_i), (int)R, k, H, (int)expert_offset, E, seg_rows,
                          scale_input ? 1 : 0, xp.data_ptr(), pos, n_active, active, seg_start, seg_count, tickets, (int)(2 * nt), st);
  SkinnyGemm a{};
  a.x = xp.data_ptr(); a.x_rows = R; a.ldx = H; a.w = w_gate_up.data_ptr(); a.bias = optr(gate_up_bias); a.y = h.data_ptr();
  a.experts = E; a.tokens = most; a.n_out = I; a.K = H; a.act = (int)act; a.limit = (float)limit; a.alpha = (float)alpha;
  a.n_active = n_active; a.active = active; a.seg_start = seg_start; a.seg_count = seg_count;
  a.ws = ws.data_ptr<float>(); a.tickets = tickets;
  skinny_gemm_launch(a, st);
  a.x = h.data_ptr(); a.ldx = I; a.w = w_down.data_ptr(); a.bias = optr(down_bias); a.y = y.data_ptr(); a.y_f32 = 1;
  a.n_out = H; a.K = I; a.act = 0; a.tickets = tickets + nt;
  skinny_gemm_launch(a, st);
  moe_small_combine_launch(y.data_ptr<float>(), topk_w.data_ptr<float>(), pos, out.data_ptr(), N, H, k, scale_input ? 1 : 0, st);
  return out;
}

// int8 / fp8 weight [N, K] x scale -> bf16.  A result per call: two streams may expand weights at the same time, and the stream order of the caching
// allocator hands the same memory to the next layer
static at::Tensor expand_bf16(const at::Tensor& w, const at::Tensor* scale) {
  TORCH_CHECK(w.is_cuda() && w.dim() == 2 && w.is_contiguous());
  const bool i8 = w.scalar_type() == at::kChar;
  TORCH_CHECK(i8 || w.scalar_type() == at::kFloat8_e4m3fn, "dequant_bf16: int8 or float8_e4m3fn weights");
  c10::cuda::CUDAGuard guard(w.device());
  auto out = at::empty({w.size(0), w.size(1)}, w.options().dtype(at::kBFloat16));
  dequant_bf16_launch(w.data_ptr(), i8 ? 1 : 2, scale != nullptr ? scale->data_ptr<float>() : nullptr, scale != nullptr ? (int)scale->numel() : 0, out.data_ptr(),
                      (int)w.size(0), (int)w.size(1), cur_stream());
  return out;
}
at::Tensor dequant_bf16(const at::Tensor& w, const at::Tensor& scale) {
  TORCH_CHECK(scale.is_cuda() && scale.scalar_type() == at::kFloat && scale.is_contiguous() && (scale.numel() == 1 || scale.numel() == w.size(0)));
  return expand_bf16(w, &scale);
}

// Routed experts of a prefill-sized batch (any N): permutation on the device + two grouped tcgen05 GEMMs + weighted combine.
// act: 1 silu*up, 2 gelu_tanh*up, 3 gelu*up.  gate_up_bias [E, 2I] / down_bias [E, H] optional (bf16).
at::Tensor moe_grouped(const at::Tensor& x, const at::Tensor& w_gate_up, const at::Tensor& w_down, const at::Tensor& topk_w,
                       const at::Tensor& topk_i, int64_t expert_offset, int64_t act, bool scale_input,
                       const c10::optional<at::Tensor>& gate_up_bias, const c10::optional<at::Tensor>& down_bias,
                       const c10::optional<at::Tensor>& gate_up_scale, const c10::optional<at::Tensor>& down_scale, double limit, double alpha) {
  // W8A8 experts: fp8-e4m3 weights with per-(expert, channel) scales; the permuted activations and the intermediate are quantised
  // per row (quant.cu) and both grouped GEMMs run on the kind::f8f6f4 tensor-core path
  const bool fp8 = gate_up_scale.has_value();
  TORCH_CHECK(x.is_cuda() && x.dim() == 2 && x.is_contiguous() && is_bf16(x));
  if (fp8) {
    TORCH_CHECK(w_gate_up.scalar_type() == at::kFloat8_e4m3fn && w_down.scalar_type() == at::kFloat8_e4m3fn && down_scale.has_value());
    TORCH_CHECK(gate_up_scale->scalar_type() == at::kFloat && gate_up_scale->is_contiguous() && down_scale->scalar_type() == at::kFloat &&
                down_scale->is_contiguous());
  } else {
    TORCH_CHECK(is_bf16(w_gate_up) && is_bf16(w_down));
  }
  TORCH_CHECK(w_gate_up.dim() == 3 && w_down.dim() == 3 && w_gate_up.is_contiguous() && w_down.is_contiguous());
  const int N = x.size(0), H = x.size(1), E = w_gate_up.size(0), I = w_gate_up.size(1) / 2, k = topk_i.size(1);
  TORCH_CHECK(w_gate_up.size(2) == H && w_down.size(0) == E && w_down.size(1) == H && w_down.size(2) == I);
  TORCH_CHECK(H % 64 == 0 && I % 64 == 0, "moe_grouped: hidden and intermediate sizes must be multiples of 64");
  if (fp8) {
    TORCH_CHECK(H % 128 == 0 && I % 128 == 0 && H <= 16384 && I <= 16384, "moe_grouped (fp8): sizes must be multiples of 128, <= 16384");
    TORCH_CHECK(gate_up_scale->numel() == (int64_t)E * 2 * I && down_scale->numel() == (int64_t)E * H);
  }
  TORCH_CHECK(topk_w.scalar_type() == at::kFloat && is_ids(topk_i) && (!fp8 || topk_i.scalar_type() == at::kInt) && topk_w.is_contiguous() &&
              topk_i.is_contiguous() && topk_w.numel() == (int64_t)N * k && topk_i.size(0) == N);
  if (gate_up_bias) TORCH_CHECK(is_bf16(*gate_up_bias) && gate_up_bias->is_contiguous() && gate_up_bias->numel() == (int64_t)E * 2 * I);
  if (down_bias) TORCH_CHECK(is_bf16(*down_bias) && down_bias->is_contiguous() && down_bias->numel() == (int64_t)E * H);
  c10::cuda::CUDAGuard guard(x.device());
  auto iopt = x.options().dtype(at::kInt);
  if (!fp8) {
    // the permuted rows lie one after the other (an expert's last tile runs on into the next one's rows and stores its own only), so the three
    // buffers hold one row per entry; the number of tiles is a static bound: graph-stable shapes
    const int64_t R = (int64_t)N * k, tiles = (R + std::min<int64_t>(E, R) * 255) / 256;
    auto out = at::empty({N, H}, x.options());
    if (R == 0) return out.zero_();
    auto st = cur_stream();
    auto pos = at::empty({R}, iopt), tile_expert = at::empty({tiles}, iopt), tile_row = at::empty({tiles}, iopt);
    auto xp = at::empty({R, H}, x.options()), h = at::empty({R, I}, x.options()), y = at::empty({R, H}, x.options());
    moe_plan256_launch(id_ptr(topk_i), id_step(topk_i), (int)R, (int)expert_offset, E, (int)tiles, pos.data_ptr<int>(), tile_expert.data_ptr<int>(),
                       tile_row.data_ptr<int>(), st);
    moe_scatter_launch(x.data_ptr(), topk_w.data_ptr<float>(), pos.data_ptr<int>(), xp.data_ptr(), N, H, k, scale_input ? 1 : 0, st);
    gemm_pair_launch(xp.data_ptr(), H, w_gate_up.data_ptr(), optr(gate_up_bias), nullptr, h.data_ptr(), (int)R, 2 * I, H, (int)act, st,
                     false, tile_expert.data_ptr<int>(), tile_row.data_ptr<int>(), (int)tiles, E, (float)limit, (float)alpha);
    gemm_pair_launch(h.data_ptr(), I, w_down.data_ptr(), optr(down_bias), nullptr, y.data_ptr(), (int)R, H, I, 0, st, false,
                     tile_expert.data_ptr<int>(), tile_row.data_ptr<int>(), (int)tiles, E);
    moe_combine_launch(y.data_ptr(), topk_w.data_ptr<float>(), pos.data_ptr<int>(), out.data_ptr(), N, H, k, scale_input ? 1 : 0, st);
    return out;
  }
  const int64_t R = (((int64_t)N * k + (int64_t)E * 127) + 127) / 128 * 128;
  auto pos = at::empty({(int64_t)N * k}, iopt);
  auto row_entry = at::empty({R}, iopt);
  auto tile_expert = at::empty({R / 128}, iopt);
  auto xp = at::empty({R, H}, x.options());
  auto h = at::empty({R, I}, x.options());
  auto y = at::empty({R, H}, x.options());
  auto out = at::empty({N, H}, x.options());
  auto st = cur_stream();
  moe_plan_launch(topk_i.data_ptr<int>(), N * k, (int)expert_offset, E, (int)R, pos.data_ptr<int>(), row_entry.data_ptr<int>(),
                  tile_expert.data_ptr<int>(), st);
  moe_gather_launch(x.data_ptr(), topk_w.data_ptr<float>(), row_entry.data_ptr<int>(), tile_expert.data_ptr<int>(), xp.data_ptr(), (int)R,
                    H, k, scale_input ? 1 : 0, st);
  const float inf = std::numeric_limits<float>::infinity();
  auto bopt = x.options().dtype(at::kByte);
  auto xq = at::empty({R, H}, bopt), hq = at::empty({R, I}, bopt);
  auto xs = at::empty({R}, x.options().dtype(at::kFloat)), hs = at::empty({R}, x.options().dtype(at::kFloat));
  rmsnorm_quant_launch(xp.data_ptr(), nullptr, xq.data_ptr(), xs.data_ptr<float>(), (int)R, H, 0.f, 0.f, inf, st);
  gemm_grouped_launch(xq.data_ptr(), w_gate_up.data_ptr(), gate_up_bias ? gate_up_bias->data_ptr() : nullptr, h.data_ptr(), (int)R, 2 * I,
                      H, E, (int)act, tile_expert.data_ptr<int>(), xs.data_ptr<float>(), gate_up_scale->data_ptr<float>(), st, (float)limit, (float)alpha);
  rmsnorm_quant_launch(h.data_ptr(), nullptr, hq.data_ptr(), hs.data_ptr<float>(), (int)R, I, 0.f, 0.f, inf, st);
  gemm_grouped_launch(hq.data_ptr(), w_down.data_ptr(), down_bias ? down_bias->data_ptr() : nullptr, y.data_ptr(), (int)R, H, I, E, 0,
                      tile_expert.data_ptr<int>(), hs.data_ptr<float>(), down_scale->data_ptr<float>(), st);
  moe_combine_launch(y.data_ptr(), topk_w.data_ptr<float>(), pos.data_ptr<int>(), out.data_ptr(), N, H, k, scale_input ? 1 : 0, st);
  return out;
}

// ---- symmetric (peer-mapped) workspace ---------------------------------------------------------------------
std::tuple<int64_t, pybind11::bytes> symm_alloc(int64_t nbytes) {
  void* p = nullptr;
  NXDI_CUDA_OK(cudaMalloc(&p, nbytes));
  NXDI_CUDA_OK(cudaMemset(p, 0, nbytes));
  cudaIpcMemHandle_t h;
  NXDI_CUDA_OK(cudaIpcGetMemHandle(&h, p));
  NXDI_CUDA_OK(cudaDeviceSynchronize());
  return {reinterpret_cast<int64_t>(p), pybind11::bytes(reinterpret_cast<const char*>(&h), sizeof(h))};
}
int64_t symm_open(const std::string& handle) {
  TORCH_CHECK(handle.size() == sizeof(cudaIpcMemHandle_t), "bad IPC handle size");
  cudaIpcMemHandle_t h;
  memcpy(&h, handle.data(), sizeof(h));
  void* p = nullptr;
  NXDI_CUDA_OK(cudaIpcOpenMemHandle(&p, h, cudaIpcMemLazyEnablePeerAccess));
  return reinterpret_cast<int64_t>(p);
}
void symm_close(int64_t ptr) { cudaIpcCloseMemHandle(reinterpret_cast<void*>(ptr)); }
void symm_free(int64_t ptr) { cudaFree(reinterpret_cast<void*>(ptr)); }
at::Tensor symm_as_tensor(int64_t ptr, int64_t nbytes, int64_t device) {
  auto opts = at::TensorOptions().dtype(at::kByte).device(at::kCUDA, device);
  return at::from_blob(reinterpret_cast<void*>(ptr), {nbytes}, opts);
}

// ---- rope / cache appends -------------------------------------------------------------------------------------
// cos / sin [.., half] of positions [..] (int32 or int64), clamped to the tables [length, half]
std::tuple<at::Tensor, at::Tensor> rope_rows(const at::Tensor& positions, const at::Tensor& cos_table, const at::Tensor& sin_table) {
  TORCH_CHECK(is_ids(positions) && positions.is_cuda() && cos_table.is_cuda() && cos_table.dim() == 2 && cos_table.scalar_type() == at::kFloat && cos_table.is_contiguous() &&
              sin_table.sizes() == cos_table.sizes() && sin_table.scalar_type() == at::kFloat && sin_table.is_contiguous() && cos_table.size(0) > 0 &&
              cos_table.size(0) <= std::numeric_limits<int>::max() && positions.numel() <= std::numeric_limits<int>::max());
  c10::cuda::CUDAGuard guard(positions.device());
  const auto pos = positions.contiguous();
  auto shape = positions.sizes().vec();
  shape.push_back(cos_table.size(1));
  auto c = at::empty(shape, cos_table.options()), s = at::empty(shape, cos_table.options());
  if (c.numel() > 0)
    rope_rows_launch(pos.data_ptr(), pos.scalar_type() == at::kLong, cos_table.data_ptr<float>(), sin_table.data_ptr<float>(), c.data_ptr<float>(), s.data_ptr<float>(),
                     (int)pos.numel(), (int)cos_table.size(1), (int)cos_table.size(0), cur_stream());
  return {c, s};
}
// ids (int32 or int64) with those outside 0 .. n_lines - 1 replaced by n_lines
at::Tensor cache_lines(const at::Tensor& ids, int64_t n_lines) {
  TORCH_CHECK(is_ids(ids) && ids.is_cuda() && n_lines >= 0 && n_lines <= std::numeric_limits<int>::max());
  c10::cuda::CUDAGuard guard(ids.device());
  const auto in = ids.contiguous();
  auto lines = at::empty(in.sizes(), in.options());
  if (in.numel() > 0) cache_lines_launch(in.data_ptr(), in.scalar_type() == at::kLong, lines.data_ptr(), in.numel(), n_lines, cur_stream());
  return lines;
}

at::Tensor rope_kv_append(const at::Tensor& qkv, const at::Tensor& cos, const at::Tensor& sin, at::Tensor& k_cache,
                          at::Tensor& v_cache, const at::Tensor& lines, const at::Tensor& positions, int64_t nq, int64_t nkv,
                          int64_t D, const c10::optional<at::Tensor>& q_norm, const c10::optional<at::Tensor>& k_norm,
                          double eps) {
  TORCH_CHECK(qkv.is_cuda() && qkv.dim() == 3 && qkv.is_contiguous() && is_bf16(qkv) && is_bf16(k_cache));
  const int B = qkv.size(0), T = qkv.size(1);
  TORCH_CHECK(qkv.size(2) == (nq + 2 * nkv) * D);
  TORCH_CHECK(cos.scalar_type() == at::kFloat && cos.is_contiguous() && sin.is_contiguous() &&
              cos.numel() == (int64_t)B * T * D / 2 && sin.numel() == cos.numel());
  TORCH_CHECK(k_cache.dim() == 4 && k_cache.size(1) == nkv && k_cache.size(3) == D && k_cache.is_contiguous() &&
              v_cache.is_contiguous());
  TORCH_CHECK(lines.scalar_type() == at::kInt && positions.scalar_type() == at::kInt && positions.is_contiguous() &&
              lines.numel() == B && positions.numel() == B * T);
  c10::cuda::CUDAGuard guard(qkv.device());
  auto q = at::empty({B, T, nq, D}, qkv.options());
  rope_kv_append_launch(qkv.data_ptr(), cos.data_ptr<float>(), sin.data_ptr<float>(), q.data_ptr(), k_cache.data_ptr(),
                        v_cache.data_ptr(), lines.data_ptr<int>(), positions.data_ptr<int>(), optr(q_norm), optr(k_norm),
                        (float)eps, B, T, (int)nq, (int)nkv, (int)D, (int)k_cache.size(0), (int)k_cache.size(2), cur_stream());
  return q;
}

// prefill flavour: the same single pass also returns the rotated k and the v of the new tokens as contiguous [B, T, nkv, D]
std::tuple<at::Tensor, at::Tensor, at::Tensor> rope_kv_split_append(const at::Tensor& qkv, const at::Tensor& cos, const at::Tensor& sin,
                                                                   at::Tensor& k_cache, at::Tensor& v_cache, const at::Tensor& lines,
                                                                   const at::Tensor& positions, int64_t nq, int64_t nkv, int64_t D,
                                                                   const c10::optional<at::Tensor>& q_norm,
                                                                   const c10::optional<at::Tensor>& k_norm, double eps) {
  TORCH_CHECK(qkv.is_cuda() && qkv.dim() == 3 && qkv.is_contiguous() && is_bf16(qkv) && is_bf16(k_cache));
  const int B = qkv.size(0), T = qkv.size(1);
  TORCH_CHECK(qkv.size(2) == (nq + 2 * nkv) * D);
  TORCH_CHECK(cos.scalar_type() == at::kFloat && cos.is_contiguous() && sin.is_contiguous() &&
              cos.numel() == (int64_t)B * T * D / 2 && sin.numel() == cos.numel());
  TORCH_CHECK(k_cache.dim() == 4 && k_cache.size(1) == nkv && k_cache.size(3) == D && k_cache.is_contiguous() &&
              v_cache.is_contiguous());
  TORCH_CHECK(lines.scalar_type() == at::kInt && positions.scalar_type() == at::kInt && positions.is_contiguous() &&
              lines.numel() == B && positions.numel() == B * T);
  c10::cuda::CUDAGuard guard(qkv.device());
  auto q = at::empty({B, T, nq, D}, qkv.options());
  auto k = at::empty({B, T, nkv, D}, qkv.options());
  auto v = at::empty({B, T, nkv, D}, qkv.options());
  rope_kv_append_launch(qkv.data_ptr(), cos.data_ptr<float>(), sin.data_ptr<float>(), q.data_ptr(), k_cache.data_ptr(),
                        v_cache.data_ptr(), lines.data_ptr<int>(), positions.data_ptr<int>(), optr(q_norm), optr(k_norm),
                        (float)eps, B, T, (int)nq, (int)nkv, (int)D, (int)k_cache.size(0), (int)k_cache.size(2), cur_stream(),
                        k.data_ptr(), v.data_ptr());
  return {q, k, v};
}

void kv_append(at::Tensor& k_cache, at::Tensor& v_cache, const at::Tensor& k_new, const at::Tensor& v_new,
               const at::Tensor& lines, const at::Tensor& positions) {
  TORCH_CHECK(k_new.is_cuda() && k_new.dim() == 4 && k_new.is_contiguous() && v_new.is_contiguous());
  TORCH_CHECK(k_cache.is_contiguous() && v_cache.is_contiguous() && k_cache.scalar_type() == k_new.scalar_type());
  const int B = k_new.size(0), T = k_new.size(1), H = k_new.size(2), D = k_new.size(3);
  TORCH_CHECK((D * k_new.element_size()) % 16 == 0 && v_new.size(3) == D && k_cache.size(1) == H && k_cache.size(3) == D);
  TORCH_CHECK(lines.scalar_type() == at::kInt && positions.scalar_type() == at::kInt && positions.is_contiguous());
  c10::cuda::CUDAGuard guard(k_new.device());
  kv_append_launch(k_new.data_ptr(), v_new.data_ptr(), k_cache.data_ptr(), v_cache.data_ptr(), lines.data_ptr<int>(),
                   positions.data_ptr<int>(), B, T, H, D * (int)k_new.element_size(), (int)k_cache.size(0),
                   (int)k_cache.size(2), cur_stream());
}

void paged_kv_append(at::Tensor& k_cache, at::Tensor& v_cache, const at::Tensor& k_new, const at::Tensor& v_new,
                     const at::Tensor& slots) {
  TORCH_CHECK(k_new.is_cuda() && k_new.is_contiguous() && v_new.is_contiguous() && k_cache.is_contiguous() &&
              v_cache.is_contiguous() && k_cache.dim() == 4);
  const int H = k_cache.size(2), D = k_cache.size(3);
  const int ntok = k_new.numel() / (H * D);
  TORCH_CHECK(slots.numel() == ntok && slots.scalar_type() == at::kInt && slots.is_contiguous());
  c10::cuda::CUDAGuard guard(k_new.device());
  paged_kv_append_launch(k_new.data_ptr(), v_new.data_ptr(), k_cache.data_ptr(), v_cache.data_ptr(), slots.data_ptr<int>(),
                         ntok, H * D * (int)k_new.element_size(), (int)(k_cache.size(0) * k_cache.size(1)), cur_stream());
}

// ---- sampling ---------------------------------------------------------------------------------------------------
at::Tensor argmax(const at::Tensor& logits, const std::vector<int64_t>& slot_ptrs, const c10::optional<at::Tensor>& step,
                  int64_t rank, int64_t parity, int64_t call, int64_t rows_max) {
  TORCH_CHECK(logits.is_cuda() && logits.dim() == 2 && logits.stride(1) == 1);
  TORCH_CHECK(logits.scalar_type() == at::kFloat || is_bf16(logits), "argmax: fp32 or bf16 logits");
  const int B = logits.size(0), V = logits.size(1);
  c10::cuda::CUDAGuard guard(logits.device());
  auto out = at::empty({B}, logits.options().dtype(at::kLong));
  const int nsplit = std::max(1, std::min(64, V / 2048));
  const auto ws = workspace(cur_stream(), (int64_t)B * nsplit, (int64_t)B * nsplit, B);
  ArgmaxSymm sy{};
  const int world = slot_ptrs.size();
  if (world > 1) {
    TORCH_CHECK(world <= SYMM_MAX_RANKS && step.has_value() && step->is_cuda() && step->scalar_type() == at::kInt && B <= rows_max,
                "argmax exchange: bad symmetric arguments");
    for (int i = 0; i < world; ++i) sy.slots[i] = reinterpret_cast<float*>(slot_ptrs[i]);
    sy.step = reinterpret_cast<const uint32_t*>(step->data_ptr<int>());
    sy.rank = rank; sy.world = world; sy.parity = parity; sy.call = call; sy.rows_max = rows_max;
  }
  argmax_launch(logits.data_ptr(), is_bf16(logits) ? 1 : 0, out.data_ptr<int64_t>(), ws.f, ws.i,
                ws.tickets, B, V, (int)logits.stride(0), nsplit,
                world > 1 ? &sy : nullptr, cur_stream());
  return out;
}

at::Tensor topk_sample(const at::Tensor& logits_in, const at::Tensor& top_k_in, const at::Tensor& top_p_in,
                       const at::Tensor& temperature_in, const c10::optional<at::Tensor>& rand_in, int64_t global_topk) {
  // (columns of one parameter matrix arrive strided)
  const auto logits = logits_in.contiguous(), top_k = top_k_in.to(at::kInt).contiguous(), top_p = top_p_in.to(at::kFloat).contiguous(),
             temperature = temperature_in.to(at::kFloat).contiguous();
  const auto rand = rand_in.has_value() ? rand_in->to(at::kFloat).contiguous() : at::full({logits.size(0)}, 0.5, logits.options().dtype(at::kFloat));
  TORCH_CHECK(logits.is_cuda() && logits.dim() == 2 && logits.stride(1) == 1);
  TORCH_CHECK(logits.scalar_type() == at::kFloat || is_bf16(logits), "topk_sample: fp32 or bf16 logits");
  TORCH_CHECK(global_topk >= 1 && global_topk <= 256);
  const int B = logits.size(0), V = logits.size(1);
  for (const auto* t : {&top_k, &top_p, &temperature, &rand})
    TORCH_CHECK(t->is_cuda() && t->numel() == B, "topk_sample: top_k, top_p, temperature and rand hold a value per row, on the GPU");
  c10::cuda::CUDAGuard guard(logits.device());
  auto out = at::empty({B}, logits.options().dtype(at::kLong));
  if (B == 0) return out;
  auto gmax = at::empty({B, (int64_t)topk_groups(V)}, logits.options().dtype(at::kInt));
  topk_sample_launch(logits.data_ptr(), is_bf16(logits) ? 1 : 0, top_k.data_ptr<int>(), top_p.data_ptr<float>(), temperature.data_ptr<float>(),
                     rand.data_ptr<float>(), reinterpret_cast<uint32_t*>(gmax.data_ptr<int>()), out.data_ptr<int64_t>(), B, V, (int)logits.stride(0),
                     (int)global_topk, cur_stream());
  return out;
}

// ---- attention -----------------------------------------------------------------------------------------------------
int pick_nsplit(int B, int Hkv, int S_hint) {
  const int ctas = B * Hkv;
  // short contexts: one 64-key tile per CTA (latency bound: tiles in parallel, not in sequence);
  // long contexts: ~4 tiles per CTA once the chip is full
  // (measured: splitting a <=512-key context costs more in the combine than the 4-deep tile prefetch hides)
  int want = S_hint <= 512 ? 1 : (S_hint + 255) / 256;
  int cap = std::max(1, (2 * 148) / std::max(ctas, 1));  // fill the chip, not more
  return std::max(1, std::min({want, cap, 64}));
}

at::Tensor attention_decode(const at::Tensor& q, const at::Tensor& k_cache, const at::Tensor& v_cache, const at::Tensor& lines,
                            const at::Tensor& positions, double scale, int64_t window, const c10::optional<at::Tensor>& sinks,
                            int64_t s_hint) {
  TORCH_CHECK(q.is_cuda() && q.dim() == 4 && q.is_contiguous() && is_bf16(q) && is_bf16(k_cache));
  TORCH_CHECK(k_cache.dim() == 4 && k_cache.is_contiguous() && v_cache.is_contiguous());
  const int B = q.size(0), T = q.size(1), Hq = q.size(2), D = q.size(3);
  const int L = k_cache.size(0), Hkv = k_cache.size(1), S = k_cache.size(2);
  TORCH_CHECK(k_cache.size(3) == D && Hq % Hkv == 0);
  TORCH_CHECK(lines.scalar_type() == at::kInt && positions.scalar_type() == at::kInt && positions.is_contiguous() &&
              lines.numel() == B && positions.numel() == B * T);
  c10::cuda::CUDAGuard guard(q.device());
  auto out = at::empty_like(q);
  AttnDecodeParams p{};
  p.q = q.data_ptr(); p.k_cache = k_cache.data_ptr(); p.v_cache = v_cache.data_ptr(); p.out = out.data_ptr();
  p.lines = lines.data_ptr<int>(); p.positions = positions.data_ptr<int>(); p.block_table = nullptr;
  p.sinks = sinks.has_value() ? sinks->data_ptr<float>() : nullptr;
  p.B = B; p.T = T; p.Hq = Hq; p.Hkv = Hkv; p.D = D; p.S = S; p.L = L; p.window = window; p.scale = (float)scale;
  p.nsplit = pick_nsplit(B, Hkv, s_hint > 0 ? (int)std::min<int64_t>(s_hint, S) : S);
  const auto ws = workspace(cur_stream(), (int64_t)B * Hkv * p.nsplit * 64 * (D + 2), 0, (int64_t)B * Hkv);
  p.ws_o = ws.f;
  p.ws_ml = p.ws_o + (int64_t)B * Hkv * p.nsplit * 64 * D;
  p.tickets = ws.tickets;
  attention_decode_launch(p, cur_stream());
  return out;
}

// q/k RMSNorm + RoPE + KV-cache append + split-KV flash decode in ONE kernel (the prologue of the attention kernel).
at::Tensor rope_attention_decode(const at::Tensor& qkv, const at::Tensor& cos, const at::Tensor& sin, at::Tensor& k_cache,
                                 at::Tensor& v_cache, const at::Tensor& lines, const at::Tensor& write_pos,
                                 const at::Tensor& positions, int64_t nq, int64_t nkv, int64_t D, double scale, int64_t window,
                                 const c10::optional<at::Tensor>& sinks, const c10::optional<at::Tensor>& q_norm,
                                 const c10::optional<at::Tensor>& k_norm, double eps, int64_t s_hint) {
  TORCH_CHECK(qkv.is_cuda() && qkv.dim() == 3 && qkv.is_contiguous() && is_bf16(qkv) && is_bf16(k_cache));
  const int B = qkv.size(0), T = qkv.size(1);
  TORCH_CHECK(qkv.size(2) == (nq + 2 * nkv) * D && (D == 64 || D == 128) && nq % nkv == 0);
  TORCH_CHECK(cos.scalar_type() == at::kFloat && cos.is_contiguous() && sin.is_contiguous() &&
              cos.numel() == (int64_t)B * T * D / 2 && sin.numel() == cos.numel());
  TORCH_CHECK(k_cache.dim() == 4 && k_cache.size(1) == nkv && k_cache.size(3) == D && k_cache.is_contiguous() &&
              v_cache.is_contiguous());
  TORCH_CHECK(lines.scalar_type() == at::kInt && positions.scalar_type() == at::kInt && write_pos.scalar_type() == at::kInt &&
              positions.is_contiguous() && write_pos.is_contiguous() && lines.numel() == B && positions.numel() == B * T &&
              write_pos.numel() == B * T);
  c10::cuda::CUDAGuard guard(qkv.device());
  auto out = at::empty({B, T, nq, D}, qkv.options());
  const int L = k_cache.size(0), S = k_cache.size(2);
  AttnDecodeParams p{};
  p.q = nullptr; p.k_cache = k_cache.data_ptr(); p.v_cache = v_cache.data_ptr(); p.out = out.data_ptr();
  p.lines = lines.data_ptr<int>(); p.positions = positions.data_ptr<int>(); p.block_table = nullptr;
  p.sinks = sinks.has_value() ? sinks->data_ptr<float>() : nullptr;
  p.B = B; p.T = T; p.Hq = nq; p.Hkv = nkv; p.D = D; p.S = S; p.L = L; p.window = window; p.scale = (float)scale;
  p.qkv = qkv.data_ptr(); p.cos = cos.data_ptr<float>(); p.sin = sin.data_ptr<float>();
  p.q_norm = optr(q_norm); p.k_norm = optr(k_norm); p.write_pos = write_pos.data_ptr<int>(); p.norm_eps = (float)eps;
  p.nsplit = pick_nsplit(B, nkv, s_hint > 0 ? (int)std::min<int64_t>(s_hint, S) : S);
  const auto ws = workspace(cur_stream(), (int64_t)B * nkv * p.nsplit * 64 * (D + 2), 0, (int64_t)B * nkv);
  p.ws_o = ws.f;
  p.ws_ml = p.ws_o + (int64_t)B * nkv * p.nsplit * 64 * D;
  p.tickets = ws.tickets;
  attention_decode_launch(p, cur_stream());
  return out;
}

// Parts of a row's keys.  The fewer (row, kv head) pairs there are, the more parts fill the chip and shorten the longest row; a part costs a pipeline
// fill and a share of the combine.  us of ragged rows, head size 128, at 1 / 2 / 4 / 8 / 16 / 24 / 37 / 64 parts:
//   1 pair:    4096 keys 66 / 41 / 29 / 21 / 19 / 21 / 23 / 25     32768: 453 / 236 / 127 / 70 / 43 / 37 / 35 / 31      131072: 1776 / 893 / 455 / 236 / 127 / 92 / 72 / 53
//   8 pairs:   4096 keys 64 / 39 / 27 / 21 / 19 / 21 / 23 / 31     32768: 453 / 234 / 127 / 72 / 49 / 47 / 45 / 53      131072: 1772 / 897 / 465 / 242 / 137 / 123 / 111 / 121
//   12 pairs:  4096 keys 65 / 41 / 27 / 21 / 20 / 21 / 27 / 33     32768: 451 / 234 / 125 / 70 / 51 / 43 / 47 / 51      131072: 1778 / 895 / 465 / 242 / 168 / 129 / 137 / 131
//   32 pairs:  1000 keys 23 / 21 / 18 / 16 / 23                    32768: 455 / 240 / 133 / 98 / 98 / 92                131072: 1778 / 918 / 471 / 322 / 268 / 256
//   64 pairs:  500 keys 16 / 16 / 16 / 23 / 31    4096: 66 / 43 / 33 / 35 / 41    8192: 121 / 74 / 53 / 53 / 55         131072: 1788 / 918 / 598 / 518 / 467
//   128 pairs: 500 keys 21 / 22 / 28 / 37         4096: 69 / 57 / 57 / 61         32768: 455 / 301 / 264 / 229 / 223
//   384 pairs: 500 keys 29 / 37 / 49 / 74         4096: 103 / 98 / 100 / 117      32768: 639 / 537 / 475 / 453          1536 pairs, 4096 keys: 256 / 274 / 312 / 391
// Head size 64 has its minima at the same numbers (32768 keys: 1 pair 303 / 172 / 92 / 52 / 33 / 29 / 27 / 25, 32 pairs 309 / 186 / 104 / 70 / 55 / 59 / 59 / 66).
// With 96 to 1023 pairs and up to 64 rows the longest rows start first (eight classes of length): in the order of the rows the parts of the longest ones finished
// last.  us, by length / in their order, at 96, 128, 256, 384 and 512 pairs (8 kv heads; 4 at 256 and 128), head size 128:
//   500 .. 8000 keys: 61 / 75, 63 / 78, 107 / 144, 133 / 157, 210 / 225    1 .. 4096: 34 / 38, 40 / 46, 59 / 73, 86 / 102, 106 / 116
//   1 .. 1500: 20 / 20, 27 / 28, 37 / 41, 52 / 51, 62 / 62    all 4096: 60 / 59, 63 / 63, 104 / 104, 152 / 153, 199 / 199    all 300: 19.5 / 17.9, 21.0 / 20.0, 24.6 / 22.5, 33 / 32, 41.5 / 41.0
// Every CTA finds its row for itself, which costs 0.5 us; an exact rank from keys in shared memory cost 2 .. 5 us.  More rows than a warp holds in two registers:
// in their order.  Parts of one size for all rows (a row as many as it needs) were as fast, but short rows then had fewer parts and errors against 64 bits
// up to 2 % larger: the largest probability of a part is exactly 1 and takes no rounding.
static int paged_nsplit(int pairs, int max_keys) {
  const int tiles = std::max(1, (max_keys + 63) / 64);
  if (pairs >= 1024) return 1;
  if (pairs >= 256) return max_keys >= 3072 ? 2 : 1;
  if (pairs >= 96) return std::max(1, std::min(4, max_keys / 1024));
  const int some = std::min(tiles, pairs > 32 && max_keys <= 8192 ? 4 : pairs > 8 ? 8 : 16);
  return std::max(some, std::min({64, 2 * 148 / pairs, max_keys / 512}));       // long rows: two CTAs per SM of at least 512 keys
}

at::Tensor paged_attention_decode(const at::Tensor& q, const at::Tensor& k_cache, const at::Tensor& v_cache,
                                  const at::Tensor& block_table, const at::Tensor& positions, double scale, int64_t window,
                                  const c10::optional<at::Tensor>& sinks) {
  TORCH_CHECK(q.is_cuda() && q.dim() == 4 && q.is_contiguous() && is_bf16(q) && is_bf16(k_cache));
  TORCH_CHECK(k_cache.dim() == 4 && k_cache.is_contiguous() && v_cache.is_contiguous());
  const int B = q.size(0), T = q.size(1), Hq = q.size(2), D = q.size(3);
  const int bs = k_cache.size(1), Hkv = k_cache.size(2);
  TORCH_CHECK(k_cache.size(3) == D && Hq % Hkv == 0 && block_table.dim() == 2 && block_table.size(0) == B &&
              block_table.scalar_type() == at::kInt && block_table.is_contiguous());
  TORCH_CHECK(positions.scalar_type() == at::kInt && positions.is_contiguous() && positions.numel() == B * T);
  c10::cuda::CUDAGuard guard(q.device());
  auto out = at::empty_like(q);
  AttnDecodeParams p{};
  p.q = q.data_ptr(); p.k_cache = k_cache.data_ptr(); p.v_cache = v_cache.data_ptr(); p.out = out.data_ptr();
  p.lines = nullptr; p.positions = positions.data_ptr<int>(); p.block_table = block_table.data_ptr<int>();
  p.sinks = sinks.has_value() ? sinks->data_ptr<float>() : nullptr;
  p.B = B; p.T = T; p.Hq = Hq; p.Hkv = Hkv; p.D = D; p.S = 0; p.L = 0; p.window = window; p.scale = (float)scale;
  p.block_size = bs; p.max_blocks = block_table.size(1);
  p.nsplit = paged_nsplit(B * Hkv, p.max_blocks * bs);
  p.by_length = B > 1 && B <= ATT_MAX_ORDER && B * Hkv >= 96 && B * Hkv < 1024 ? 1 : 0;
  const int64_t rows = (int64_t)B * Hkv * p.nsplit * T * (Hq / Hkv);
  const auto ws = workspace(cur_stream(), rows * (D + 2), 0, (int64_t)B * Hkv);
  p.ws_o = ws.f;
  p.ws_ml = p.ws_o + rows * D;
  p.tickets = ws.tickets;
  attention_decode_launch(p, cur_stream());
  return out;
}

at::Tensor attention_prefill(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, double scale, int64_t window,
                             const c10::optional<at::Tensor>& sinks, bool causal) {
  TORCH_CHECK(q.is_cuda() && q.dim() == 4 && q.is_contiguous() && k.is_contiguous() && v.is_contiguous() && is_bf16(q) &&
              is_bf16(k) && is_bf16(v));
  const int B = q.size(0), T = q.size(1), Hq = q.size(2), D = q.size(3), Hkv = k.size(2);
  TORCH_CHECK(k.size(0) == B && k.size(1) == T && k.size(3) == D && v.sizes() == k.sizes() && Hq % Hkv == 0);
  c10::cuda::CUDAGuard guard(q.device());
  auto out = at::empty_like(q);
  AttnPrefillParams p{};
  p.q = q.data_ptr(); p.k = k.data_ptr(); p.v = v.data_ptr(); p.out = out.data_ptr();
  p.sinks = sinks.has_value() ? sinks->data_ptr<float>() : nullptr;
  p.B = B; p.T = T; p.Hq = Hq; p.Hkv = Hkv; p.D = D; p.window = window; p.scale = (float)scale;
  p.causal = causal ? 1 : 0;
  attention_prefill_launch(p, cur_stream());
  return out;
}

}  // namespace nxdi

namespace nxdi {
// ---- W8A8 fp8 ------------------------------------------------------------------------------------------------------------------
std::tuple<at::Tensor, at::Tensor> rmsnorm_quant(const at::Tensor& x, const c10::optional<at::Tensor>& gamma, double eps, double offset,
                                                 double clamp) {
  TORCH_CHECK(x.is_cuda() && x.dim() == 2 && x.is_contiguous() && is_bf16(x));
  c10::optional<at::Tensor> g;
  if (gamma.has_value()) {
    g = gamma->contiguous();
    check_norm_weight(*g, x.size(1));
  }
  c10::cuda::CUDAGuard guard(x.device());
  auto q = at::empty(x.sizes(), x.options().dtype(at::kFloat8_e4m3fn));
  auto scale = at::empty({x.size(0)}, x.options().dtype(at::kFloat));
  rmsnorm_quant_launch(x.data_ptr(), optr(g), q.data_ptr(), scale.data_ptr<float>(), (int)x.size(0), (int)x.size(1), (float)eps,
                       (float)offset, (float)clamp, cur_stream());
  return {q, scale};
}
at::Tensor gemm_fp8(const at::Tensor& xq, const at::Tensor& a_scale, const at::Tensor& w, const at::Tensor& w_scale_in,
                    const c10::optional<at::Tensor>& bias_in, int64_t act, const c10::optional<at::Tensor>& residual) {
  TORCH_CHECK(xq.is_cuda() && xq.dim() == 2 && xq.is_contiguous() && xq.scalar_type() == at::kFloat8_e4m3fn);
  TORCH_CHECK(w.dim() == 2 && w.is_contiguous() && w.scalar_type() == at::kFloat8_e4m3fn && w.size(1) == xq.size(1));
  const int M = xq.size(0), K = xq.size(1), N = w.size(0);
  TORCH_CHECK(K % 128 == 0 && a_scale.scalar_type() == at::kFloat && a_scale.numel() == M && w_scale_in.scalar_type() == at::kFloat &&
              (w_scale_in.numel() == 1 || w_scale_in.numel() == N) && a_scale.is_contiguous() && w_scale_in.is_contiguous());
  TORCH_CHECK(w.is_cuda() && a_scale.is_cuda() && w_scale_in.is_cuda(), "gemm_fp8: weights and scales on the GPU expected");
  // (the kernel loads four scales at a time: those of a slice are copied)
  const at::Tensor w_scale = reinterpret_cast<uintptr_t>(w_scale_in.data_ptr()) % 16 == 0 ? w_scale_in : w_scale_in.clone();
  c10::optional<at::Tensor> bias;
  if (bias_in.has_value()) {
    TORCH_CHECK(bias_in->is_cuda() && is_bf16(*bias_in) && bias_in->numel() == N, "gemm_fp8: a bias of ", N, " bf16 values on the GPU expected");
    bias = bias_in->contiguous();
  }
  const bool glu = act != 0;
  const int n_out = glu ? N / 2 : N;
  TORCH_CHECK(n_out % 8 == 0);
  c10::cuda::CUDAGuard guard(xq.device());
  auto y = at::empty({M, n_out}, xq.options().dtype(at::kBFloat16));
  if (residual.has_value()) TORCH_CHECK(!glu && is_bf16(*residual) && residual->is_contiguous() && residual->numel() == y.numel());
  gemm_fp8_launch(xq.data_ptr(), K, w.data_ptr(), a_scale.data_ptr<float>(), w_scale.data_ptr<float>(), (int)w_scale.numel(), optr(bias),
                  optr(residual), y.data_ptr(), n_out, M, N, K, (int)act, cur_stream());
  return y;
}

// Row-parallel GEMM with the reduce-scatter fused into the kernel: x [M, K] (M = segs * rows_per_seg, rows of a segment split
// evenly over the ranks) -> private output [M / world, N] = sum over ranks of x_r w_r^T (+ bias on rank 0) (+ residual).
// `staging` is this rank's symmetric buffer for the partial sums, `mc_ptr` its multicast address.
at::Tensor gemm_reduce_scatter(const at::Tensor& x, const at::Tensor& w, const c10::optional<at::Tensor>& bias, at::Tensor& staging,
                               int64_t mc_ptr, const std::vector<int64_t>& flag_ptrs, int64_t max_tiles, const at::Tensor& step,
                               int64_t call, int64_t rank, int64_t rows_per_seg, const c10::optional<at::Tensor>& residual,
                               int64_t bcast_mc_ptr, const std::vector<int64_t>& done_ptrs, const c10::optional<at::Tensor>& cta_counter) {
  TORCH_CHECK(x.is_cuda() && x.dim() == 2 && w.dim() == 2 && x.size(1) == w.size(1) && is_bf16(x) && is_bf16(w) && w.is_contiguous());
  const int M = x.size(0), K = x.size(1), N = w.size(0), world = flag_ptrs.size();
  TORCH_CHECK(K % 64 == 0 && x.stride(1) == 1 && x.stride(0) % 8 == 0 && world >= 2 && world <= SYMM_MAX_RANKS);
  TORCH_CHECK(is_bf16(staging) && staging.is_contiguous() && staging.numel() == (int64_t)M * N);
  c10::cuda::CUDAGuard guard(x.device());
  const bool bcast = bcast_mc_ptr != 0;   // all-reduce flavour: result lands in the symmetric output buffer of every rank
  auto out = bcast ? at::empty({0}, x.options()) : at::empty({M / world, N}, x.options());
  if (residual.has_value())
    TORCH_CHECK(is_bf16(*residual) && residual->is_contiguous() && residual->numel() == (bcast ? (int64_t)M * N : out.numel()));
  if (bcast) TORCH_CHECK((int)done_ptrs.size() == world && cta_counter.has_value() && cta_counter->is_cuda() && cta_counter->scalar_type() == at::kInt);
  GemmRsArgs rs{};
  for (int i = 0; i < world; ++i) rs.flag_ptrs[i] = flag_ptrs[i];
  rs.mc = reinterpret_cast<const void*>(mc_ptr);
  rs.out = bcast ? nullptr : out.data_ptr();
  rs.bcast_mc = reinterpret_cast<const void*>(bcast_mc_ptr);
  for (int i = 0; i < world && bcast; ++i) rs.done_ptrs[i] = done_ptrs[i];
  rs.cta_counter = bcast ? cta_counter->data_ptr() : nullptr;
  rs.residual = residual.has_value() ? residual->data_ptr() : nullptr;
  rs.step = step.data_ptr();
  rs.call = (int)call; rs.rank = (int)rank; rs.world = world; rs.rows_per_seg = (int)rows_per_seg; rs.max_tiles = (int)max_tiles;
  gemm_tcgen05_launch(x.data_ptr(), (int)x.stride(0), w.data_ptr(), optr(bias), nullptr, staging.data_ptr(), N, M, N, K, 0, cur_stream(), &rs);
  return out;
}

at::Tensor attention_prefill_tc(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, double scale, int64_t window,
                                const c10::optional<at::Tensor>& sinks, bool causal, double softcap) {
  TORCH_CHECK(q.is_cuda() && q.dim() == 4 && q.is_contiguous() && k.is_contiguous() && v.is_contiguous() && is_bf16(q) && is_bf16(k) && is_bf16(v));
  const int B = q.size(0), T = q.size(1), Hq = q.size(2), D = q.size(3), Hkv = k.size(2);
  TORCH_CHECK((D == 128 || (D == 64 && softcap <= 0.0)) && k.size(0) == B && k.size(1) == T && k.size(3) == D && v.sizes() == k.sizes() && Hq % Hkv == 0,
              "attention_prefill_tc: head_dim 128, or 64 without a soft cap; equal q/k lengths");
  c10::cuda::CUDAGuard guard(q.device());
  auto out = at::empty_like(q);
  attention_prefill_tc_launch(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), sinks.has_value() ? sinks->data_ptr<float>() : nullptr,
                              B, T, Hq, Hkv, D, (float)scale, causal ? 1 : 0, (int)window, (float)softcap, cur_stream());
  return out;
}

// ---- symmetric heap + NVLS collectives -------------------------------------------------------------------------------------
// mode 0 all-reduce (in place in the symmetric buffer; `out` = private copy (+ residual) when given), 1 reduce-scatter, 2 all-gather
void nvls_collective(int64_t mode, const std::vector<int64_t>& sig_ptrs, const at::Tensor& step, int64_t rank, int64_t call,
                     int64_t mc_ptr, int64_t local_ptr, const c10::optional<at::Tensor>& residual, const c10::optional<at::Tensor>& out,
                     int64_t segs, int64_t rows_per_seg, int64_t row_elems) {
  TORCH_CHECK(step.is_cuda() && step.scalar_type() == at::kInt);
  if (residual.has_value()) TORCH_CHECK(is_bf16(*residual) && residual->is_contiguous());
  if (out.has_value()) TORCH_CHECK(is_bf16(*out) && out->is_contiguous());
  c10::cuda::CUDAGuard guard(step.device());
  std::vector<long long> sp(sig_ptrs.begin(), sig_ptrs.end());
  nvls_collective_launch((int)mode, sp.data(), step.data_ptr(), (int)rank, (int)sp.size(), (int)call, reinterpret_cast<void*>(mc_ptr),
                         reinterpret_cast<void*>(local_ptr), residual.has_value() ? residual->data_ptr() : nullptr,
                         out.has_value() ? out->data_ptr() : nullptr, (int)segs, (int)rows_per_seg, (int)row_elems, cur_stream());
}

// ---- persistent decode-step kernel -------------------------------------------------------------------------------------
int64_t dstep_new_b(int64_t T) { return dstep_new((int)T); }
void dstep_set_symm_b(int64_t h, const std::vector<int64_t>& recv_ptrs, const at::Tensor& step, int64_t rank, int64_t n_max) {
  std::vector<long long> v(recv_ptrs.begin(), recv_ptrs.end());
  dstep_set_symm(h, v, step.data_ptr(), (int)rank, (int)n_max);
}
void dstep_add_gemv_b(int64_t h, const at::Tensor& w, const at::Tensor& x, const c10::optional<at::Tensor>& bias,
                      const c10::optional<at::Tensor>& norm_w, double eps, double offset, int64_t act,
                      const c10::optional<at::Tensor>& residual, at::Tensor& y, bool allreduce) {
  TORCH_CHECK(w.is_cuda() && w.dim() == 2 && w.is_contiguous() && is_bf16(w) && is_bf16(x) && is_bf16(y));
  TORCH_CHECK(x.dim() == 2 && x.stride(1) == 1 && x.size(1) == w.size(1) && y.dim() == 2 && y.stride(1) == 1 && x.stride(0) % 8 == 0);
  const int N = w.size(0), K = w.size(1);
  TORCH_CHECK(K % 64 == 0 && y.size(1) == (act != 0 ? N / 2 : N) && y.size(0) == x.size(0));
  if (residual.has_value()) TORCH_CHECK(residual->stride(0) == y.stride(0) && residual->stride(1) == 1 && is_bf16(*residual));
  dstep_add_gemv(h, w.data_ptr(), N, K, x.data_ptr(), (int)x.stride(0), optr(bias), optr(norm_w), (float)eps, (float)offset, (int)act,
                 optr(residual), y.data_ptr(), (int)y.stride(0), allreduce);
}
void dstep_add_attn_b(int64_t h, const at::Tensor& qkv, at::Tensor& out, at::Tensor& k_cache, at::Tensor& v_cache,
                      const c10::optional<at::Tensor>& q_norm, const c10::optional<at::Tensor>& k_norm, double eps, int64_t B,
                      int64_t T, int64_t nq, int64_t nkv, int64_t D, double scale, int64_t window, const c10::optional<at::Tensor>& sinks,
                      int64_t s_hint) {
  TORCH_CHECK(is_bf16(qkv) && is_bf16(out) && is_bf16(k_cache) && k_cache.dim() == 4 && k_cache.is_contiguous() && v_cache.is_contiguous());
  TORCH_CHECK(k_cache.size(1) == nkv && k_cache.size(3) == D && qkv.is_contiguous() && out.is_contiguous());
  const int S = k_cache.size(2), L = k_cache.size(0);
  const int nsplit = pick_nsplit((int)B, (int)nkv, s_hint > 0 ? (int)std::min<int64_t>(s_hint, S) : S);
  dstep_add_attn(h, qkv.data_ptr(), out.data_ptr(), k_cache.data_ptr(), v_cache.data_ptr(), optr(q_norm), optr(k_norm), (float)eps,
                 (int)B, (int)T, (int)nq, (int)nkv, (int)D, S, L, (float)scale, (int)window,
                 sinks.has_value() ? sinks->data_ptr<float>() : nullptr, nsplit);
}
void dstep_launch_b(int64_t h, const at::Tensor& positions, const at::Tensor& write_pos, const at::Tensor& lines,
                    const at::Tensor& cos, const at::Tensor& sin, int64_t call_base, int64_t parity_base) {
  TORCH_CHECK(positions.is_cuda() && positions.scalar_type() == at::kInt && write_pos.scalar_type() == at::kInt &&
              lines.scalar_type() == at::kInt && positions.is_contiguous() && write_pos.is_contiguous() && lines.is_contiguous());
  TORCH_CHECK(cos.scalar_type() == at::kFloat && sin.scalar_type() == at::kFloat && cos.is_contiguous() && sin.is_contiguous());
  c10::cuda::CUDAGuard guard(positions.device());
  dstep_launch(h, positions.data_ptr<int>(), write_pos.data_ptr<int>(), lines.data_ptr<int>(), cos.data_ptr<float>(),
               sin.data_ptr<float>(), (int)call_base, (int)parity_base, cur_stream());
}
void register_seqmix(pybind11::module_& m);   // seqmix_bind.cpp
}  // namespace nxdi

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  nxdi::register_seqmix(m);
  m.def("symm_heap_create", [](int64_t bytes, int64_t dev, int64_t world, int64_t rank) { return (int64_t)nxdi::symm_heap_create(bytes, (int)dev, (int)world, (int)rank); });
  m.def("symm_heap_size", [](int64_t h) { return (int64_t)nxdi::symm_heap_size(h); });
  m.def("symm_heap_local_va", [](int64_t h) { return (int64_t)nxdi::symm_heap_local_va(h); });
  m.def("symm_heap_export_fd", [](int64_t h) { return (int64_t)nxdi::symm_heap_export_fd(h); });
  m.def("symm_heap_import_peer", [](int64_t h, int64_t peer, int64_t fd) { return (int64_t)nxdi::symm_heap_import_peer(h, (int)peer, (int)fd); });
  m.def("symm_heap_multicast_supported", [](int64_t dev) { return nxdi::symm_heap_multicast_supported((int)dev); });
  m.def("symm_heap_mc_create", [](int64_t h, int64_t world) { return (int64_t)nxdi::symm_heap_mc_create(h, (int)world); });
  m.def("symm_heap_mc_import", [](int64_t h, int64_t fd) { nxdi::symm_heap_mc_import(h, (int)fd); });
  m.def("symm_heap_mc_add_device", [](int64_t h) { nxdi::symm_heap_mc_add_device(h); });
  m.def("symm_heap_mc_bind_map", [](int64_t h) { return (int64_t)nxdi::symm_heap_mc_bind_map(h); });
  m.def("symm_heap_destroy", [](int64_t h) { nxdi::symm_heap_destroy(h); });
  m.def("nvls_collective", &nxdi::nvls_collective);
  m.def("attention_prefill_tc", &nxdi::attention_prefill_tc);
  m.def("gemm_reduce_scatter", &nxdi::gemm_reduce_scatter);
  m.def("rmsnorm_quant", &nxdi::rmsnorm_quant);
  m.def("gemm_fp8", &nxdi::gemm_fp8);
  m.def("dstep_new", &nxdi::dstep_new_b);
  m.def("dstep_set_symm", &nxdi::dstep_set_symm_b);
  m.def("dstep_add_gemv", &nxdi::dstep_add_gemv_b);
  m.def("dstep_add_attn", &nxdi::dstep_add_attn_b);
  m.def("dstep_finalize", [](int64_t h) { nxdi::dstep_finalize(h); });
  m.def("dstep_num_allreduce", [](int64_t h) { return (int64_t)nxdi::dstep_num_allreduce(h); });
  m.def("dstep_free", [](int64_t h) { nxdi::dstep_free(h); });
  m.def("dstep_launch", &nxdi::dstep_launch_b);
  m.def("rmsnorm", &nxdi::rmsnorm);
  m.def("gemv", &nxdi::gemv);
  m.def("linear", &nxdi::linear);
  m.def("gemv_allreduce", &nxdi::gemv_allreduce);
  m.def("set_prof", [](const c10::optional<at::Tensor>& buf) {
    if (!buf.has_value()) { nxdi::gemv2_set_prof(nullptr, 0); return; }
    TORCH_CHECK(buf->is_cuda() && buf->scalar_type() == at::kLong && buf->is_contiguous());
    nxdi::gemv2_set_prof(reinterpret_cast<unsigned long long*>(buf->data_ptr<int64_t>()), buf->numel() / (148 * 8));
  });
  m.def("prof_count", []() { return (int64_t)nxdi::prof_count(); });
  m.def("gemv2_supported", [](int64_t T, int64_t K, int64_t wt) { return nxdi::gemv2_supported((int)T, (int)K, (int)wt); },
        pybind11::arg("T"), pybind11::arg("K"), pybind11::arg("wt") = 0);
  m.def("moe_decode", &nxdi::moe_decode);
  m.def("moe_small", &nxdi::moe_small);
  m.def("check_waits", &nxdi::check_waits);
  m.def("kernel_launches", &nxdi::kernel_launches);
  m.def("wait_probe", [](int64_t clocks, at::Tensor out) {
    TORCH_CHECK(out.is_cuda() && out.scalar_type() == at::kInt && out.numel() >= 1);
    c10::cuda::CUDAGuard guard(out.device());
    nxdi::wait_probe_launch(clocks, out.data_ptr<int>(), nxdi::cur_stream());
  });
  m.def("moe_grouped", &nxdi::moe_grouped);
  m.def("dequant_bf16", &nxdi::dequant_bf16);
  m.def("gemm", &nxdi::gemm, pybind11::arg("x"), pybind11::arg("w"), pybind11::arg("bias"), pybind11::arg("act"), pybind11::arg("residual"),
        pybind11::arg("out"), pybind11::arg("fresh_weight") = false);
  m.def("symm_alloc", &nxdi::symm_alloc);
  m.def("symm_open", &nxdi::symm_open);
  m.def("symm_close", &nxdi::symm_close);
  m.def("symm_free", &nxdi::symm_free);
  m.def("symm_as_tensor", &nxdi::symm_as_tensor);
  m.def("workspace_rows_in_use", [](int64_t device) { return nxdi::workspace_rows_in_use((int)device); });
  m.def("rope_rows", &nxdi::rope_rows);
  m.def("cache_lines", &nxdi::cache_lines);
  m.def("rope_kv_append", &nxdi::rope_kv_append);
  m.def("rope_kv_split_append", &nxdi::rope_kv_split_append);
  m.def("kv_append", &nxdi::kv_append);
  m.def("paged_kv_append", &nxdi::paged_kv_append);
  m.def("argmax", &nxdi::argmax);
  m.def("topk_sample", &nxdi::topk_sample);
  m.def("attention_decode", &nxdi::attention_decode);
  m.def("paged_attention_decode", &nxdi::paged_attention_decode);
  m.def("rope_attention_decode", &nxdi::rope_attention_decode);
  m.def("attention_prefill", &nxdi::attention_prefill);
}
