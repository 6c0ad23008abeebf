// The Mamba-2 recurrence step by step, two head channels per thread: a (row, head, 32 head channels) by 128 threads.  ssd_scan_pair_kernel (seqmix.cu) runs it for
// rows of any length, ssd_chunk_kernel (ssd_chunk.cu) for the short rows of a call with prompts.  Included by files that are compiled without fast-math.
#pragma once
#include <cuda_bf16.h>
#include <math.h>

#include "common.cuh"
#include "seqmix.h"

namespace nxdi {
namespace {

template <typename T> __device__ __forceinline__ float ldf(const T* p);
template <> __device__ __forceinline__ float ldf<float>(const float* p) { return *p; }
template <> __device__ __forceinline__ float ldf<__nv_bfloat16>(const __nv_bfloat16* p) { return __bfloat162float(*p); }
__device__ __forceinline__ float sigmoidf_acc(float x) { return 1.f / (1.f + expf(-x)); }

constexpr int SCAN_PT = 16;      // head channels per block
constexpr int SCAN_NS = 8;       // lanes that split the state axis for one channel
constexpr int SCAN_TT = 16;      // time steps staged per batch
constexpr int SCAN_THREADS = SCAN_PT * SCAN_NS;

constexpr int SC2_PT = 32;       // head channels per block
__device__ __forceinline__ unsigned long long f2_pack(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 f2_get(unsigned long long v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ unsigned long long f2_fma(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ unsigned long long f2_mul(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
constexpr int SC2_FLOATS = 2 * (2 * SCAN_TT * 160 + SCAN_TT * SC2_PT) + 2 * SCAN_TT * SC2_PT + 2 * SCAN_TT;       // shared memory

// `sm`: SC2_FLOATS floats on a 16-byte boundary; `tid`: thread of the 128; `sync`: a barrier of the 128; n_tok > 0
template <typename T, class Sync>
__device__ __forceinline__ void ssd_steps(const SsdScanParams& p, float* sm, int b, int n_tok, int line, int ctx, int h, int p0, int tid, Sync&& sync) {
  constexpr int NPT = 16, NP = 160;        // state values per lane: n = ns * 16 + i; padded row of staged B / C (4 floats after every 16)
  constexpr int STAGE = 2 * SCAN_TT * NP + SCAN_TT * SC2_PT;       // B, C, x of a batch of steps
  const int N = p.N, P = p.P;
  float* ys = sm + 2 * STAGE;              // [TT][PT]
  float* zs = ys + SCAN_TT * SC2_PT;       // [TT][PT]
  float* dts = zs + SCAN_TT * SC2_PT;      // [TT]
  float* dAs = dts + SCAN_TT;              // [TT]
  const int pl = tid / SCAN_NS, ns = tid % SCAN_NS;
  const int c0 = 2 * pl, pc = p0 + c0;     // this thread's two head channels (both exist or neither: P is even)
  const int g = h / (p.nh / p.G);
  const int inner = p.nh * P, Cd = inner + 2 * p.G * N;
  const float* xrow = p.xBC + (long long)b * p.T * Cd;
  const T* dtp = (const T*)p.dt_raw + (long long)b * p.dt_sb + h;
  const T* zp = (const T*)p.z + (long long)b * p.z_sb + h * P;
  float rz[4], rdt = 0.f;
  // batch of steps from t0: B, C (zero past N) and x by asynchronous 16-byte copies into stage `buf`, z and dt into registers
  auto fetch = [&](int t0, int buf) {
    const int tt = min(SCAN_TT, n_tok - t0);
    float* st = sm + buf * STAGE;
    const float* rows = xrow + (long long)t0 * Cd;
#pragma unroll
    for (int k = 0; k < SCAN_TT * 32 / SCAN_THREADS; ++k) {
      const int i = tid + SCAN_THREADS * k, t = i >> 5, n = (i & 31) * 4;
      const bool ok = t < tt && n < N;
      const float* src = ok ? rows + (long long)t * Cd + inner + g * N + n : xrow;
      const int at = t * NP + n + (n >> 4) * 4;
      cp_async16(st + at, src, ok);
      cp_async16(st + SCAN_TT * NP + at, ok ? src + p.G * N : xrow, ok);
    }
    {
      const int t = tid >> 3, c = (tid & 7) * 4;
      const bool ok = t < tt && p0 + c < P;
      cp_async16(st + 2 * SCAN_TT * NP + t * SC2_PT + c, ok ? rows + (long long)t * Cd + h * P + p0 + c : xrow, ok);
    }
    cp_async_commit();
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int i = tid + SCAN_THREADS * k, t = i / SC2_PT, c = p0 + i % SC2_PT;
      rz[k] = (t < tt && c < P) ? ldf(zp + (long long)(t0 + t) * p.z_st + c) : 0.f;
    }
    rdt = tid < tt ? ldf(dtp + (long long)(t0 + tid) * p.dt_st) : 0.f;
  };
  fetch(0, 0);
  float* Sg = p.state + ((long long)line * p.nh + h) * N * P + pc;
  unsigned long long S[2][NPT / 2];        // [channel][pair of neighbouring n]
  const bool load = ctx > 0 && pc < P;
#pragma unroll
  for (int i = 0; i < NPT; i += 2) {
    const int n = ns * NPT + i;
    const float2 a = load && n < N ? *reinterpret_cast<const float2*>(Sg + (long long)n * P) : make_float2(0.f, 0.f);
    const float2 d = load && n + 1 < N ? *reinterpret_cast<const float2*>(Sg + (long long)(n + 1) * P) : make_float2(0.f, 0.f);
    S[0][i / 2] = f2_pack(a.x, d.x);
    S[1][i / 2] = f2_pack(a.y, d.y);
  }
  const float negA = -expf(p.A_log[h]), dtb = p.dt_bias[h], Dh = p.D_skip[h];
  int buf = 0;
  for (int t0 = 0; t0 < n_tok; t0 += SCAN_TT, buf ^= 1) {
    const int tt = min(SCAN_TT, n_tok - t0);
    const float *Bs = sm + buf * STAGE, *Cs = Bs + SCAN_TT * NP, *xs = Cs + SCAN_TT * NP;
#pragma unroll
    for (int k = 0; k < 4; ++k) zs[tid + SCAN_THREADS * k] = rz[k];      // read back by the thread that writes it
    if (tid < SCAN_TT) {
      const float v = rdt + dtb;
      const float dt = v > 20.f ? v : log1pf(expf(v));
      dts[tid] = dt;
      dAs[tid] = expf(negA * dt);
    }
    cp_async_wait<0>();
    sync();
    if (t0 + SCAN_TT < n_tok) fetch(t0 + SCAN_TT, buf ^ 1);              // in flight while the current steps are computed
#pragma unroll 1
    for (int tg = 0; tg < tt; tg += 8) {
      float y[2][8];
      auto step = [&](int u) {
        const int t = tg + u;
        const float dA = dAs[t], dt = dts[t];
        const float2 xv = *reinterpret_cast<const float2*>(xs + t * SC2_PT + c0);
        const unsigned long long dA2 = f2_pack(dA, dA);
        const unsigned long long dx[2] = {f2_pack(dt * xv.x, dt * xv.x), f2_pack(dt * xv.y, dt * xv.y)};
        const ulonglong2* Bt = reinterpret_cast<const ulonglong2*>(Bs + t * NP) + ns * 5;
        const ulonglong2* Ct = reinterpret_cast<const ulonglong2*>(Cs + t * NP) + ns * 5;
        unsigned long long acc[2][2] = {{0ull, 0ull}, {0ull, 0ull}};
#pragma unroll
        for (int q = 0; q < 4; ++q) {     // B and C are zero past N: those S stay zero and add nothing
          const ulonglong2 bv = Bt[q], cv = Ct[q];
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            S[c][2 * q] = f2_fma(dA2, S[c][2 * q], f2_mul(dx[c], bv.x));
            S[c][2 * q + 1] = f2_fma(dA2, S[c][2 * q + 1], f2_mul(dx[c], bv.y));
            acc[c][0] = f2_fma(S[c][2 * q], cv.x, acc[c][0]);
            acc[c][1] = f2_fma(S[c][2 * q + 1], cv.y, acc[c][1]);
          }
        }
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const float2 a = f2_get(acc[c][0]), d = f2_get(acc[c][1]);
          y[c][u] = (a.x + a.y) + (d.x + d.y);
        }
      };
      if (tt - tg >= 8) {
#pragma unroll
        for (int u = 0; u < 8; ++u) step(u);
      } else {
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          y[0][u] = y[1][u] = 0.f;
          if (tg + u < tt) step(u);
        }
      }
      // sums over the 8 lanes for 8 steps at once: lane ns ends up with step tg + ns
#pragma unroll
      for (int c = 0; c < 2; ++c) {
#pragma unroll
        for (int o = 4; o > 0; o >>= 1)
#pragma unroll
          for (int i = 0; i < o; ++i) {
            const bool up = ns & o;
            const float other = __shfl_xor_sync(0xffffffffu, up ? y[c][i] : y[c][i + o], o);
            y[c][i] = (up ? y[c][i + o] : y[c][i]) + other;
          }
        const int at = (tg + ns) * SC2_PT + c0 + c;
        ys[at] = y[c][0] + Dh * xs[at];
      }
    }
    sync();
    for (int i = tid; i < tt * SC2_PT; i += SCAN_THREADS) {
      const int t = i / SC2_PT, c = p0 + i % SC2_PT;
      if (c < P) {
        const float zv = zs[i];
        p.y[((long long)b * p.T + t0 + t) * inner + h * P + c] = ys[i] * (zv * sigmoidf_acc(zv));
      }
    }
  }
  if (pc < P) {
#pragma unroll
    for (int i = 0; i < NPT; i += 2) {
      const int n = ns * NPT + i;
      const float2 a = f2_get(S[0][i / 2]), d = f2_get(S[1][i / 2]);
      if (n < N) *reinterpret_cast<float2*>(Sg + (long long)n * P) = make_float2(a.x, d.x);
      if (n + 1 < N) *reinterpret_cast<float2*>(Sg + (long long)(n + 1) * P) = make_float2(a.y, d.y);
    }
  }
}

}  // namespace
}  // namespace nxdi
