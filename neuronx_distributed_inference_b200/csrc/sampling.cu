// On-device sampling kernels: split arg-max over the vocabulary and global-top-k / top-p / temperature
// multinomial sampling (reference K8 cumsum + K9 topk/argmax kernels, modules/generation/sampling.py:241-464).
#include <cfloat>

#include "api.h"
#include "common.cuh"

namespace nxdi {

template <typename T>
__device__ __forceinline__ float to_f(T v);
template <>
__device__ __forceinline__ float to_f<float>(float v) { return v; }
template <>
__device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

// ---- arg-max -------------------------------------------------------------------------------------------
// grid (nsplit, B).  Partial (value,index) per CTA -> workspace; the last CTA of a row (atomic ticket) reduces.
// Vocabulary-sharded lm_head (sy.world > 1): the row's winner is exchanged with every peer INSIDE this kernel — the
// {value, tag} / {global index, tag} pairs go straight into each rank's slot over NVLink (LL stores), every rank polls its
// `world` slots and picks the same global winner (ties -> lowest index, like a flat arg-max).  Replaces local arg-max +
// NCCL all-gather + five torch glue kernels in the decode graph (reference: modules/generation/sampling.py:306-326).
template <typename T>
__global__ void __launch_bounds__(256) argmax_kernel(const T* __restrict__ logits, int64_t* __restrict__ out,
                                                     float* __restrict__ ws_val, int* __restrict__ ws_idx,
                                                     unsigned* __restrict__ tickets, int V, int ld, const ArgmaxSymm sy) {
  pdl_launch_dependents();
  pdl_wait();
  const int b = blockIdx.y, split = blockIdx.x, nsplit = gridDim.x, tid = threadIdx.x;
  const int chunk = (V + nsplit - 1) / nsplit;
  const int beg = split * chunk, end = min(V, beg + chunk);
  const T* row = logits + (size_t)b * ld;
  float best = -FLT_MAX;
  int bi = 0x7fffffff;
  for (int i = beg + tid; i < end; i += 256) {
    const float v = to_f(row[i]);
    if (v > best || (v == best && i < bi)) { best = v; bi = i; }
  }
  __shared__ float sv[8];
  __shared__ int si[8];
  __shared__ bool last;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
  }
  if ((tid & 31) == 0) { sv[tid >> 5] = best; si[tid >> 5] = bi; }
  __syncthreads();
  if (tid == 0) {
    for (int w = 1; w < 8; ++w)
      if (sv[w] > best || (sv[w] == best && si[w] < bi)) { best = sv[w]; bi = si[w]; }
    ws_val[b * nsplit + split] = best;
    ws_idx[b * nsplit + split] = bi;
    __threadfence();
    last = (atomicAdd(&tickets[b], 1u) == (unsigned)(nsplit - 1));
  }
  __syncthreads();
  if (last && tid < 32) {
    __threadfence();
    float v = -FLT_MAX;
    int ix = 0x7fffffff;
    for (int s = tid; s < nsplit; s += 32) {
      const float ov = reinterpret_cast<volatile float*>(ws_val)[b * nsplit + s];
      const int oi = reinterpret_cast<volatile int*>(ws_idx)[b * nsplit + s];
      if (ov > v || (ov == v && oi < ix)) { v = ov; ix = oi; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, v, o);
      const int oi = __shfl_xor_sync(0xffffffffu, ix, o);
      if (ov > v || (ov == v && oi < ix)) { v = ov; ix = oi; }
    }
    if (sy.world > 1) {
      const uint32_t tag = ll_tag(sy.step, sy.call);
      const int gix = ix + sy.rank * V;
      if (tid < sy.world) {
        float* dst = sy.slots[0];
#pragma unroll
        for (int d = 1; d < SYMM_MAX_RANKS; ++d)
          if (d == tid) dst = sy.slots[d];
        dst += (((size_t)sy.parity * sy.rows_max + b) * sy.world + sy.rank) * 4;
        st_ll(dst, v, tag);
        st_ll(dst + 2, __int_as_float(gix), tag);
      }
      v = -FLT_MAX;
      ix = 0x7fffffff;
      if (tid < sy.world) {
        const float* src = sy.slots[0];
#pragma unroll
        for (int d = 1; d < SYMM_MAX_RANKS; ++d)
          if (d == sy.rank) src = sy.slots[d];
        src += (((size_t)sy.parity * sy.rows_max + b) * sy.world + tid) * 4;
        float a, c;
        uint32_t fa, fc;
        const long long t0 = clock64();
        while (true) {
          ld_ll(src, a, fa);
          ld_ll(src + 2, c, fc);
          if (fa == tag && fc == tag) break;
          if (clock64() - t0 > 8000000000LL) {
            printf("argmax exchange: rank %d timed out waiting for rank %d (row %d, tag %u, seen %u %u)\n", sy.rank, tid, b, tag, fa, fc);
            __trap();
          }
        }
        v = a;
        ix = __float_as_int(c);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, v, o);
        const int oi = __shfl_xor_sync(0xffffffffu, ix, o);
        if (ov > v || (ov == v && oi < ix)) { v = ov; ix = oi; }
      }
    }
    if (tid == 0) {
      out[b] = ix;
      tickets[b] = 0;  // ready for the next launch / graph replay
    }
  }
}

void argmax_launch(const void* logits, int dtype, int64_t* out, float* ws_val, int* ws_idx, unsigned* tickets, int B, int V,
                   int ld, int nsplit, const ArgmaxSymm* symm, cudaStream_t stream) {
  dim3 grid(nsplit, B);
  ArgmaxSymm sy{};
  if (symm != nullptr) sy = *symm;
  if (dtype == 0)
    launch_pdl(argmax_kernel<float>, grid, dim3(256), 0, stream, reinterpret_cast<const float*>(logits), out, ws_val, ws_idx,
               tickets, V, ld, sy);
  else
    launch_pdl(argmax_kernel<__nv_bfloat16>, grid, dim3(256), 0, stream, reinterpret_cast<const __nv_bfloat16*>(logits), out,
               ws_val, ws_idx, tickets, V, ld, sy);
}

// ---- top-k / top-p / temperature sampling ------------------------------------------------------------------
__device__ __forceinline__ uint32_t order_key(float f) {
  uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key_to_float(uint32_t k) {
  uint32_t u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
  return __uint_as_float(u);
}

constexpr int TOPK_MAX = 256;
constexpr int TOPK_THREADS = 1024;
constexpr int TOPK_SLICE = 8192;            // row elements per block of the first kernel: 256 groups of 32
constexpr int TOPK_CAND = 1024;             // candidates kept for the exact choice
constexpr unsigned TOPK_SLACK = 64;         // groups that may be read beyond the k that reach the bound
constexpr int TOPK_MAX_GROUPS = 8192;       // groups per row that fit the second kernel's shared memory (rows up to 262144)

// 16 bytes of a row (8 bf16 or 4 fp32 values) as ordered keys; positions past V give 0
template <typename T> struct RowVec;
template <> struct RowVec<__nv_bfloat16> { static constexpr int N = 8; };
template <> struct RowVec<float> { static constexpr int N = 4; };
template <typename T>
__device__ __forceinline__ void row_keys(const T* __restrict__ row, int i, int V, bool vec, uint32_t (&k)[RowVec<T>::N]) {
  constexpr int N = RowVec<T>::N;
  if (vec && i + N <= V) {
    const uint4 q = *reinterpret_cast<const uint4*>(row + i);
    if constexpr (N == 4) {
      k[0] = order_key(__uint_as_float(q.x)); k[1] = order_key(__uint_as_float(q.y));
      k[2] = order_key(__uint_as_float(q.z)); k[3] = order_key(__uint_as_float(q.w));
    } else {
      k[0] = order_key(bf16lo(q.x)); k[1] = order_key(bf16hi(q.x)); k[2] = order_key(bf16lo(q.y)); k[3] = order_key(bf16hi(q.y));
      k[4] = order_key(bf16lo(q.z)); k[5] = order_key(bf16hi(q.z)); k[6] = order_key(bf16lo(q.w)); k[7] = order_key(bf16hi(q.w));
    }
  } else {
#pragma unroll
    for (int e = 0; e < N; ++e) k[e] = i + e < V ? order_key(to_f(row[i + e])) : 0u;
  }
}

// Kernel 1: the largest key of every group of 32 elements (thread t of a block: the 16-byte pieces t, t + 256, ... of its slice), one
// coalesced pass over the row spread over the whole chip.
template <typename T>
__global__ void __launch_bounds__(256) topk_group_max_kernel(const T* __restrict__ logits, uint32_t* __restrict__ gmax, int V, int ld, int groups) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int N = RowVec<T>::N;
  const T* row = logits + (size_t)blockIdx.x * ld;
  const bool vec = (reinterpret_cast<uintptr_t>(row) & 15) == 0;
  uint32_t m = 0;
#pragma unroll
  for (int j = 0; j < 32 / N; ++j) {
    uint32_t k[N];
    row_keys<T>(row, blockIdx.y * TOPK_SLICE + (j * 256 + (int)threadIdx.x) * N, V, vec, k);
#pragma unroll
    for (int e = 0; e < N; ++e) m = max(m, k[e]);
  }
  gmax[(size_t)blockIdx.x * groups + blockIdx.y * 256 + threadIdx.x] = m;
}

// key of the need-th largest element that `each` visits (it calls its argument with every key of this thread), and how many of those equal
// to it are among the need largest: radix select, most significant byte first.  Ends early, with the smallest key of the bytes found, when at most `slack` more
// elements than needed reach it (after two bytes that is the rule: a pass costs 0.9 us).
template <typename F>
__device__ __forceinline__ void radix_select(unsigned* hist, unsigned* s_prefix, unsigned* s_need, unsigned* s_extra, unsigned need, unsigned slack, F each) {
  const int tid = threadIdx.x;
  if (tid == 0) { *s_prefix = 0; *s_need = need; }
  for (int pass = 0; pass < 4; ++pass) {
    const int shift = 24 - 8 * pass;
    if (tid < 256) hist[tid] = 0;
    __syncthreads();
    if (pass >= 2 && *s_extra <= slack) break;
    const unsigned prefix = *s_prefix, mask = pass == 0 ? 0u : (0xffffffffu << (shift + 8));
    each([&](uint32_t k) {
      if ((k & mask) == prefix) atomicAdd(&hist[(k >> shift) & 0xffu], 1u);
    });
    __syncthreads();
    if (tid < 32) {                         // lane l owns digits 255 - 8 l .. 248 - 8 l, the largest first
      unsigned c[8], sum = 0;
#pragma unroll
      for (int e = 0; e < 8; ++e) { c[e] = hist[255 - 8 * tid - e]; sum += c[e]; }
      unsigned incl = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned n = __shfl_up_sync(0xffffffffu, incl, o);
        if (tid >= o) incl += n;
      }
      const unsigned want = *s_need;
      unsigned acc = incl - sum;
      __syncwarp();
      if (acc < want && (incl >= want || tid == 31)) {
        int e = 0;
        for (; e < 7 && acc + c[e] < want; ++e) acc += c[e];
        *s_prefix = prefix | ((unsigned)(255 - 8 * tid - e) << shift);
        *s_need = want - acc;
        *s_extra = acc + c[e] - want;
      }
    }
    __syncthreads();
  }
}

// Kernel 2, one CTA per row: the k-th largest group maximum is a lower bound of the k-th largest element (k groups hold one at least as
// large), and only groups that reach it can hold one of the k largest: k groups plus ties, 32 elements each, are read again.  Their elements
// from the bound upwards (k plus a few percent for rows in no particular order) are ranked by counting (value, then lowest index).  More than
// TOPK_CAND of them (long runs of equal values, or one group that holds most of the large ones): the row is selected by radix passes over all of
// it, as every row was before (32 rows of 128256 bf16 values: 84 us a call, six scalar passes per row; 12.5 us in a graph with the groups, 14.9 with their bound found to
// its last bit; fp32 13.8 and 15.9).
template <typename T>
__global__ void __launch_bounds__(TOPK_THREADS) topk_sample_kernel(const T* __restrict__ logits, const uint32_t* __restrict__ gmax, int groups,
                                                                   const int* __restrict__ top_k, const float* __restrict__ top_p,
                                                                   const float* __restrict__ temperature, const float* __restrict__ rand,
                                                                   int64_t* __restrict__ out, int V, int ld, int K) {
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ uint32_t s_gmax[];        // [groups]
  __shared__ unsigned hist[256];
  __shared__ unsigned long long cand[TOPK_MAX], raw[TOPK_CAND];
  __shared__ int s_group[TOPK_CAND];
  __shared__ unsigned s_prefix, s_need, s_extra, s_ngroups, s_ncand;
  const int b = blockIdx.x, tid = threadIdx.x;
  const T* row = logits + (size_t)b * ld;
  K = min(K, V);
  int k_eff = top_k[b];
  k_eff = (k_eff <= 0) ? K : min(k_eff, K);
  if (tid == 0) { s_ngroups = 0; s_ncand = 0; }
  for (int i = tid; i < TOPK_MAX; i += TOPK_THREADS) cand[i] = 0ull;
  bool ranked = groups > 0;
  if (ranked) {
    for (int i = tid; i < groups; i += TOPK_THREADS) s_gmax[i] = gmax[(size_t)b * groups + i];
    __syncthreads();
    radix_select(hist, &s_prefix, &s_need, &s_extra, (unsigned)k_eff, TOPK_SLACK, [&](auto f) {
      for (int i = tid; i < groups; i += TOPK_THREADS) f(s_gmax[i]);
    });
    const uint32_t thr = s_prefix;
    for (int i = tid; i < groups; i += TOPK_THREADS)
      if (s_gmax[i] >= thr) {
        const unsigned at = atomicAdd(&s_ngroups, 1u);
        if (at < TOPK_CAND) s_group[at] = i;
      }
    __syncthreads();
    const unsigned ng = s_ngroups;
    ranked = ng <= TOPK_CAND;
    if (ranked) {
      constexpr int N = RowVec<T>::N, PIECES = 32 / N;
      const bool vec = (reinterpret_cast<uintptr_t>(row) & 15) == 0;
      for (unsigned i = tid; i < ng * PIECES; i += TOPK_THREADS) {
        const int g = s_group[i / PIECES], j = i % PIECES;
        const int at = (g >> 8) * TOPK_SLICE + (j * 256 + (g & 255)) * N;
        uint32_t k[N];
        row_keys<T>(row, at, V, vec, k);
#pragma unroll
        for (int e = 0; e < N; ++e)
          if (k[e] >= thr && at + e < V) {
            const unsigned slot = atomicAdd(&s_ncand, 1u);
            if (slot < TOPK_CAND) raw[slot] = ((unsigned long long)k[e] << 32) | (0xffffffffu - (unsigned)(at + e));
          }
      }
      __syncthreads();
      const unsigned n = s_ncand;
      ranked = n <= TOPK_CAND;
      if (ranked && tid < n) {
        const unsigned long long mine = raw[tid];
        int rank = 0;
#pragma unroll 8
        for (unsigned j = 0; j < n; ++j) rank += raw[j] > mine;
        if (rank < k_eff) cand[rank] = mine;
      }
    }
  }
  if (!ranked) {
    __syncthreads();
    radix_select(hist, &s_prefix, &s_need, &s_extra, (unsigned)K, 0u, [&](auto f) {
      for (int i = tid; i < V; i += TOPK_THREADS) f(order_key(to_f(row[i])));
    });
    const unsigned thr = s_prefix, n_eq_take = s_need;       // key of the K-th largest element; how many equal to it belong to the K largest
    if (tid == 0) { s_ngroups = 0; s_ncand = 0; }
    __syncthreads();
    for (int i = tid; i < V; i += TOPK_THREADS) {
      const unsigned k = order_key(to_f(row[i]));
      if (k > thr) {
        const unsigned slot = atomicAdd(&s_ngroups, 1u);
        if (slot < (unsigned)K) cand[slot] = ((unsigned long long)k << 32) | (unsigned)(0xffffffffu - (unsigned)i);
      }
    }
    __syncthreads();
    const unsigned n_gt = min(s_ngroups, (unsigned)K);
    for (int i = tid; i < V; i += TOPK_THREADS) {
      const unsigned k = order_key(to_f(row[i]));
      if (k == thr) {
        const unsigned slot = atomicAdd(&s_ncand, 1u);
        if (slot < n_eq_take && n_gt + slot < (unsigned)K)
          cand[n_gt + slot] = ((unsigned long long)k << 32) | (unsigned)(0xffffffffu - (unsigned)i);
      }
    }
    __syncthreads();
    // bitonic sort (descending) of TOPK_MAX 64-bit keys; empty slots are 0 and sink to the end
    for (int size = 2; size <= TOPK_MAX; size <<= 1) {
      for (int stride = size >> 1; stride > 0; stride >>= 1) {
        if (tid < TOPK_MAX / 2) {
          const int lo = 2 * tid - (tid & (stride - 1));
          const int hi = lo + stride;
          const bool desc = ((lo & size) == 0);
          const unsigned long long a = cand[lo], c = cand[hi];
          if ((a < c) == desc) { cand[lo] = c; cand[hi] = a; }
        }
        __syncthreads();
      }
    }
  }
  __syncthreads();
  if (tid < 32) {
    const int lane = tid;
    const float temp = temperature[b];
    const bool greedy = (temp == 0.f) || (k_eff == 1);
    const float inv_t = (temp == 0.f) ? 1.f : 1.f / temp;
    const float vmax = key_to_float((uint32_t)(cand[0] >> 32)) * inv_t;
    constexpr int PER = TOPK_MAX / 32;
    float e[PER];
    float lsum = 0.f;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      const int i = lane * PER + j;
      float v = 0.f;
      if (i < k_eff) v = __expf(key_to_float((uint32_t)(cand[i] >> 32)) * inv_t - vmax);
      e[j] = v;
      lsum += v;
    }
    const float total = warp_sum(lsum);
    // inclusive scan of lane sums
    float incl = lsum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float n = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += n;
    }
    float run = (incl - lsum) / total;  // exclusive cumulative prob before my chunk
    const float tp = top_p[b];
    float kept = 0.f;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      const float pj = e[j] / total;
      const bool keep = run < tp;  // (cum - p) < top_p : always keeps the first token
      e[j] = keep ? pj : 0.f;
      kept += e[j];
      run += pj;
    }
    const float ktot = warp_sum(kept);
    float kincl = kept;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float n = __shfl_up_sync(0xffffffffu, kincl, o);
      if (lane >= o) kincl += n;
    }
    float cdf = (kincl - kept) / ktot;
    const float r = rand[b];
    int below = 0, nkept = 0;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      cdf += e[j] / ktot;
      if (e[j] > 0.f) {
        ++nkept;
        if (cdf < r) ++below;
      }
    }
    int choice = (int)warp_sum((float)below);
    nkept = (int)warp_sum((float)nkept);
    choice = min(choice, max(nkept, 1) - 1);
    if (greedy) choice = 0;
    if (lane == 0) out[b] = (int64_t)(0xffffffffu - (unsigned)(cand[choice] & 0xffffffffull));
  }
}

// uint32 workspace per row (0: rows too long for the grouped path)
int topk_groups(int V) {
  const long long g = (long long)((V + TOPK_SLICE - 1) / TOPK_SLICE) * 256;
  return g <= TOPK_MAX_GROUPS ? (int)g : 0;
}

void topk_sample_launch(const void* logits, int dtype, const int* top_k, const float* top_p, const float* temperature,
                        const float* rand, uint32_t* gmax, int64_t* out, int B, int V, int ld, int K, cudaStream_t stream) {
  const int groups = topk_groups(V);
  auto go = [&](auto* row) {
    using T = std::remove_const_t<std::remove_pointer_t<decltype(row)>>;
    if (groups > 0) launch_pdl(topk_group_max_kernel<T>, dim3(B, groups / 256), dim3(256), 0, stream, row, gmax, V, ld, groups);
    launch_pdl(topk_sample_kernel<T>, dim3(B), dim3(TOPK_THREADS), (size_t)groups * 4, stream, row, static_cast<const uint32_t*>(gmax), groups, top_k,
               top_p, temperature, rand, out, V, ld, K);
  };
  if (dtype == 0) go(reinterpret_cast<const float*>(logits));
  else go(reinterpret_cast<const __nv_bfloat16*>(logits));
}

}  // namespace nxdi
