// Host side of the bounded waits (mbar_wait.cuh): one pinned word per kernel, written by a kernel whose wait ran out.
#include <atomic>
#include <mutex>
#include <stdexcept>
#include <string>

#include "api.h"
#include "common.cuh"
#include "mbar_wait.cuh"

namespace nxdi {

static const char* const kWaitNames[WAIT_KERNELS] = {"attention_prefill_tc_kernel", "gemm_pair_kernel", "skinny_gemm_kernel", "ssd_chunk_kernel", "router_logits_tc_kernel", "wait_probe_kernel"};
static std::atomic<unsigned*> g_words{nullptr};

unsigned* wait_word(WaitKernel which) {
  unsigned* w = g_words.load(std::memory_order_acquire);
  if (w == nullptr) {
    static std::mutex m;
    std::lock_guard<std::mutex> lock(m);
    w = g_words.load(std::memory_order_relaxed);
    if (w == nullptr) {
      cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;      // the first launch may be inside a capture
      cudaThreadExchangeStreamCaptureMode(&mode);
      void* p = nullptr;
      const cudaError_t e = cudaHostAlloc(&p, WAIT_KERNELS * sizeof(unsigned), cudaHostAllocPortable | cudaHostAllocMapped);
      cudaThreadExchangeStreamCaptureMode(&mode);
      if (e != cudaSuccess) throw std::runtime_error(std::string("wait status: ") + cudaGetErrorString(e));
      w = static_cast<unsigned*>(p);
      for (int i = 0; i < WAIT_KERNELS; ++i) w[i] = 0u;
      g_words.store(w, std::memory_order_release);
    }
  }
  return w + which;
}

// raises (once) for waits that ran out in kernels that have ended since the last call
void check_waits() {
  unsigned* w = g_words.load(std::memory_order_acquire);
  if (w == nullptr) return;
  for (int i = 0; i < WAIT_KERNELS; ++i)
    if (*const_cast<volatile unsigned*>(w + i) != 0u) {
      *const_cast<volatile unsigned*>(w + i) = 0u;
      throw std::runtime_error(std::string(kWaitNames[i]) + ": a wait inside the kernel ran out; its results and all that was computed from them are invalid");
    }
}

static std::atomic<long long> g_launches[COUNT_KERNELS];
void count_launch(CountedKernel which) { g_launches[which].fetch_add(1, std::memory_order_relaxed); }
std::vector<std::pair<std::string, long long>> kernel_launches() {
  static const char* const names[COUNT_KERNELS] = {"attention_prefill_tc", "attention_prefill_tc_two_tiles", "gemm_pair", "skinny_gemm", "gemm_tcgen05", "ssd_chunk", "router_logits_tc"};
  std::vector<std::pair<std::string, long long>> r;
  for (int i = 0; i < COUNT_KERNELS; ++i) r.emplace_back(names[i], g_launches[i].load(std::memory_order_relaxed));
  return r;
}

// one wait on a barrier that nobody arrives on, given up after `clocks`: what a kernel with such an error reports
__global__ void __launch_bounds__(32) wait_probe_kernel(long long clocks, unsigned* word, int* out) {
  __shared__ uint64_t bar;
  __shared__ int stop;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    stop = 0;
  }
  __syncwarp();
  if (threadIdx.x == 0) *out = mbar_wait(&bar, 0, &stop, word, clocks) ? 1 : 0;
}
void wait_probe_launch(long long clocks, int* out, cudaStream_t stream) {
  if (clocks < 0 || clocks > WAIT_LIMIT) throw std::runtime_error("wait probe: 0 .. WAIT_LIMIT clocks");
  wait_probe_kernel<<<1, 32, 0, stream>>>(clocks, wait_word(WAIT_PROBE), out);
}

}  // namespace nxdi
