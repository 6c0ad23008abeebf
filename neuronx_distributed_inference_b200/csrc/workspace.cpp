// Memory in which the CTAs of one launch meet: fp32 partials, indices, and tickets, which are zero at launch and which the kernel that counts in them leaves zero.
//
// Two launches may share it only if one comes after the other, so it goes by stream and not by device (two engines, or a graph's replay beside eager calls, run at
// the same time):
//   * eager calls: kept for the KEPT (device, stream) pairs that were used last.  Buffers that are outgrown or given up go back to the caching allocator, which
//     hands them out again in the order of their stream; a call holds its own until its kernel is enqueued.
//   * calls under capture: the graph may be replayed on any stream, beside eager calls and other graphs.  Partials come from the graph's memory pool, call by call.
//     Tickets would have to be cleared by a launch of their own then (1.5 us a call); they are a row of a slab that was cleared before, one for each memory pool of
//     graphs and stream of a capture.  (Graphs of one pool share the rest of their memory too, and are not replayed at the same time.)  The row is free again once
//     the pool has no graph left: a CUDA user object, which would tell of that, costs every replay 2 us.  With no row left tickets are cleared call by call.
#include <algorithm>
#include <array>
#include <map>
#include <memory>
#include <mutex>
#include <vector>

#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAFunctions.h>
#include <cuda_runtime.h>
#include <torch/types.h>

#include "api.h"

namespace nxdi {
namespace {

constexpr size_t KEPT = 8;
constexpr int64_t FLOATS = 4 << 20, INTS = 1 << 16, TICKETS = 1 << 14;      // first sizes: growth is rare
constexpr int ROWS = 256;                                                    // of the slab, TICKETS each: 16 MB
constexpr c10::MempoolId_t NO_POOL{0, 0};

struct Buffers {
  at::Tensor f, i, t;
  int64_t nf = 0, ni = 0, nt = 0;
  Workspace ws{};
  void take(int64_t f_, int64_t i_, int64_t t_, at::TensorOptions o) {      // (what is large enough stays)
    if (nf < f_) ws.f = (f = at::empty({nf = f_}, o.dtype(at::kFloat))).data_ptr<float>();
    if (ni < i_) ws.i = (i = at::empty({ni = i_}, o.dtype(at::kInt))).data_ptr<int>();
    if (nt < t_) ws.tickets = reinterpret_cast<unsigned*>((t = at::zeros({nt = t_}, o.dtype(at::kInt))).data_ptr<int>());
  }
};
struct Entry {
  int device;
  cudaStream_t stream;
  unsigned long long used;
  std::shared_ptr<const Buffers> b;
};
struct Row {
  c10::MempoolId_t pool = NO_POOL;      // of the graphs that use it; none: free
  cudaStream_t stream = nullptr;
};
struct Slab {
  at::Tensor t;
  std::array<Row, ROWS> rows;
  int next = 0;
};
struct State {
  std::mutex m;
  std::vector<Entry> entries;
  std::map<int, Slab> slabs;
  std::vector<std::pair<unsigned long long, c10::MempoolId_t>> captures;      // the last few and their pools
  unsigned long long clock = 0;
};
State& state() {
  static State* s = new State;      // never destroyed: its tensors would meet an allocator that is gone
  return *s;
}

void check(cudaError_t e, const char* what) { TORCH_CHECK(e == cudaSuccess, what, " failed: ", cudaGetErrorString(e)); }

Workspace give(const std::shared_ptr<const Buffers>& b) { return {b->ws.f, b->ws.i, b->ws.tickets, b}; }

// the memory pool that a capture allocates from (one look at the allocator's segments for each capture)
c10::MempoolId_t pool_of(State& st, int device, unsigned long long capture) {
  for (auto& c : st.captures)
    if (c.first == capture) return c.second;
  const auto probe = at::empty({1}, at::TensorOptions().device(at::kCUDA, (c10::DeviceIndex)device).dtype(at::kInt));
  const size_t p = reinterpret_cast<size_t>(probe.data_ptr());
  c10::MempoolId_t pool = NO_POOL;
  for (const auto& segment : c10::cuda::CUDACachingAllocator::snapshot(NO_POOL, false).segments)
    if (segment.device == device && p >= segment.address && p - segment.address < segment.total_size) pool = segment.owner_private_pool_id;
  if (st.captures.size() == KEPT) st.captures.erase(st.captures.begin());
  st.captures.emplace_back(capture, pool);
  return pool;
}
// rows whose pools have no graph any more
void free_rows(Slab& s, int device) {
  for (auto& row : s.rows) {
    if (row.pool == NO_POOL) continue;
    int graphs = 0;
    try {
      graphs = c10::cuda::CUDACachingAllocator::getPoolUseCount((c10::DeviceIndex)device, row.pool);
    } catch (const c10::Error&) {      // the allocator has forgotten the pool
    }
    if (graphs == 0) row = Row{};
  }
}
// the capture's row of the slab, or null
unsigned* captured_tickets(State& st, int device, unsigned long long capture, cudaStream_t stream) {
  auto it = st.slabs.find(device);
  if (it == st.slabs.end()) return nullptr;
  const c10::MempoolId_t pool = pool_of(st, device, capture);
  if (pool == NO_POOL) return nullptr;
  Slab& s = it->second;
  auto at_row = [&](int r) { return reinterpret_cast<unsigned*>(s.t.data_ptr<int>()) + (int64_t)r * TICKETS; };
  for (int r = 0; r < ROWS; ++r)
    if (s.rows[r].pool == pool && s.rows[r].stream == stream) return at_row(r);
  free_rows(s, device);
  for (int k = 0; k < ROWS; ++k) {      // in turn: a row rests as long as possible before it is used again
    const int r = (s.next + k) % ROWS;
    if (s.rows[r].pool != NO_POOL) continue;
    s.rows[r] = Row{pool, stream};
    s.next = (r + 1) % ROWS;
    return at_row(r);
  }
  return nullptr;
}

}  // namespace

Workspace workspace(cudaStream_t stream, int64_t nf, int64_t ni, int64_t nt) {
  const int device = c10::cuda::current_device();
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  check(cudaStreamIsCapturing(stream, &status), "cudaStreamIsCapturing");
  const auto options = [&] { return at::TensorOptions().device(at::kCUDA, (c10::DeviceIndex)device); };
  State& st = state();
  std::lock_guard<std::mutex> lock(st.m);
  if (status != cudaStreamCaptureStatusNone) {
    unsigned long long capture = 0;
    check(cudaStreamGetCaptureInfo(stream, &status, &capture), "cudaStreamGetCaptureInfo");
    auto b = std::make_shared<Buffers>();
    if (nt <= TICKETS) b->ws.tickets = captured_tickets(st, device, capture, stream);
    b->take(nf, ni, b->ws.tickets != nullptr ? 0 : nt, options());
    return give(b);
  }
  Entry* e = nullptr;
  for (auto& x : st.entries)
    if (x.stream == stream && x.device == device) e = &x;
  if (e == nullptr) {
    if (st.slabs.find(device) == st.slabs.end()) {
      auto t = at::zeros({(int64_t)ROWS * TICKETS}, options().dtype(at::kInt));
      check(cudaStreamSynchronize(stream), "cudaStreamSynchronize");       // once per device: replays on any stream find the rows zero
      st.slabs[device].t = t;
    }
    if (st.entries.size() == KEPT)
      st.entries.erase(std::min_element(st.entries.begin(), st.entries.end(), [](const Entry& x, const Entry& y) { return x.used < y.used; }));
    st.entries.push_back({device, stream, 0, std::make_shared<const Buffers>()});
    e = &st.entries.back();
  }
  e->used = ++st.clock;
  if (e->b->nf < nf || e->b->ni < ni || e->b->nt < nt) {
    auto b = std::make_shared<Buffers>(*e->b);
    b->take(std::max(nf, FLOATS), std::max(ni, INTS), std::max(nt, TICKETS), options());
    e->b = b;
  }
  return give(e->b);
}

int workspace_rows_in_use(int device) {
  State& st = state();
  std::lock_guard<std::mutex> lock(st.m);
  auto it = st.slabs.find(device);
  if (it == st.slabs.end()) return 0;
  free_rows(it->second, device);
  return (int)std::count_if(it->second.rows.begin(), it->second.rows.end(), [](const Row& r) { return r.pool != NO_POOL; });
}

}  // namespace nxdi
