// Who has the scratch of the K-cut tiles, and for how long (see split_scratch.h).
//
// A captured launch runs whenever its graph is replayed, on whatever stream, beside eager launches and
// other graphs. Its scratch is therefore the graph's: a block per capture and captured stream, tied to
// the graph by a user object, which CUDA destroys when the graph, the executables made from it and
// their last replay are done. The block then serves the next capture, or is freed.
#include "split_scratch.h"

#include <cuda_runtime.h>

#include <map>
#include <mutex>
#include <stdexcept>
#include <string>
#include <utility>
#include <vector>

namespace tdb {
namespace {

void check(cudaError_t e, const char* what) {
  if (e != cudaSuccess)
    throw std::runtime_error(std::string("tridist_b200: ") + what + ": " + cudaGetErrorString(e));
}

constexpr int64_t kWordBytes = 2048;      // the words stand in front of the partials
static_assert(2 * kSkSlots * sizeof(uint32_t) <= kWordBytes, "meeting words");

struct Block {
  uint8_t* base = nullptr;
  int64_t bytes = 0;
};

SplitScratch view(const Block& b) {
  SplitScratch s;
  s.words = reinterpret_cast<uint32_t*>(b.base);
  s.partials = reinterpret_cast<float*>(b.base + kWordBytes);
  return s;
}

// A capture of this thread forbids allocation and synchronisation unless they are asked for as safe.
class OutsideCapture {
 public:
  OutsideCapture() { check(cudaThreadExchangeStreamCaptureMode(&mode_), "capture mode"); }
  ~OutsideCapture() { cudaThreadExchangeStreamCaptureMode(&mode_); }
  OutsideCapture(const OutsideCapture&) = delete;
  OutsideCapture& operator=(const OutsideCapture&) = delete;

 private:
  cudaStreamCaptureMode mode_ = cudaStreamCaptureModeRelaxed;
};

// Clears the words of a block that no launch uses.
cudaError_t clear_words(uint8_t* base) {
  cudaStream_t side = nullptr;
  cudaError_t e = cudaStreamCreateWithFlags(&side, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaMemsetAsync(base, 0, kWordBytes, side);
  if (e == cudaSuccess) e = cudaStreamSynchronize(side);
  if (side) cudaStreamDestroy(side);
  return e;
}

Block new_block(int64_t bytes) {
  Block b;
  b.bytes = bytes;
  cudaError_t e = cudaMalloc(&b.base, static_cast<size_t>(bytes));
  if (e == cudaSuccess && (e = clear_words(b.base)) != cudaSuccess) cudaFree(b.base);
  check(e, "split-K scratch");
  return b;
}

// ---- captured launches ---------------------------------------------------------------------------
constexpr int kIdleBlocks = 4;            // blocks of ended graphs kept per process for the next captures

struct Lease {
  int dev;
  std::pair<unsigned long long, cudaStream_t> key;      // capture, captured stream
  Block block;
};
struct Pool {
  std::mutex mu;
  std::map<std::pair<unsigned long long, cudaStream_t>, Lease*> open;
  std::vector<std::pair<int, Block>> idle;               // (device, block)
};
Pool& pool() {
  static Pool* p = new Pool;              // graphs may outlive the static objects of this library
  return *p;
}

// Destructor of a graph's user object: no CUDA call is allowed in it, and it can run on any thread, also
// inside another thread's CUDA call, so the pool's lock is never held across one.
void end_lease(void* arg) {
  Lease* l = static_cast<Lease*>(arg);
  {
    Pool& p = pool();
    std::lock_guard<std::mutex> lk(p.mu);
    auto it = p.open.find(l->key);
    if (it != p.open.end() && it->second == l) p.open.erase(it);
    p.idle.emplace_back(l->dev, l->block);
  }
  delete l;
}

// Gives back what ended graphs have left beyond kIdleBlocks.
void trim() {
  Pool& p = pool();
  std::vector<Block> extra;
  {
    std::lock_guard<std::mutex> lk(p.mu);
    while (p.idle.size() > kIdleBlocks) {
      extra.push_back(p.idle.front().second);
      p.idle.erase(p.idle.begin());
    }
  }
  if (extra.empty()) return;
  OutsideCapture guard;
  for (const Block& b : extra) cudaFree(b.base);
}

SplitScratch of_capture(int dev, cudaStream_t stream, unsigned long long id, cudaGraph_t graph, int64_t bytes) {
  Pool& p = pool();
  const std::pair<unsigned long long, cudaStream_t> key{id, stream};
  Block b;
  {
    std::lock_guard<std::mutex> lk(p.mu);
    auto it = p.open.find(key);
    if (it != p.open.end() && it->second->block.bytes >= bytes) return view(it->second->block);
    auto best = p.idle.end();
    for (auto i = p.idle.begin(); i != p.idle.end(); ++i)
      if (i->first == dev && i->second.bytes >= bytes && (best == p.idle.end() || i->second.bytes < best->second.bytes))
        best = i;
    if (best != p.idle.end()) {
      b = best->second;
      p.idle.erase(best);
    }
  }
  {
    OutsideCapture guard;
    if (b.base == nullptr) b = new_block(bytes);
    else check(clear_words(b.base), "split-K scratch");
  }
  Lease* l = new Lease{dev, key, b};
  cudaUserObject_t obj = nullptr;
  cudaError_t e = cudaUserObjectCreate(&obj, l, end_lease, 1, cudaUserObjectNoDestructorSync);
  if (e != cudaSuccess) {
    end_lease(l);
    check(e, "split-K scratch of a graph");
  }
  e = cudaGraphRetainUserObject(graph, obj, 1, cudaGraphUserObjectMove);
  if (e != cudaSuccess) {
    cudaUserObjectRelease(obj, 1);
    check(e, "split-K scratch of a graph");
  }
  std::lock_guard<std::mutex> lk(p.mu);
  p.open[key] = l;                        // (a smaller one before it stays with the graph)
  return view(b);
}

// ---- eager launches ------------------------------------------------------------------------------
// One block per stream, allocated on its first use and never freed. Past kSkStreams streams of a
// device there is none, and the launch deals whole tiles.
constexpr int kSkStreams = 8;
constexpr int64_t kEagerBytes = kWordBytes + kSkSlots * 2ll * 128 * 256 * 4;

SplitScratch of_stream(int dev, cudaStream_t stream) {
  struct Slot {
    cudaStream_t stream = nullptr;
    Block block;
  };
  static std::mutex mu;
  static Slot per_dev[64][kSkStreams];
  std::lock_guard<std::mutex> lk(mu);
  for (Slot& s : per_dev[dev & 63]) {
    if (s.block.base != nullptr && s.stream != stream) continue;
    if (s.block.base == nullptr) {
      OutsideCapture guard;               // (another stream may be capturing)
      s.block = new_block(kEagerBytes);
      s.stream = stream;
    }
    return view(s.block);
  }
  return {};
}

}  // namespace

SplitScratch split_scratch(cudaStream_t stream, int64_t words) {
  int dev = 0;
  check(cudaGetDevice(&dev), "cudaGetDevice");
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  unsigned long long id = 0;
  cudaGraph_t graph = nullptr;
  check(cudaStreamGetCaptureInfo(stream, &status, &id, &graph), "cudaStreamGetCaptureInfo");
  trim();
  if (status == cudaStreamCaptureStatusInvalidated)
    throw std::runtime_error("tridist_b200: the capture of this stream has failed");
  if (status == cudaStreamCaptureStatusActive)
    return of_capture(dev, stream, id, graph, kWordBytes + words * static_cast<int64_t>(sizeof(float)));
  return of_stream(dev, stream);
}

}  // namespace tdb
