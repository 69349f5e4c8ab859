// Who has the scratch of the K-cut tiles, and for how long (see split_scratch.h).
//
// A captured launch runs whenever its graph is replayed, on whatever stream, beside eager launches and
// other graphs. Its scratch is therefore the graph's: a block per capture and captured stream, tied to
// the graph by a user object, which CUDA destroys when the graph, the executables made from it and
// their last replay are done. The block then serves the next capture, or is freed.
#include "split_scratch.h"

#include <c10/cuda/CUDACachingAllocator.h>
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
// A block per stream, kept from call to call, from torch's allocator: memory allocated on a stream goes
// back to that stream's work only, so a block can be dropped while launches that use it are pending.
// The streams used last keep theirs (38 MB at most); a program that goes round more of them pays for
// an allocation from the cache and a clear of the words (a 2 KB memset) on its calls.
constexpr size_t kStreamBlocks = 16;

struct StreamBlock {
  int dev = -1;
  unsigned long long stream = 0;          // id: a handle can be given out again while old work is pending
  uint64_t used = 0;
  int64_t bytes = 0;
  std::shared_ptr<void> mem;
};
struct StreamBlocks {
  std::mutex mu;
  uint64_t clock = 0;
  std::vector<StreamBlock> blocks;
};

SplitScratch of_stream(int dev, cudaStream_t stream, int64_t bytes) {
  static StreamBlocks& sb = *new StreamBlocks;            // not destroyed under a driver that is gone
  unsigned long long id = 0;
  check(cudaStreamGetId(stream, &id), "cudaStreamGetId");
  std::lock_guard<std::mutex> lk(sb.mu);
  StreamBlock* b = nullptr;
  for (StreamBlock& x : sb.blocks)
    if (x.stream == id && x.dev == dev) b = &x;
  if (b == nullptr) {
    if (sb.blocks.size() < kStreamBlocks) {
      sb.blocks.emplace_back();
      b = &sb.blocks.back();
    } else {
      b = &sb.blocks[0];
      for (StreamBlock& x : sb.blocks)
        if (x.used < b->used) b = &x;
      *b = StreamBlock{};
    }
    b->dev = dev;
    b->stream = id;
  }
  b->used = ++sb.clock;
  if (b->bytes < bytes) {
    b->bytes = 0;
    b->mem.reset();
    std::shared_ptr<void> mem(c10::cuda::CUDACachingAllocator::raw_alloc_with_stream(static_cast<size_t>(bytes), stream),
                              c10::cuda::CUDACachingAllocator::raw_delete);
    check(cudaMemsetAsync(mem.get(), 0, kWordBytes, stream), "split-K scratch");
    b->mem = std::move(mem);
    b->bytes = bytes;
  }
  SplitScratch s = view({static_cast<uint8_t*>(b->mem.get()), b->bytes});
  s.hold = b->mem;
  return s;
}

}  // namespace

SplitScratch split_scratch(cudaStream_t stream, int64_t words) {
  int dev = 0;
  check(cudaGetDevice(&dev), "cudaGetDevice");
  const int64_t bytes = kWordBytes + words * static_cast<int64_t>(sizeof(float));
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  unsigned long long id = 0;
  cudaGraph_t graph = nullptr;
  check(cudaStreamGetCaptureInfo(stream, &status, &id, &graph), "cudaStreamGetCaptureInfo");
  trim();
  if (status == cudaStreamCaptureStatusInvalidated)
    throw std::runtime_error("tridist_b200: the capture of this stream has failed");
  if (status == cudaStreamCaptureStatusActive)
    return of_capture(dev, stream, id, graph, bytes);
  return of_stream(dev, stream, bytes);
}

}  // namespace tdb
