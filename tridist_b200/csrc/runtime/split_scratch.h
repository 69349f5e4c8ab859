// Device scratch of the GEMM tiles that are cut along K (partials and the words their workers meet at).
#pragma once
#include <cuda_runtime_api.h>

#include <cstdint>
#include <memory>

namespace tdb {

constexpr int kSkSlots = 160;     // CTAs of a launch that can take part in a cut tile

struct SplitScratch {
  float* partials = nullptr;
  uint32_t* words = nullptr;      // [2][kSkSlots], zero between launches
  std::shared_ptr<void> hold;     // keeps the memory until the launch is in the stream
};

// Scratch for the next launch on `stream`, with room for `words` fp32 partials. No other launch that
// could run at the same time has it: launches of one stream follow one another and share one; a launch
// that is being captured gets one that belongs to the graph, for as long as the graph lives.
SplitScratch split_scratch(cudaStream_t stream, int64_t words);

}  // namespace tdb
