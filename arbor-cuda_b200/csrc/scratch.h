// scratch.h - library-owned scratch of one call, and the launches that the
// entries and the engine share.
#pragma once
#include "abi_util.h"

namespace arbor {

// The tight boxes (tight.cuh) of n scenes for one call on `stream`: made by a
// kernel queued at construction in memory that is freed, in stream order, at
// destruction.  `boxes` is null - the pass then traverses Nodes in a fixed order
// (orderbatch.cuh), with the same results - during stream capture (an allocation would become part of the
// graph and bar a second instantiation), when no memory can be had, and above
// kTightMaxScenes.  The memory comes from a pool of the library's own, which
// keeps at most kScratchKeep bytes when nothing uses it; calls on several
// threads and streams each have their own block.
constexpr int kTightMaxScenes = 32;
constexpr size_t kScratchKeep = size_t(56) << 20;
struct TightScratch {
  uint32_t* boxes = nullptr;
  int status = 0;
  cudaStream_t stream;
  TightScratch(const float* P, const uint32_t* Order, const float* Nodes, int n_scenes, const float* C, bool shadows, cudaStream_t s);
  ~TightScratch();
  TightScratch(const TightScratch&) = delete;
  TightScratch& operator=(const TightScratch&) = delete;
};

size_t tight_bytes(int n_scenes);  // n scenes' tight boxes and an instance table
int launch_tight(const float* P, const uint32_t* Order, const float* Nodes, int n_scenes, uint32_t* T, const float* C, bool shadows,
                 cudaStream_t stream);
int launch_trace(const char* name, bool forest, const float* P, const float* Nodes, const uint32_t* Order, const uint32_t* T, const float* C,
                 float* Hit, int width, int height, cudaStream_t stream);
int launch_shade(const char* name, bool forest, const float* P, const float* Nodes, const uint32_t* Order, const uint32_t* T, const float* C,
                 const float* Hit, float* Linear, float* Guide, float* Normal, int width, int height, cudaStream_t stream);

}  // namespace arbor
