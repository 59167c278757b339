// block_emu.h - runs one thread block of device code on the CPU.
//
// The device headers are compiled by the host compiler with the names below in
// place of CUDA's.  Each thread of the block is a fiber (ucontext) of one OS
// thread; a barrier, vote or shuffle gives the others their turn until all have
// arrived, so a run is deterministic.  Loads through __ldg are checked against
// the registered buffers: one outside them is counted and reads zeros.
#pragma once
#include <cuda_runtime.h>
#include <ucontext.h>

#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <functional>
#include <vector>

#undef __shared__
#undef __noinline__
#define __noinline__ __attribute__((noinline))
#define __shared__ static

namespace emu {

struct Range {
  const char *begin, *end;
};
inline std::vector<Range> buffers;
inline long bad_loads = 0, loads = 0;
template <class T>
T load(const T* p) {
  const char* c = reinterpret_cast<const char*>(p);
  loads++;
  for (const Range& r : buffers)
    if (c >= r.begin && c + sizeof(T) <= r.end) return *p;
  bad_loads++;
  T zero;
  memset(&zero, 0, sizeof zero);
  return zero;
}

struct Fiber {
  ucontext_t ctx;
  std::vector<char> stack;
  bool live = false;
};
inline std::vector<Fiber> fibers;
inline ucontext_t scheduler;
inline int current = 0, n_live = 0;
inline unsigned block_x = 0, grid_x = 1;
inline std::function<void()> body;
inline void yield() { swapcontext(&fibers[current].ctx, &scheduler); }

// A group's collective: every member leaves a value, the last to arrive lets
// the others go on.  Two sets of values, so that a thread that is already at
// the next collective does not overwrite what a slower one still reads.
struct Group {
  int arrived = 0;
  unsigned turn = 0;
  uint32_t value[2][1024];
};
inline Group warps[32], block;
inline const uint32_t* meet(Group& g, int rank, int size, uint32_t v) {
  const unsigned t = g.turn;
  g.value[t & 1][rank] = v;
  if (++g.arrived == size) {
    g.arrived = 0;
    g.turn++;
  } else {
    while (g.turn == t) yield();
  }
  return g.value[t & 1];
}
inline const uint32_t* warp_meet(uint32_t v) { return meet(warps[current >> 5], current & 31, 32, v); }

inline void entry() {
  body();
  fibers[current].live = false;
  n_live--;
  for (;;) yield();
}
// Runs f by `threads` threads (whole warps) of block `bx` of `gx`.
inline void run(int threads, unsigned bx, unsigned gx, std::function<void()> f) {
  body = std::move(f);
  block_x = bx;
  grid_x = gx;
  if ((int)fibers.size() != threads) fibers = std::vector<Fiber>(threads);
  block.arrived = 0;
  for (Group& w : warps) w.arrived = 0;
  for (int k = 0; k < threads; k++) {
    Fiber& b = fibers[k];
    b.stack.resize(128 * 1024);
    getcontext(&b.ctx);
    b.ctx.uc_stack.ss_sp = b.stack.data();
    b.ctx.uc_stack.ss_size = b.stack.size();
    b.ctx.uc_link = nullptr;
    b.live = true;
    makecontext(&b.ctx, entry, 0);
  }
  n_live = threads;
  while (n_live > 0)
    for (current = 0; current < threads; current++)
      if (fibers[current].live) swapcontext(&scheduler, &fibers[current].ctx);
}
struct Index {
  unsigned x, y, z;
};

}  // namespace emu

#define threadIdx (emu::Index{(unsigned)emu::current, 0u, 0u})
#define blockIdx (emu::Index{emu::block_x, 0u, 0u})
#define blockDim (emu::Index{(unsigned)emu::fibers.size(), 1u, 1u})
#define gridDim (emu::Index{emu::grid_x, 1u, 1u})

template <class T>
T __ldg(const T* p) { return emu::load(p); }
inline uint32_t __float_as_uint(float f) { uint32_t u; memcpy(&u, &f, 4); return u; }
inline int __float_as_int(float f) { return (int)__float_as_uint(f); }
inline float __uint_as_float(uint32_t u) { float f; memcpy(&f, &u, 4); return f; }
inline float __int_as_float(int i) { return __uint_as_float((uint32_t)i); }
inline float __fmaf_rn(float a, float b, float c) { return fmaf(a, b, c); }
inline float __sinf(float x) { return sinf(x); }
inline float __cosf(float x) { return cosf(x); }
inline float __expf(float x) { return expf(x); }
inline int __clz(uint32_t x) { return x ? __builtin_clz(x) : 32; }
inline int __popc(uint32_t x) { return __builtin_popcount(x); }
inline uint32_t __byte_perm(uint32_t x, uint32_t y, uint32_t s) {
  const uint64_t v = (uint64_t)y << 32 | x;
  uint32_t r = 0;
  for (int k = 0; k < 4; k++) r |= (uint32_t)(v >> (8 * ((s >> (4 * k)) & 7)) & 255) << (8 * k);
  return r;
}
inline int min(int a, int b) { return a < b ? a : b; }
inline uint32_t min(uint32_t a, uint32_t b) { return a < b ? a : b; }
inline int max(int a, int b) { return a > b ? a : b; }
inline uint32_t max(uint32_t a, uint32_t b) { return a > b ? a : b; }
inline int atomicAdd(int* p, int v) { const int o = *p; *p += v; return o; }
inline int atomicMax(int* p, int v) { const int o = *p; *p = o > v ? o : v; return o; }
inline void __syncthreads() { emu::meet(emu::block, emu::current, (int)emu::fibers.size(), 0); }
inline int __syncthreads_or(int v) {
  const uint32_t* a = emu::meet(emu::block, emu::current, (int)emu::fibers.size(), v != 0);
  for (size_t k = 0; k < emu::fibers.size(); k++)
    if (a[k]) return 1;
  return 0;
}
inline void __syncwarp() { emu::warp_meet(0); }
inline unsigned __ballot_sync(unsigned, int p) {
  const uint32_t* a = emu::warp_meet(p != 0);
  unsigned m = 0;
  for (int k = 0; k < 32; k++) m |= a[k] << k;
  return m;
}
inline int __any_sync(unsigned f, int p) { return __ballot_sync(f, p) != 0; }
inline int __all_sync(unsigned f, int p) { return __ballot_sync(f, p) == 0xffffffffu; }
inline int __shfl_sync(unsigned, int v, int from) { return (int)emu::warp_meet((uint32_t)v)[from & 31]; }
inline int __reduce_max_sync(unsigned, int v) {
  const uint32_t* a = emu::warp_meet((uint32_t)v);
  int m = (int)a[0];
  for (int k = 1; k < 32; k++) m = m > (int)a[k] ? m : (int)a[k];
  return m;
}
