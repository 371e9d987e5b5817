// Barrier over all blocks of a cooperative launch (every block resident).
//
// One thread of a block arrives with a release reduction on a counter and
// polls it with acquire loads: 0.9 us with 148 blocks (a relaxed poll with a
// fence 1.3 us, a flag per block that every block polls 7 us, clusters that
// arrive as one 2.2 us).  The counter only ever grows over the launches that
// share it; `epoch` counts the barriers passed before this launch, and the
// last block out of a launch writes it back (finish).
#pragma once
#include <stdint.h>

namespace hp {

struct GridSync {
  unsigned long long* count;  // arrivals since creation
  unsigned long long* epoch;  // barriers passed since creation
  unsigned int* ticket;       // blocks that are through with the launch
  int32_t* err;               // set when a barrier ran out of its polls (device or pinned host memory)
};
constexpr int GRID_SYNC_WORDS = 4;  // 8-byte words the four counters take, all zero at first

// A poll takes about 0.4 us, so a barrier gives up after about a second.
constexpr int GRID_MAX_POLLS = 1 << 22;

// One thread of a block: arrive at barrier `epoch`, then wait for the other
// blocks.  False if they did not come.
__device__ __forceinline__ bool grid_arrive_wait(const GridSync& g, unsigned long long epoch) {
  asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(g.count) : "memory");
  const unsigned long long all = epoch * gridDim.x;
  for (int k = 0; k < GRID_MAX_POLLS; ++k) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(g.count) : "memory");
    if (v >= all) return true;
  }
  *g.err = 1;
  return false;
}

// All threads of a block.
__device__ __forceinline__ bool grid_sync(const GridSync& g, unsigned long long& epoch) {
  __shared__ int s_ok;
  ++epoch;
  __syncthreads();
  if (threadIdx.x == 0) s_ok = grid_arrive_wait(g, epoch);
  __syncthreads();
  return s_ok;  // rewritten only after the next barrier's first __syncthreads
}

// All threads of a block, at the end of the launch: true in one thread of the
// last block out.  A block counts as out once every warp of it is here, so
// what the last one then writes (the counters here, a step count) has been
// read by all threads of the launch, also where it passed no barrier.
__device__ __forceinline__ bool grid_last_out(const GridSync& g, unsigned long long epoch) {
  __syncthreads();
  if (threadIdx.x != 0) return false;
  __threadfence();
  if (atomicAdd(g.ticket, 1u) != gridDim.x - 1) return false;
  *g.ticket = 0u;
  *g.epoch = epoch;
  return true;
}

static inline GridSync grid_sync_at(void* words) {
  unsigned long long* w = (unsigned long long*)words;
  return GridSync{w, w + 1, (unsigned int*)(w + 2), (int32_t*)(w + 3)};
}

}  // namespace hp
