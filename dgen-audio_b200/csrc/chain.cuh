// Blocks of one launch that hand values to later blocks of the same launch (tiles of a scan along time).
//
// A launch takes its work in the order of a ticket, so a block only ever waits for blocks that already run; the wait
// is bounded all the same (on expiry the status word is set and the block goes on with a zero).  A cell is one 64-bit
// word: the launch's epoch above, the value below, written and read whole, so a cell needs no clearing between
// launches -- what an earlier launch left there carries an older epoch.  The ticket word holds the epoch too: the
// block that takes a launch's last ticket moves it on, which also makes a recorded launch replayable.
#pragma once
#include <stdint.h>

namespace dgchain {

constexpr int WAIT_EXPIRED = 203;          // status word: a tile's predecessor did not answer in time
constexpr uint32_t MAX_POLLS = 1u << 22;

struct Ticket {
  uint32_t index, epoch;
};

// called by ONE thread of every block of the launch
__device__ __forceinline__ Ticket take_ticket(unsigned long long *word, uint32_t total) {
  const unsigned long long v = atomicAdd(word, 1ull);
  const uint32_t index = (uint32_t)v, epoch = (uint32_t)(v >> 32) + 1u;
  if (index == total - 1) atomicAdd(word, (1ull << 32) - total);   // count back to zero, epoch one further
  return {index, epoch};
}

__device__ __forceinline__ void publish(unsigned long long *cell, uint32_t epoch, float v) {
  const unsigned long long w = ((unsigned long long)epoch << 32) | __float_as_uint(v);
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(cell), "l"(w) : "memory");
}

__device__ __forceinline__ bool peek(const unsigned long long *cell, uint32_t epoch, float &v) {
  unsigned long long w;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(cell) : "memory");
  v = __uint_as_float((uint32_t)w);
  return (uint32_t)(w >> 32) == epoch;
}

__device__ __forceinline__ float await(const unsigned long long *cell, uint32_t epoch, int32_t *status) {
  float v;
  for (uint32_t i = 0; i < MAX_POLLS; ++i)
    if (peek(cell, epoch, v)) return v;
  if (status) atomicExch(status, WAIT_EXPIRED);
  return 0.0f;
}

}  // namespace dgchain
