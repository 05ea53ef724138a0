// The ring through which the warps of a launch pass tracers (k_adaptive) and announce
// that they wait (k_gc_share). Any warp may put and any may take, without locks.
//
// An entry carries the position it was published for in its upper half (plus one, so
// that a cleared ring matches no position), and a taker accepts only the entry of the
// position it is about to claim: a slot that a slower warp has claimed but that still
// holds the old value, or that is not written yet, is not taken for a new one. Nothing
// is cleared behind a taker, so no clear can meet a slot that is in use again. At most
// `entries` values may be in the ring at a time, which the callers' own counts give
// (a tracer is in one ring at most, a warp waits once).
//
// Mem: get (not cached), put, add and cas on 64-bit words; on the device Atomics below.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define RAPT_RING_FN __device__ __forceinline__
#else
#define RAPT_RING_FN inline
#endif

namespace rapt {

using RingWord = unsigned long long;

template <class Mem>
RAPT_RING_FN void ring_put(RingWord* ring, RingWord entries, RingWord* tail, int32_t value) {
  const RingWord at = Mem::add(tail, 1);
  Mem::put(&ring[at % entries], (at + 1) << 32 | (RingWord)(uint32_t)value);
}

// The value at the ring's head, or -1 where there is none (or other takers were faster).
template <class Mem>
RAPT_RING_FN int64_t ring_take(RingWord* ring, RingWord entries, RingWord* head) {
  for (int tries = 0; tries < 4; ++tries) {
    const RingWord at = Mem::get(head);
    const RingWord v = Mem::get(&ring[at % entries]);
    if ((uint32_t)(v >> 32) != (uint32_t)(at + 1)) return -1;
    if (Mem::cas(head, at, at + 1) == at) return (int64_t)(uint32_t)v;
  }
  return -1;
}

#ifdef __CUDACC__
struct Atomics {
  static RAPT_RING_FN RingWord get(const RingWord* p) { return *(const volatile RingWord*)p; }
  static RAPT_RING_FN void put(RingWord* p, RingWord v) { atomicExch(p, v); }
  static RAPT_RING_FN RingWord add(RingWord* p, RingWord v) { return atomicAdd(p, v); }
  static RAPT_RING_FN RingWord cas(RingWord* p, RingWord was, RingWord v) { return atomicCAS(p, was, v); }
};
#endif

}  // namespace rapt
