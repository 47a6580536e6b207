// The copying side of a ring of shared-memory slots: one thread that brings
// `total` blocks in order and ends only when none of its copies is in flight.
// The barrier and copy primitives are those of bulk.cuh (included before this
// file), or a test's.
#pragma once

namespace c3d {

// Block g goes to slot g % RING once the readers have arrived on that slot's
// `empty` barrier behind block g - RING; its arrival is signalled on `full`.
// False when a wait gave up (after `wait` clocks): no further block is brought,
// and those in flight are waited for all the same, since the slots become
// another CTA's memory when this one ends.
template <int RING, typename Slot, typename Bar, typename Src>
__device__ inline bool copy_ring(int total, Slot* ring, Bar* full, Bar* empty, unsigned bytes, long long wait,
                                 Src src) {
  bool ok = true;
  int g = 0;
  for (; g < total; ++g) {
    const int slot = g % RING;
    if (g >= RING && !mbar_wait(&empty[slot], (unsigned)(g / RING - 1) & 1u, wait)) {
      ok = false;
      break;
    }
    mbar_arrive_expect_tx(&full[slot], bytes);
    bulk_load(ring[slot], src(g), bytes, &full[slot]);
  }
  for (int k = g > RING ? g - RING : 0; k < g; ++k)
    if (!mbar_wait(&full[k % RING], (unsigned)(k / RING) & 1u, wait)) ok = false;
  return ok;
}

}  // namespace c3d
