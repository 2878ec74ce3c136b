// A warp's queue in shared memory, kept apart from the kernels so that a host compiler can
// run it with the lanes in any order between two __syncwarp().
#pragma once
#include <stdint.h>

namespace ds {

// Appends `first` + bit for the bits of `word`, in order, to the `pend` (< 32) indices in
// buf[64]; 32 of them, once there, go to place(32), which reads buf[0..32), and leave.
// Returns how many wait.  The next call stores from pend on, so a lane moves an index
// down only where one is kept: what lies past them belongs to the next call's lanes,
// and nothing orders their stores with these.
template <class Place>
__device__ __forceinline__ int warp_gather(uint16_t* buf, int pend, uint32_t word, int first,
                                           int lane, Place&& place) {
  if (word >> lane & 1u)
    buf[pend + __popc(word & ((1u << lane) - 1u))] = (uint16_t)(first + lane);
  pend += __popc(word);
  if (pend < 32) return pend;
  __syncwarp();
  place(32);
  const uint16_t rest = buf[32 + lane];
  __syncwarp();
  pend -= 32;
  if (lane < pend) buf[lane] = rest;
  return pend;
}

}  // namespace ds
