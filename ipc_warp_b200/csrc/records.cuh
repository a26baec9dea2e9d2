// Appending contact records (contact.py:171-183) from converged code.
#pragma once
#include "common.cuh"

namespace ipcb {

template <class S>
IPCB_D void write_record(const ipcb_contacts& c, int slot, int a1, int a2, int b1, int b2, int e0, int e1, S l0) {
  if (slot < c.capacity) {
    reinterpret_cast<int4*>(c.a1a2b1b2)[slot] = make_int4(a1, a2, b1, b2);
    reinterpret_cast<int2*>(c.e0e1)[slot] = make_int2(e0, e1);
    static_cast<S*>(c.l0)[slot] = l0;
    static_cast<S*>(c.alpha)[slot] = S(1e-6);
    static_cast<S*>(c.lam)[slot] = S(0);
  }
}

// One ballot and one atomicAdd per warp.
IPCB_D int warp_reserve(int* cnt, bool accept) {
  const unsigned lane = threadIdx.x & 31;
  unsigned m = __ballot_sync(0xffffffffu, accept);
  int base = 0;
  if (lane == 0 && m) base = atomicAdd(cnt, __popc(m));
  base = __shfl_sync(0xffffffffu, base, 0);
  return base + __popc(m & ((1u << lane) - 1u));
}

}  // namespace ipcb
