// The apply engine's ring of stages and the consumers' wait for one of them, apart
// from the barriers, so that plain C++ can run it too.
#pragma once

#ifdef __CUDACC__
#define RSCHOL_STAGE_FN __device__ __forceinline__
#else
#define RSCHOL_STAGE_FN inline
#endif

namespace rschol {
namespace solvedev {

constexpr int NSTAGE = 3;   // stages of a CTA: item k goes to stage k % NSTAGE, its use k / NSTAGE of it
constexpr int NGRP = 2;     // consumer groups of a CTA: item k belongs to group k % NGRP

// Waits until item k has landed in its stage.  full(s, parity) and empty(s, parity)
// wait for the phase of that parity of a stage's barriers and return false when they
// gave up (in a model: when they would still wait).
//
// A phase is named by its parity alone, so the wait for use u of a stage must not be
// entered while use u - 1 is still on its way: the completed phase u - 2 has the same
// parity.  A stage's uses alternate between the groups (NSTAGE is odd), copies complete
// out of order, and having worked off item k - 2 tells a group nothing about item
// k - 3.  So it first waits until that one has been worked off: its own item
// k - 2 NSTAGE was use u - 2, and use u needs this group, so the empty barrier is in
// phase u - 1 or u and the parity is unambiguous, and then so is the full barrier's.
template <class Full, class Empty>
RSCHOL_STAGE_FN bool stage_landed(int k, Full full, Empty empty) {
  const int s = k % NSTAGE, use = k / NSTAGE;
  if (use > 0 && !empty(s, (use - 1) & 1)) return false;
  return full(s, use & 1);
}

}  // namespace solvedev
}  // namespace rschol
