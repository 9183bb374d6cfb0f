// The coarse-grid side of one RK stage (lesstep.cu): everything between the
// LES right-hand sides and their Poisson solves, and everything after them,
// one launch each for all fields of an LES grid.
#pragma once
#include "internal.cuh"

namespace exc {

// One LES grid of m^3 cells (M = m^3) at an RK stage.  Vector fields are 3 M
// words; `k` holds the batch of right-hand sides slot after slot: [0] that of
// the target, then `nst` states (exact, no-model, learned), then the fields
// that are only projected.
template <typename T>
struct LesStage {
  int n, c, kind, m;   // fine cells per side, ratio, filter, coarse cells per side
  int s, nst;          // RK stage, states
  const T* ksums;      // box sums of the DNS k
  const T* ssums;      // box sums of the next stage state (null: no target here)
  T* k;
  const T* ub;         // target of this stage
  T* ublast;           // stage 0: keeps ub
  T* mlast;            // stage 0: the projected closure
  T* next;             // target of the next stage
  const T* net;        // closure of the learned state (slot 3), null: none
  const double* fb;    // its fallback flag
  const T* x0;         // states at the step's start, slot after slot
  T *xs, *xfin;        // stage states and the step's result, likewise
  const double* dt;
};

// Slots to project: the states, then at stage 0 the closure, then the next
// target of a volume filter.
template <typename T>
inline int les_slots(const LesStage<T>& a) {
  return a.nst + (a.s == 0 ? 1 : 0) + (a.ssums && a.kind == EXC_FILTER_VOLUME ? 1 : 0);
}

template <typename T>
cudaError_t launch_les_combine(const LesStage<T>& a, cudaStream_t st);
// Slots first .. first + count - 1 of the projection batch (0 = the exact
// state); p: their pressures at row pitch `ppitch`, `pstride` words apart.
template <typename T>
cudaError_t launch_les_apply(const LesStage<T>& a, T h, const T* p, int ppitch, long long pstride, int first, int count,
                             cudaStream_t st);

}  // namespace exc
