// Separable filtering of several quantities of one DNS at once (sepfilter.cu).
#pragma once
#include <vector>

#include "filter.cuh"

namespace exc {

// Quantity filtered: a velocity component, a component of sigma(u) in the
// order s11, s22, s33, s12, s23, s31, or the pressure.
enum SepSource { SEP_U = 0, SEP_SIGMA = 3, SEP_P = 9, SEP_SOURCES = 10 };

// Tap lists of one batch of filters; targets name them by index.
struct SepTaps {
  std::vector<Taps1D> list;
  // index of the taps of build_taps(...) shifted by `shift` fine cells
  int add(int c, bool stag, bool point, const double* fdelta, int nfd, int shift = 0);
  bool bad = false;  // a stencil longer than MAX_TAPS was asked for
};

// One output on the LES grid: source `src` filtered with taps t[0..2] along
// x, y, z; with `src2` >= 0 that source filtered with the same taps is added.
struct SepTarget {
  int src, src2;
  int t[3];
  double* out;
};

// Scratch of the passes, grown to the largest batch asked for and freed by
// the owner.  A batch that would take more than `limit` bytes (some 600^3 with
// ratio 5 for the five LES), or more than there is, goes slab by slab.
struct SepWork {
  double* a = nullptr;  // x-filtered sources, n m words a fine plane each
  double* b = nullptr;  // xy-filtered ones, m^2 words a fine plane each
  size_t na = 0, nb = 0;
  size_t limit = size_t(4) << 30;
};
void sep_free(SepWork* w);

// Fills every target from the velocity u (and the pressure p, if a target
// uses it): three launches for the whole batch, or for each slab of it.  FP64.
int sep_filter(SepWork* w, int n, int c, double inv_h, double visc, const SepTaps& taps,
               const std::vector<SepTarget>& targets, const double* u, const double* p, cudaStream_t st);

}  // namespace exc
