// Separable filter stencils (see filter.cu).
#pragma once
#include "exc_common.cuh"

namespace exc {

constexpr int MAX_TAPS = 40;

struct Taps1D {
  int cnt;
  int off[MAX_TAPS];
  double w[MAX_TAPS];
};
struct Taps3 {
  Taps1D a[3];  // x, y, z
};

Taps1D build_taps(int c, bool stag, bool point, const double* fdelta, int nfd);
int make_taps3(int c, const bool stag[3], const bool point[3], const double* fdelta, int nfd, Taps3* out);

// Coarse cell g of a vector component on an m^3 grid, and its value of the
// own-axis taps over the transverse sums tb: accumulated in the field's word
// type (FP32 form: no FP64-pipe work), the scaling rounded by itself.
struct OaCell {
  int ix, iy, iz, own;
  __device__ __forceinline__ OaCell(const IdxDiv& dm, int m, long long g, int comp) {
    const long long r = dm.div(g);
    ix = (int)(g - r * m);
    iz = (int)dm.div(r);
    iy = (int)(r - (long long)iz * m);
    own = comp == 0 ? ix : (comp == 1 ? iy : iz);
  }
};
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
template <typename T>
__device__ __forceinline__ T oa_value(const T* __restrict__ tb, int n, int c, int m, const Taps1D& taps, double scale,
                                      const OaCell& q, int comp) {
  T acc = (T)0;
  for (int t = 0; t < taps.cnt; ++t) {
    int fi = c * q.own + taps.off[t];
    fi = fi >= n ? fi - n : (fi < 0 ? fi + n : fi);
    long long idx;
    if (comp == 0) idx = ((long long)q.iz * m + q.iy) * n + fi;
    else if (comp == 1) idx = ((long long)q.iz * n + fi) * m + q.ix;
    else idx = ((long long)fi * m + q.iy) * m + q.ix;
    acc += (T)taps.w[t] * tb[idx];
  }
  return mul_rn(acc, (T)scale);
}

template <typename T>
int filter_vector(int n, int c, int kind, const double* fdelta, int nfd, const T* u, T* ub, cudaStream_t st);
// Box-only volume/face filter in two coalesced passes; tb: 3 n (n/c)^2 words
// of scratch.
template <typename T>
cudaError_t filter_vector_box(int n, int c, int kind, const T* u, T* ub, T* tb, cudaStream_t st);
// Its passes: transverse c x c sums of the fine field (tb), the same sums of
// ratio ct = r cf from those of ratio cf, and the own-axis taps into ub.
template <typename T>
cudaError_t box_tb(int n, int c, const T* u, T* tb, cudaStream_t st);
template <typename T>
cudaError_t box_tb_coarsen(int n, int cf, int ct, const T* tbf, T* tbt, cudaStream_t st);
template <typename T>
cudaError_t box_oa(int n, int c, int kind, const T* tb, T* ub, cudaStream_t st);
template <typename T>
int closure_flux(int n, int c, double l, double visc, const double* fdelta, int nfd, const T* u, const T* p,
                 T* r9, cudaStream_t st);
template <typename T>
int filtered_stress(int n, int c, double l, double visc, const double* fdelta, int nfd, const T* u, T* s6,
                    cudaStream_t st);

}  // namespace exc
