// Coarse-grid kernels of an RK stage: the closure and the right-hand sides of
// every LES state in one pass (les_combine_kernel), then pressure gradient,
// RK update and targets in another (les_apply_kernel).
//
// An LES grid of a stepper has 16^3 to 64^3 cells, where a launch costs more
// than its work: the RHS, the Poisson solve and the updates of the target and
// of the two or three states are one batch of slots, so that a stage takes a
// right-hand side, this combine, one batched solve and this apply instead of
// three or four of each with copies and additions between them.
// Ten steps with the LES beside the DNS, separate passes against batched:
//   FP64 90^3, ratios 5 and 3   19.9 -> 12.8 ms    FP32  72^3, 4 and 2  18.8 -> 12.3
//   FP64 128^3, ratio 4         17.5 -> 14.6       FP32  72^3, 3        10.2 ->  7.1
// and four of FP32 512^3 with four LES 75.5 -> 71.0 ms (fewer passes over
// memory).  Both kernels are bound by launch and latency at these sizes.
#include "filter.cuh"
#include "internal.cuh"
#include "lesstep.cuh"

namespace exc {

// For cell g of component blockIdx.y:
//   m_s = filter(k_s) - RHS_H(ubar_s);  exact: RHS_H(v) + m_s;
//   stage 0: m_0 to be projected, ubar_0 kept;  learned: RHS_H(v) + net(v);
//   the own-axis taps of the next target.
// The rounding is that of the separate passes (filter, subtract, add).
template <typename T>
__global__ void les_combine_kernel(LesStage<T> a, Taps1D taps, double scale, T* __restrict__ mdst,
                                   T* __restrict__ tdst) {
  const int comp = blockIdx.y;
  const long long M = (long long)a.m * a.m * a.m;
  const long long Mt = (long long)a.n * a.m * a.m;
  const bool learned = a.net && a.fb[0] == 0.0;
  const IdxDiv dm(a.m);
  for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < M; g += (long long)gridDim.x * blockDim.x) {
    const long long i = comp * M + g;
    const OaCell cell(dm, a.m, g, comp);
    T m = oa_value<T>(a.ksums + comp * Mt, a.n, a.c, a.m, taps, scale, cell, comp);
    m -= a.k[i];
    a.k[3 * M + i] += m;
    if (mdst) {
      mdst[i] = m;
      a.ublast[i] = a.ub[i];
    }
    if (learned) a.k[9 * M + i] += a.net[i];
    if (tdst) tdst[i] = oa_value<T>(a.ssums + comp * Mt, a.n, a.c, a.m, taps, scale, cell, comp);
  }
}

template <typename T>
cudaError_t launch_les_combine(const LesStage<T>& a, cudaStream_t st) {
  const long long M = (long long)a.m * a.m * a.m;
  const Taps1D taps = build_taps(a.c, true, a.kind == EXC_FILTER_FACE, nullptr, 0);
  const double scale = 1.0 / ((double)a.c * a.c);
  T* p = a.k + 3 * M * (1 + a.nst);
  T* const mdst = a.s == 0 ? p : nullptr;
  if (mdst) p += 3 * M;
  T* const tdst = !a.ssums ? nullptr : a.kind == EXC_FILTER_VOLUME ? p : a.next;
  const long long blocks = (M + 127) / 128;
  les_combine_kernel<T><<<dim3((int)std::min(blocks, 152LL * 16), 3), 128, 0, st>>>(a, taps, scale, mdst, tdst);
  return cudaGetLastError();
}

// k = rhs - grad p of one slot, two cells of a row per thread (m is even):
// gradient2_kernel's and rk_stage_kernel's expressions.  States take the RK
// update, the other slots go to their fields.
template <typename T>
__global__ void les_apply_kernel(LesStage<T> a, T inv_h, const T* __restrict__ p, int ppitch, long long pstride,
                                 int first) {
  using V2 = typename std::conditional<sizeof(T) == 8, double2, float2>::type;
  const int m = a.m, slot = first + blockIdx.y;
  const long long M = (long long)m * m * m;
  const T* const k = a.k + 3 * M * (1 + slot);
  p += blockIdx.y * pstride;
  const bool state = slot < a.nst;
  T* const out = a.s == 0 && slot == a.nst ? a.mlast : a.next;
  const T* const x0 = a.x0 + 3 * M * slot;
  T* const xs = a.xs + 3 * M * slot;
  T* const xfin = a.xfin + 3 * M * slot;
  T cf = 0, cs = 0;
  if (state) {
    const double dt = a.dt[0];
    cf = (T)((a.s == 0 || a.s == 3) ? dt / 6.0 : dt / 3.0);
    cs = (T)(a.s == 2 ? dt : 0.5 * dt);
  }
  const IdxDiv dh(m / 2), dm(m);
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < M / 2; t += (long long)gridDim.x * blockDim.x) {
    const long long row = dh.div(t);
    const int x = 2 * (int)(t - row * (m / 2));
    const int z = (int)dm.div(row), y = (int)(row - (long long)z * m);
    const T* const pr = p + row * ppitch;
    const V2 pc = *reinterpret_cast<const V2*>(pr + x);
    const T pn = pr[x + 2 == m ? 0 : x + 2];
    const V2 py = *reinterpret_cast<const V2*>(p + ((long long)z * m + wrap_up(y, m)) * ppitch + x);
    const V2 pz = *reinterpret_cast<const V2*>(p + ((long long)wrap_up(z, m) * m + y) * ppitch + x);
    const V2 d[3] = {{pc.y - pc.x, pn - pc.y}, {py.x - pc.x, py.y - pc.y}, {pz.x - pc.x, pz.y - pc.y}};
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const long long g = c * M + 2 * t;
      V2 v = *reinterpret_cast<const V2*>(k + g);
      v.x -= d[c].x * inv_h;
      v.y -= d[c].y * inv_h;
      if (!state) {
        *reinterpret_cast<V2*>(out + g) = v;
        continue;
      }
      V2 b{}, f;
      if (a.s < 3) b = *reinterpret_cast<const V2*>(x0 + g);
      f = a.s == 0 ? b : *reinterpret_cast<const V2*>(xfin + g);
      f.x += cf * v.x;
      f.y += cf * v.y;
      *reinterpret_cast<V2*>(xfin + g) = f;
      if (a.s < 3) {
        b.x += cs * v.x;
        b.y += cs * v.y;
        *reinterpret_cast<V2*>(xs + g) = b;
      }
    }
  }
}

template <typename T>
cudaError_t launch_les_apply(const LesStage<T>& a, T h, const T* p, int ppitch, long long pstride, int first, int count,
                             cudaStream_t st) {
  const long long M = (long long)a.m * a.m * a.m;
  const long long blocks = (M / 2 + 127) / 128;
  les_apply_kernel<T><<<dim3((int)std::min(blocks, 152LL * 16), count), 128, 0, st>>>(
      a, (T)(1.0 / (double)h), p, ppitch, pstride, first);
  return cudaGetLastError();
}

#define INST(T)                                                                             \
  template cudaError_t launch_les_combine<T>(const LesStage<T>&, cudaStream_t);             \
  template cudaError_t launch_les_apply<T>(const LesStage<T>&, T, const T*, int, long long, int, int, cudaStream_t);
INST(double)
INST(float)
#undef INST

}  // namespace exc
