// RHS sweep: du = doadd*du - div sigma(u) (`stresstensor` + `tensordivergence!`,
// src/N.jl:94-160), marching along z.
//
// A CTA of 32 x 8 threads owns a PTX x PTY column of cells (PTY = 8 NC, NC
// consecutive rows per thread) and walks ptz planes (4 to 32).  Three plane buffers of u
// with a one-cell x/y halo sit in shared memory: planes z and z+1 are read
// while plane z+2 streams in with cp.async; each thread evaluates the six
// stress components at its own cells (the edge stresses s13, s23 and the
// diagonal s33 of the next plane are kept in registers for the next plane),
// six warps evaluate the halo stresses lane-parallel (one task per warp), and
// the divergence is formed from shared memory and registers.  Every stress
// value is computed once (plus the x/y halo), copy offsets are computed once
// per thread, and global loads and stores are row-contiguous.
#include <cuda.h>  // CUtensorMap (the encoder is reached through the runtime's driver entry point)

#include <cstring>
#include <mutex>
#include <type_traits>

#include "fixed.cuh"
#include "internal.cuh"

namespace exc {

// Set when a wait for a TMA plane gave up (the copy never completed): the
// sweep then ran on incomplete data; read and cleared by exc_device_faults.
__device__ int g_rhs_tma_fault = 0;
// Wait drill (exc_debug_wait_drill bit 0): tiles that would take their planes
// by TMA issue no copy at all, so their plane waits give up after
// RHS_DRILL_POLLS polls with nothing in flight (the sweep's output is then
// not valid); 0 in normal operation.
__device__ int g_rhs_drill = 0;
constexpr int RHS_POLLS = 1 << 20, RHS_DRILL_POLLS = 64;

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// 4-D tiled TMA load of one box (x, y, z, component)
__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* map, int x, int y, int z, int c,
                                            unsigned long long* bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];\n" ::"r"(
          smem_u32(dst)),
      "l"(reinterpret_cast<unsigned long long>(map)), "r"(x), "r"(y), "r"(z), "r"(c), "r"(smem_u32(bar))
      : "memory");
}
// 3-D tiled TMA load of one box (x, y, z) of the tensor map into shared memory
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int x, int y, int z,
                                            unsigned long long* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n" ::"r"(
          smem_u32(dst)),
      "l"(reinterpret_cast<unsigned long long>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
      : "memory");
}

constexpr int PTX = 32, NWARP = 8;
constexpr int PBX = PTX + 2;  // plane box with one-cell halo (box x = x - x0 + 1)
// u rows in shared memory: box x index xb sits at xb + SH<T>, so the 32
// interior cells start on a 16-byte boundary and arrive by 16-byte copies
template <typename T> constexpr int SH = 16 / (int)sizeof(T) - 1;
template <typename T> constexpr int UROW = ((SH<T> + PBX) + 16 / (int)sizeof(T) - 1) / (16 / (int)sizeof(T)) *
                                           (16 / (int)sizeof(T));
// NC cells per thread along y: a tile is PTY = 8 NC rows
template <int NC> constexpr int PTYT = NWARP * NC;
template <int NC> constexpr int PBYT = PTYT<NC> + 2;

// One component plane of a buffer: PBY rows of UROW words, padded to a
// multiple of 128 bytes (TMA destinations); u[c][row] is the row's pointer.
template <typename T, int NC>
struct CompPlane {
  static constexpr int WORDS = PBYT<NC> * UROW<T>;
  static constexpr int PADDED = (WORDS * (int)sizeof(T) + 127) / 128 * 128 / (int)sizeof(T);
  T r[PBYT<NC>][UROW<T>];
  T pad[PADDED > WORDS ? PADDED - WORDS : 128 / (int)sizeof(T)];
  __device__ __forceinline__ const T* operator[](int row) const { return r[row]; }
  __device__ __forceinline__ T* operator[](int row) { return r[row]; }
};

template <typename T, int NC>
struct PlaneSmem {
  CompPlane<T, NC> u[3][3];  // [plane buffer][component]
  T s[5][PBYT<NC>][PBX];     // s11, s22, s12, s13, s23 of the current plane
  unsigned long long bar[3];  // TMA completion of each plane buffer
};
// dynamic shared memory of rhs_kernel: the struct plus room to align it to
// 128 bytes
template <typename T, int NC>
constexpr size_t plane_smem_bytes() {
  return sizeof(PlaneSmem<T, NC>) + 128;
}

// Stress values, kept as 4 sigma; the divergence takes 1/(4h).  Diagonal: a
// at the cell, b its lower neighbour along i; cd = 2 rv, rv = 4 visc / h.
template <typename T>
__device__ __forceinline__ T sdiag_of(T a, T b, T cd) {
  const T s = a + b, d = a - b;
  return s * s - cd * d;
}
// Off-diagonal: a = u_i, b = u_i(+e_j), c = u_j, d = u_j(+e_i); co = rv.
template <typename T>
__device__ __forceinline__ T soff_of(T a, T b, T c, T d, T co) {
  return (a + b) * (c + d) - co * ((b - a) + (d - c));
}
// sigma_ii at box (bx, by) of plane buffer b (uses u_i at the cell and at -e_i)
template <typename T, int I, typename U>
__device__ __forceinline__ T sdiag(const U& u, int bx, int by, T cd) {
  bx += SH<T>;
  return sdiag_of(u[I][by][bx], I == 0 ? u[0][by][bx - 1] : u[1][by - 1][bx], cd);
}
// sigma_12 at box (bx, by): u1, u1(+y), u2, u2(+x)
template <typename T, typename U>
__device__ __forceinline__ T s12(const U& u, int bx, int by, T co) {
  bx += SH<T>;
  return soff_of(u[0][by][bx], u[0][by + 1][bx], u[1][by][bx], u[1][by][bx + 1], co);
}
// sigma_13 at box (bx, by): u1, u1(+z) [next plane], u3, u3(+x)
template <typename T, typename U>
__device__ __forceinline__ T s13(const U& uc, const U& un, int bx, int by, T co) {
  bx += SH<T>;
  return soff_of(uc[0][by][bx], un[0][by][bx], uc[2][by][bx], uc[2][by][bx + 1], co);
}
// sigma_23 at box (bx, by): u2, u2(+z) [next plane], u3, u3(+y)
template <typename T, typename U>
__device__ __forceinline__ T s23(const U& uc, const U& un, int bx, int by, T co) {
  bx += SH<T>;
  return soff_of(uc[1][by][bx], un[1][by][bx], uc[2][by][bx], uc[2][by + 1][bx], co);
}
// sigma_33 between planes: u3 of the upper plane and of the lower plane
template <typename T>
__device__ __forceinline__ T s33(T up, T lo, T cd) {
  return sdiag_of(up, lo, cd);
}

template <typename T, int NC, bool DOADD>
__global__ void __launch_bounds__(PTX * NWARP, 4)
rhs_kernel(int n, T inv_h, T visc, const T* __restrict__ u, T* __restrict__ du, SlotBatch sb, int zblocks, int ptz,
           const __grid_constant__ CUtensorMap umap, int have_map) {
  chain_wait();
  constexpr int PTY = PTYT<NC>, PBY = PBYT<NC>;
  constexpr int CSTRIDE = (int)(sizeof(CompPlane<T, NC>) / sizeof(T));
  extern __shared__ __align__(128) unsigned char rhs_smem[];
  PlaneSmem<T, NC>& sm =
      *reinterpret_cast<PlaneSmem<T, NC>*>(rhs_smem + ((128u - (smem_u32(rhs_smem) & 127u)) & 127u));
  const long long N = (long long)n * n * n;
  // slot of a batch of same-size solves (serving form): blockIdx.z = slot * zblocks + zb
  const int slot = blockIdx.z / zblocks;
  const int zb = blockIdx.z - slot * zblocks;
  if (sb.active && !sb.active[slot]) return;
  u += slot * sb.ustride;
  du += slot * sb.ustride;
  if (sb.visc) visc = reinterpret_cast<const T*>(sb.visc)[slot];
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int lane = tx, warp = ty;
  const int x0 = blockIdx.x * PTX, y0 = blockIdx.y * PTY, z0 = zb * ptz;
  // stresses kept as 4 sigma (rv = 4 visc / h), the divergence takes 1/(4h)
  const T kd = (T)0.25 * inv_h;
  const T rv = (T)4 * visc * inv_h;
  const T cd = (T)2 * rv, co = rv;
  auto wrap = [n](int g) { return g < 0 ? g + n : (g >= n ? g - n : g); };
  auto wrapm = [n](int g) { return ((g % n) + n) % n; };
  const bool big = n >= PBX;
  // asynchronous copy of plane gz (with halo) into buffer buf; the caller
  // commits and waits (cp_async_wait_all) before the __syncthreads that
  // publishes it.  Full x tiles of a grid whose rows are 16-byte multiples
  // copy each box row as NV + 2 aligned 16-byte pieces: the interior, the
  // piece ending at x0 - 1 (left halo in its last word) and the piece starting
  // at x0 + PTX (right halo in its first word).  Each thread's pieces are the
  // same in every plane: their offsets are computed once, and a plane adds
  // gz n^2.  Other tiles copy word by word.
  constexpr int VE = 16 / (int)sizeof(T), NV = PTX / VE;
  constexpr int NPIECE = 3 * PBY * (NV + 2);
  constexpr int NSLOT = (NPIECE + PTX * NWARP - 1) / (PTX * NWARP);
  const bool vec = big && x0 + PTX <= n && (n % VE) == 0 && (reinterpret_cast<uintptr_t>(u) & 15) == 0;
  const int tid = ty * PTX + tx;
  long long goff[NSLOT];
  int soff[NSLOT];
  if (vec) {
#pragma unroll
    for (int i = 0; i < NSLOT; ++i) {
      const int t = tid + i * PTX * NWARP;
      goff[i] = -1;
      soff[i] = 0;
      if (t < NPIECE) {
        const int c = t / (PBY * (NV + 2));
        const int rem = t - c * (PBY * (NV + 2));
        const int rr = rem / (NV + 2), j = rem - rr * (NV + 2);
        const int gy = wrap(y0 - 1 + rr);
        const int gx = j < NV ? x0 + j * VE : (j == NV ? wrap(x0 - VE) : wrap(x0 + PTX));
        const int bx0 = j < NV ? SH<T> + 1 + j * VE : (j == NV ? 0 : SH<T> + 1 + PTX);
        goff[i] = c * N + (long long)gy * n + gx;
        soff[i] = c * CSTRIDE + rr * UROW<T> + bx0;
      }
    }
  }
  const long long nn = (long long)n * n;
  // full tiles whose box (x0 - VE .. x0 - VE + UROW - 1, y0 - 1 .. y0 + PTY)
  // lies inside the grid take each component plane as one TMA box, completed
  // on the buffer's mbarrier; the others use the cp.async pieces
  const bool tma = vec && have_map && x0 >= VE && x0 - VE + UROW<T> <= n && y0 >= 1 && y0 + PTY + 1 <= n;
  unsigned parity = 0;  // bit b: phase of buffer b's mbarrier to wait for
  const bool drill = tma && g_rhs_drill != 0;
  const int poll_limit = drill ? RHS_DRILL_POLLS : RHS_POLLS;
  if (tma) {
    if (tid == 0) {
#pragma unroll
      for (int b = 0; b < 3; ++b) mbar_init(&sm.bar[b], 1);
      asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncthreads();
  }
  auto load_plane = [&](int buf, int gz) {
    if (tma) {
      if (tid == 0 && !drill) {
        mbar_expect_tx(&sm.bar[buf], 3u * CompPlane<T, NC>::WORDS * sizeof(T));
#pragma unroll
        for (int c = 0; c < 3; ++c)
          tma_load_3d(&sm.u[buf][c].r[0][0], &umap, x0 - VE, y0 - 1, (slot * 3 + c) * n + gz, &sm.bar[buf]);
      }
      return;
    }
    if (vec) {
      T* const sb0 = &sm.u[buf][0].r[0][0];
      const T* const ub = u + gz * nn;
#pragma unroll
      for (int i = 0; i < NSLOT; ++i)
        if (goff[i] >= 0) cp_async_16(sb0 + soff[i], ub + goff[i]);
    } else {
      const long long pz = (long long)gz * n;
      for (int rr = ty; rr < PBY; rr += NWARP) {
        const int gy = big ? wrap(y0 - 1 + rr) : wrapm(y0 - 1 + rr);
        for (int bxx = tx; bxx < PBX; bxx += PTX) {
          const int gx = big ? wrap(x0 - 1 + bxx) : wrapm(x0 - 1 + bxx);
#pragma unroll
          for (int c = 0; c < 3; ++c)
            cp_async_word(&sm.u[buf][c][rr][bxx + SH<T>], u + c * N + (pz + gy) * n + gx);
        }
      }
    }
    cp_async_commit();
  };
  auto zwrap = [&](int z) { return big ? wrap(z) : wrapm(z); };
  const int bx = tx + 1;
  // prologue: planes z0-1 (buffer 0) and z0 (buffer 1) give s13, s23 of plane
  // z0-1 and s33 of plane z0 for this thread's cells
  // completion of the loads of buffer buf (its mbarrier phase, or every
  // cp.async of this thread); a TMA wait gives up after about 2^20 polls
  // (RHS_DRILL_POLLS in the wait drill), records the fault and goes on
  auto wait_plane = [&](int buf) {
    if (!tma) {
      cp_async_wait_all();
      return;
    }
    int polls = 0;
    while (!mbar_try_wait(&sm.bar[buf], (parity >> buf) & 1u)) {
      if (++polls > poll_limit) {
        if (tid == 0) atomicExch(&g_rhs_tma_fault, 1);
        break;
      }
    }
    parity ^= 1u << buf;
  };
  load_plane(0, zwrap(z0 - 1));
  load_plane(1, zwrap(z0));
  load_plane(2, zwrap(z0 + 1));
  wait_plane(0);
  wait_plane(1);
  wait_plane(2);
  __syncthreads();
  T s13_prev[NC], s23_prev[NC], s33_cur[NC];
#pragma unroll
  for (int i = 0; i < NC; ++i) {
    const int by = NC * ty + 1 + i;
    s13_prev[i] = s13<T>(sm.u[0], sm.u[1], bx, by, co);
    s23_prev[i] = s23<T>(sm.u[0], sm.u[1], bx, by, co);
    s33_cur[i] = s33<T>(sm.u[1][2][by][bx + SH<T>], sm.u[0][2][by][bx + SH<T>], cd);
  }
  __syncthreads();  // buffer 0 is refilled by the first prefetch
  // buffers: cur = plane z, nxt = plane z + 1, pre = the free one
  int cur = 1, nxt = 2, pre = 0;
  const int gx = x0 + tx;
  T* const du1 = du;
  T* const du2 = du + N;
  T* const du3 = du + 2 * N;
  for (int kz = 0; kz < ptz; ++kz) {
    const int z = z0 + kz;
    if (z >= n) break;  // uniform across the CTA
    // plane z + 2 streams into the free buffer while plane z is processed
    // (its last reader finished before the previous iteration's barrier)
    if (kz + 1 < ptz && z + 1 < n) load_plane(pre, zwrap(z + 2));
    const auto& uc = sm.u[cur];
    const auto& un = sm.u[nxt];
    // own-cell stresses
    T v11[NC], v22[NC], v12[NC], v13[NC], v23[NC], v33n[NC];
#pragma unroll
    for (int i = 0; i < NC; ++i) {
      const int by = NC * ty + 1 + i;
      v11[i] = sdiag<T, 0>(uc, bx, by, cd);
      v22[i] = sdiag<T, 1>(uc, bx, by, cd);
      v12[i] = s12<T>(uc, bx, by, co);
      v13[i] = s13<T>(uc, un, bx, by, co);
      v23[i] = s23<T>(uc, un, bx, by, co);
      v33n[i] = s33<T>(un[2][by][bx + SH<T>], uc[2][by][bx + SH<T>], cd);
      // s22 is read from the row above and s23 from the row below: inside a
      // thread's rows they stay in registers
      sm.s[0][by][bx] = v11[i];
      if (i == 0) sm.s[1][by][bx] = v22[i];
      sm.s[2][by][bx] = v12[i];
      sm.s[3][by][bx] = v13[i];
      if (i == NC - 1) sm.s[4][by][bx] = v23[i];
    }
    // halo stresses, one task per warp: s12, s23 on the lower halo row, s22
    // on the upper halo row, s12 and s13 on the left halo column, s11 on the
    // right halo column
    if (warp == 0) {
      sm.s[2][0][lane + 1] = s12<T>(uc, lane + 1, 0, co);
    } else if (warp == 1) {
      sm.s[4][0][lane + 1] = s23<T>(uc, un, lane + 1, 0, co);
    } else if (warp == 2) {
      sm.s[1][PTY + 1][lane + 1] = sdiag<T, 1>(uc, lane + 1, PTY + 1, cd);
    } else if (warp == 3) {
      for (int r = lane; r <= PTY; r += 32) sm.s[2][r][0] = s12<T>(uc, 0, r, co);
    } else if (warp == 4) {
      for (int r = lane + 1; r <= PTY; r += 32) sm.s[3][r][0] = s13<T>(uc, un, 0, r, co);
    } else if (warp == 5) {
      for (int r = lane + 1; r <= PTY; r += 32) sm.s[0][r][PTX + 1] = sdiag<T, 0>(uc, PTX + 1, r, cd);
    }
    __syncthreads();
    if (gx < n) {
      const auto& S = sm.s;
#pragma unroll
      for (int i = 0; i < NC; ++i) {
        const int by = NC * ty + 1 + i;
        const int gy = y0 + by - 1;
        if (gy < n) {
          // a thread's cells are consecutive rows: the stresses of the row
          // below and above come from registers where the thread owns them
          const T s12_below = i > 0 ? v12[i > 0 ? i - 1 : 0] : S[2][by - 1][bx];
          const T s22_above = i < NC - 1 ? v22[i < NC - 1 ? i + 1 : 0] : S[1][by + 1][bx];
          const T s23_below = i > 0 ? v23[i > 0 ? i - 1 : 0] : S[4][by - 1][bx];
          const T d1 = (S[0][by][bx + 1] - v11[i]) + (v12[i] - s12_below) + (v13[i] - s13_prev[i]);
          const T d2 = (v12[i] - S[2][by][bx - 1]) + (s22_above - v22[i]) + (v23[i] - s23_prev[i]);
          const T d3 = (v13[i] - S[3][by][bx - 1]) + (v23[i] - s23_below) + (v33n[i] - s33_cur[i]);
          const long long g = ((long long)z * n + gy) * n + gx;
          if (DOADD) {
            du1[g] -= kd * d1;
            du2[g] -= kd * d2;
            du3[g] -= kd * d3;
          } else {
            du1[g] = -kd * d1;
            du2[g] = -kd * d2;
            du3[g] = -kd * d3;
          }
        }
        s13_prev[i] = v13[i];
        s23_prev[i] = v23[i];
        s33_cur[i] = v33n[i];
      }
    }
    if (kz + 1 < ptz && z + 1 < n) wait_plane(pre);
    __syncthreads();
    const int freed = cur;
    cur = nxt;
    nxt = pre;
    pre = freed;
  }
}

// ---------------------------------------------------------------------------
// FP64 sweep on the integer pipe.
//
// The FP64 pipe bounds the sweep, so it forms the stresses and their divergence
// in fixed point (fixed.cuh), with more bits than FP64 carries, and rounds once
// at the end.
//
// Fixed point.  All values a CTA holds share one scale 2^(57 - E), |u| + |S| <
// 2^E: a velocity becomes an integer U, |U| <= 2^57, split as U = h 2^29 + l
// with h and l int32 and l in [-2^28, 2^28].  A double whose exponent is within
// five of the largest value's converts exactly; smaller ones round to 2^-58
// of the scale.  E follows the planes: it is the exponent of the largest
// value of the three planes held plus one, kept while the next plane fits and
// is not much smaller, else the planes are loaded and converted again.  Every
// `block` planes of the grid it starts afresh, so that a cell's bits depend on
// the field alone: a launch gives each CTA one block or several.
//
// Arithmetic.  With S = 2 visc/h (an integer in the same scale), A = u_i +
// u_i(+e_j) - 2S, B = u_j + u_j(+e_i) - 2S,
//   4 sigma_ij = A B + 4S (u_i + u_j) + const,
//   4 sigma_ii = (u_i + u_i(-e_i) - 2S)^2 + 8S u_i(-e_i) + const
// (the shifted stress form, constants cancel in the divergence), so
//   -4h du_i = D_i S_i + sum_{j != i} [A B - (A B)(-e_j)]
//              + 4S [sum_j (u_i - u_i(-e_j)) + sum_j (u_j - u_j(-e_j))],
//   D_i = u_i(+e_i) - u_i(-e_i),  S_i = u_i(+e_i) + 2 u_i + u_i(-e_i) - 4S.
// Products of (h, l) pairs accumulate in three int64 sums of weight 2^58,
// 2^29 and 1 -- the addition is part of the multiply-add, no carries travel --
// and the bounds above keep every sum below 2^63:
//   in weight 2^29, the largest of the three, the four A B give at most 3 2^60
//   (|A.h| <= 2^29, |A.l| <= 3 2^28), D_i S_i 1.2 2^60 and the three groups of
//   the linear term 1.5 2^60 (4S < 2^57): 5.7 2^60 in all.
// The sum is exact to 2^-85 of the squared scale, converted to a double with
// one rounding and multiplied by -1/(4h).
//
// What remains is the rounding of the inputs to 2^-58 of the scale.  The FP64
// operations it replaces round products of sums of u_i and S, so a component's
// error goes with max(|u_i|, S) there and with the scale here: relative L2 of
// the third component, white noise with that component 2^-k of the others, S
// below it, FP64 form 2.2-2.9e-16 throughout:
//   k = 0: 0.9e-16   3: 1.3e-16   4: 2.2e-16   5: 4.0e-16   7: 1.5e-15   10: 1e-14
// So a component that is not zero and with S below 2^-FX_WEAK of the scale
// in the three planes takes rhs_cell_f64.  S would be rounded with them, or the
// velocity with a larger S: where |S| is below 2^-FX_SMALL_S of the velocities'
// scale or above half of it, it stays out of the integers, and the linear term is
// summed by itself, exactly, and multiplied by S in FP64 (a shear flow u_1(y),
// whose advection vanishes, is nothing else: ten cells of noise at visc 1e-5
// 2.9e-14 with S rounded, FP64 form 1.8e-16).
// The cells whose velocity is below 2^-7 of the tile's largest take rhs_cell_f64
// too (their error is below the larger cells' in any norm over the tile), and
// planes with values that are not finite or out of range.
//
// Per cell 650 instructions, 88 of them the multiply-adds, 57 shared-memory
// accesses per 32 cells and 6 FP64 operations (45 before).  512^3: 11.4 -> 3.64
// ms (HBM floor 0.95), 250^3 1470 -> 518 us, 128^3 215 -> 85, 90^3 102 -> 46,
// 32^3 47 -> 14; with the linear term by itself 4.14 ms, 579, 93, 48 and 15 us; with
// a third component weak everywhere 11.2 ms, 1560, 236, 108 and 20 (its cells share
// nothing).  Bound by the latency of the multiply-add pipe (66% busy) at 8
// warps per scheduler.  Error against 113-bit arithmetic, relative L2: white
// noise 0.7-1.1e-16 (FP64 form 1.7-2.1e-16), smooth fields 0.8e-16 (1.2e-15), a
// mean flow of 100 7e-17 (1.3e-14), visc 0.1 1.4e-16 (7.7e-16).
// ---------------------------------------------------------------------------
constexpr int FX_BITS = 57, FX_LOW = 29;
// E of the fixed-point path: well inside the range of the FP32 bound that
// finds it, and squares and their scaling stay normal doubles
constexpr int FX_EMIN = -100, FX_EMAX = FX_BITS;
constexpr int FX_WEAK = 4, FX_SMALL_S = 6;

// Component I of one cell in FP64, from global memory: what the fixed-point sweep
// leaves out.  WEAK: a weak component, whose S is small beside the velocities: the
// products as differences of sums and the viscous term of the sums at hand (31 FP64
// operations); else the reference's arithmetic (42).
template <int I, bool WEAK>
__device__ __noinline__ double rhs_cell_f64(const double* __restrict__ u, int n, int x, int y, int z, double inv_h,
                                            double visc) {
  constexpr int J = I == 0 ? 1 : 0, K = I == 2 ? 1 : 2;
  const long long N = (long long)n * n * n;
  const int at[3] = {x, y, z};
  const long long step[3] = {1, n, (long long)n * n};
  auto up = [&](int d) { return at[d] + 1 == n ? (1 - n) * step[d] : step[d]; };
  auto dn = [&](int d) { return at[d] == 0 ? (n - 1) * step[d] : -step[d]; };
  const double* const p = u + I * N + z * step[2] + y * step[1] + x;
  const double *const q = p + (J - I) * N, *const r = p + (K - I) * N;
  const long long iu = up(I), id = dn(I), ju = up(J), jd = dn(J), ku = up(K), kd = dn(K);
  // all loads first: they are independent
  const double p0 = p[0], piu = p[iu], pid = p[id], pju = p[ju], pjd = p[jd], pku = p[ku], pkd = p[kd];
  const double q0 = q[0], qiu = q[iu], qjd = q[jd], qjdiu = q[jd + iu];
  const double r0 = r[0], riu = r[iu], rkd = r[kd], rkdiu = r[kd + iu];
  double sum;
  if constexpr (WEAK) {
    const double t = fma(2.0, p0, piu + pid), aj = p0 + pju, bj = p0 + pjd, ak = p0 + pku, bk = p0 + pkd;
    sum = (piu - pid) * t;
    sum = fma(aj, q0 + qiu, sum);
    sum = fma(-bj, qjd + qjdiu, sum);
    sum = fma(ak, r0 + riu, sum);
    sum = fma(-bk, rkd + rkdiu, sum);
    const double lin = fma(-16.0, p0, fma(2.0, t, (aj + bj) + (ak + bk))) + ((qiu - q0) - (qjdiu - qjd)) +
                       ((riu - r0) - (rkdiu - rkd));
    sum = fma(-4.0 * visc * inv_h, lin, sum);
  } else {
    const double rv = 4.0 * visc * inv_h;
    auto diag = [rv](double a, double b) { return (a + b) * (a + b) - 2.0 * rv * (a - b); };
    auto off = [rv](double a, double b, double c, double d) { return (a + b) * (c + d) - rv * ((b - a) + (d - c)); };
    const double di = diag(piu, p0) - diag(p0, pid);
    const double dj = off(p0, pju, q0, qiu) - off(pjd, p0, qjd, qjdiu);
    const double dk = off(p0, pku, r0, riu) - off(pkd, p0, rkd, rkdiu);
    sum = I == 2 ? (dj + dk) + di : (di + dj) + dk;
  }
  return -0.25 * inv_h * sum;
}

// Tile of the fixed-point sweep: 32 x 16 cells, FXC rows per thread, FX_CTAS
// CTAs per SM (64 registers).  512^3 / 250^3 / 128^3 / 32^3, before the weak
// components and the viscous term had paths of their own: 3.43 ms / 488 / 78
// / 10 us; three CTAs (80 registers) 3.75 / 497 / 84 / 10; one row per thread 5.3
// ms / 701 / 108 / 10 (every shared value loaded once per cell); four rows, five
// CTAs 3.27 ms / 462 / 88 / 12: the larger tile of work per thread loses on the
// LES grids and on 128^3.
constexpr int FXC = 2, FX_CTAS = 4, FXY = 16, FXW = FXY / FXC, FXBY = FXY + 2, FXROW = 36;  // box rows and words per row
constexpr int FXPIECES = 3 * FXBY * FXROW / 2;                                      // 16-byte pieces of a plane
constexpr int FXTHREADS = PTX * FXW;

struct FixedSmem {
  // plane buffers: the box of each component, row after row (one 4-D TMA box),
  // x = x0 - 2 first; doubles on arrival, then Fx pairs
  double u[3][3 * FXBY * FXROW + 8];
  unsigned piece[FXPIECES];      // word offset in the field of each 16-byte piece of a plane
  unsigned red[3][3][FXW];       // largest magnitude (high word) per plane buffer, component and warp
  unsigned long long bar[3];     // TMA completion of each plane buffer
  double by_s;                   // factor of the linear term of a small S
};
static_assert(sizeof(FixedSmem::u[0]) % 128 == 0, "TMA destinations");
constexpr size_t FIXED_SMEM = sizeof(FixedSmem) + 128;

template <bool DOADD>
__global__ void __launch_bounds__(FXTHREADS, FX_CTAS)
rhs_fixed_kernel(int n, double inv_h, double visc, const double* __restrict__ u, double* __restrict__ du, SlotBatch sb,
                 int zblocks, int ptz, int block, const __grid_constant__ CUtensorMap umap, int have_map) {
  chain_wait();
  using T = double;
  constexpr int NC = FXC;
  extern __shared__ __align__(128) unsigned char rhs_smem[];
  FixedSmem& sm = *reinterpret_cast<FixedSmem*>(rhs_smem + ((128u - (smem_u32(rhs_smem) & 127u)) & 127u));
  const long long N = (long long)n * n * n, nn = (long long)n * n;
  const int slot = blockIdx.z / zblocks;
  const int zb = blockIdx.z - slot * zblocks;
  if (sb.active && !sb.active[slot]) return;
  u += slot * sb.ustride;
  du += slot * sb.ustride;
  if (sb.visc) visc = reinterpret_cast<const T*>(sb.visc)[slot];
  const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * PTX + tx;
  const int x0 = blockIdx.x * PTX, y0 = blockIdx.y * FXY, z0 = zb * ptz;
  auto wrapm = [n](int g) { return ((g % n) + n) % n; };
  // plane copies: one TMA box where the box lies inside the grid, else 16-byte
  // pieces (n is even, so a piece never straddles the periodic boundary), or
  // words when the field is not 16-byte aligned
  const bool vec = (reinterpret_cast<uintptr_t>(u) & 15) == 0;
  const bool tma = vec && have_map && x0 >= 2 && x0 - 2 + FXROW <= n && y0 >= 1 && y0 + FXY + 1 <= n;
  unsigned parity = 0;
  const bool drill = tma && g_rhs_drill != 0;
  const int poll_limit = drill ? RHS_DRILL_POLLS : RHS_POLLS;
  if (tma) {
    if (tid == 0) {
#pragma unroll
      for (int b = 0; b < 3; ++b) mbar_init(&sm.bar[b], 1);
      asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
  } else {
    for (int t = tid; t < FXPIECES; t += FXTHREADS) {
      const int c = t / (FXBY * FXROW / 2), rem = t - c * (FXBY * FXROW / 2);
      const int rr = rem / (FXROW / 2), j = rem - rr * (FXROW / 2);
      // 3 n^3 <= 3 2^30 words: an unsigned offset
      sm.piece[t] = (unsigned)(c * N) + (unsigned)wrapm(y0 - 1 + rr) * n + wrapm(x0 - 2 + 2 * j);
    }
  }
  __syncthreads();
  constexpr int NSLOT = (FXPIECES + FXTHREADS - 1) / FXTHREADS;
  auto load_plane = [&](int buf, int gz) {
    if (tma) {
      if (tid == 0 && !drill) {
        mbar_expect_tx(&sm.bar[buf], 3u * FXBY * FXROW * sizeof(T));
        tma_load_4d(sm.u[buf], &umap, x0 - 2, y0 - 1, gz, 3 * slot, &sm.bar[buf]);
      }
      return;
    }
    const T* const ub = u + gz * nn;
#pragma unroll
    for (int i = 0; i < NSLOT; ++i) {
      const int t = tid + i * FXTHREADS;
      if (t < FXPIECES) {
        T* const d = sm.u[buf] + 2 * t;
        const T* const g = ub + sm.piece[t];
        if (vec) {
          cp_async_16(d, g);
        } else {
          cp_async_word(d, g);
          cp_async_word(d + 1, g + 1);
        }
      }
    }
    cp_async_commit();
  };
  auto wait_plane = [&](int buf) {
    if (!tma) {
      cp_async_wait_all();
      return;
    }
    int polls = 0;
    while (!mbar_try_wait(&sm.bar[buf], (parity >> buf) & 1u)) {
      if (++polls > poll_limit) {
        if (tid == 0) atomicExch(&g_rhs_tma_fault, 1);
        break;
      }
    }
    parity ^= 1u << buf;
  };
  // f(piece) over this thread's pieces of plane buffer buf, after its wait (a
  // TMA plane's mbarrier wait makes every copy visible, else it copied them)
  auto each_piece = [&](int buf, auto f) {
#pragma unroll
    for (int i = 0; i < NSLOT; ++i) {
      const int t = tid + i * FXTHREADS;
      if (t < FXPIECES) f(reinterpret_cast<double2*>(sm.u[buf])[t]);
    }
  };
  // largest magnitude of each component of a plane (high words), this warp's
  // part, into sm.red: of the pieces it copied itself, which it may read before the
  // barrier; the plane is only read
  auto scan_plane = [&](int buf) {
    constexpr int PC = FXPIECES / 3;  // pieces of a component
    unsigned m[3] = {0, 0, 0};
#pragma unroll
    for (int i = 0; i < NSLOT; ++i) {
      const int t = tid + i * FXTHREADS;
      if (t < FXPIECES) {
        const double2 v = reinterpret_cast<const double2*>(sm.u[buf])[t];
        const unsigned q = max((unsigned)__double2hiint(v.x) & 0x7fffffffu, (unsigned)__double2hiint(v.y) & 0x7fffffffu);
#pragma unroll
        for (int c = 0; c < 3; ++c)  // the components that slot i of any thread reaches
          if (c * PC < (i + 1) * FXTHREADS && (c + 1) * PC > i * FXTHREADS)
            m[c] = max(m[c], t >= c * PC && t < (c + 1) * PC ? q : 0u);
      }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      m[c] = __reduce_max_sync(0xffffffffu, m[c]);
      if (tx == 0) sm.red[buf][c][ty] = m[c];
    }
  };
  static_assert(3 * FXW <= 32, "a lane per warp and plane");
  // a component's largest magnitude in the three planes held
  auto held_max = [&](int c) {
    return __reduce_max_sync(0xffffffffu, tx < 3 * FXW ? sm.red[tx / FXW][c][tx % FXW] : 0u);
  };
  int E = 0;                     // |u| + S < 2^E for the planes held
  int kexp = 0;                  // (57 - E) << 20
  double scale = 0;              // -1/(4h) 2^58 in fixed-point units squared
  auto convert_plane = [&](int buf) {
    each_piece(buf, [&](double2& v) {
      const Fx q = fx_from_double<FX_BITS, FX_LOW>(v.x, kexp), r = fx_from_double<FX_BITS, FX_LOW>(v.y, kexp);
      v = make_double2(__hiloint2double(q.h, q.l), __hiloint2double(r.h, r.l));
    });
  };
  Fx S2{}, S4{};  // 2S and 4S in fixed point
  int tiny = 0;   // cells whose h words are all below this take the FP64 path
  int weak = 0;   // bits 0-2: components that take it in every cell of the plane
  bool s_out = false;  // S is not among the integers
  unsigned below = 0;  // high word of 2^(E - FX_WEAK), 0 where S is above that
  bool slow = false;
  // |S| in FP32, whose range covers the fixed-point path's, rounded up (a
  // negative viscosity is taken)
  float Sf = 2.0 * fabs(visc) * inv_h < 1e30 ? __double2float_ru(2.0 * fabs(visc) * inv_h) : 1e30f;
  asm volatile("" : "+f"(Sf));  // kept, not recomputed on the FP64 pipe
  // E for planes whose largest magnitude has high word mx, bounds rounded up:
  // above |u|, with S among the integers above |u| + |S| and 4|S|
  auto exponent_for = [&](unsigned mx, bool out) {
    if (mx == 0) return FX_EMIN;
    const float m = __uint_as_float(mx < 0x39000000u ? 0u : mx >= 0x47000000u ? 0x7f000000u : ((mx - 0x38000000u) << 3) + 8u);
    const float bound = out ? m : fmaxf(__fadd_ru(m, Sf), 4.0f * Sf);
    return (int)(__float_as_uint(bound) >> 23) - 126;
  };
  // and whether S stays out of them, for planes taken afresh
  auto fresh = [&](unsigned mx, bool& out) {
    const int e = exponent_for(mx, true);
    // |u| < 2^e: S above 2^(e - 1), which may be above |u|, or far below
    out = Sf > __int_as_float((e + 126) << 23) || Sf < __int_as_float((e - FX_SMALL_S + 127) << 23);
    return out ? e : exponent_for(mx, false);
  };
  auto fxat = [&](int buf, int c, int row, int col) {
    const double v = sm.u[buf][(c * FXBY + row) * FXROW + col];
    return Fx{__double2hiint(v), __double2loint(v)};
  };
  // what the maxima m of the three planes held send to the FP64 path
  auto choose = [&](const unsigned (&m)[3]) {
    // 2^-7 of the top of the largest magnitude's binade, in units of h (the
    // FP64 path at 2^-5 costs 250^3 27% of its time, at 2^-7 nothing)
    const unsigned top = max(m[0], max(m[1], m[2]));
    const int q = FX_BITS - FX_LOW - 7 - (E - (int)((top >> 20) & 0x7ff) + 1022);
    tiny = top == 0 ? 0 : q < 0 ? 0 : 1 << q;
    weak = 0;
#pragma unroll
    for (int c = 0; c < 3; ++c) weak |= m[c] != 0 && m[c] < below ? 1 << c : 0;
  };
  // -4h du's linear term in units of S and of the velocity: its three groups, D
  // and the two pair sums A + B - (A + B)(-e_j) without S; at most 48 2^57
  auto linear = [](Fx g1, Fx g2, Fx g3, Fx d, Fx p, Fx q) {
    auto word = [](Fx v) { return (long long)v.h * (1 << FX_LOW) + v.l; };
    return (double)(4 * (word(g1) + word(g2) + word(g3) - word(d)) - 2 * (word(p) + word(q)));
  };
  const int col = tx + 2;
  // previous plane at this thread's cells: the velocities and B of s13, s23
  Fx pw1[NC], pw2[NC], pw3[NC], pb13[NC], pb23[NC];
  auto keep = [&](int buf) {
#pragma unroll
    for (int i = 0; i < NC; ++i) {
      const int r = NC * ty + 1 + i;
      pw1[i] = fxat(buf, 0, r, col);
      pw2[i] = fxat(buf, 1, r, col);
      pw3[i] = fxat(buf, 2, r, col);
      pb13[i] = pw3[i] + fxat(buf, 2, r, col + 1) - S2;
      pb23[i] = pw3[i] + fxat(buf, 2, r + 1, col) - S2;
    }
  };
  // planes z - 1, z, z + 1 into buffers 0, 1, 2, the scale for them, and the
  // previous plane's values
  int cur = 1, nxt = 2, pre = 0;
  auto start = [&](int z) {
    load_plane(0, wrapm(z - 1));
    load_plane(1, wrapm(z));
    load_plane(2, wrapm(z + 1));
#pragma unroll 1
    for (int b = 0; b < 3; ++b) wait_plane(b);
#pragma unroll 1
    for (int b = 0; b < 3; ++b) scan_plane(b);
    __syncthreads();
    const unsigned m[3] = {held_max(0), held_max(1), held_max(2)};
    const unsigned mx = max(m[0], max(m[1], m[2]));
    const double S = 2.0 * visc * inv_h;
    E = fresh(mx, s_out);
    weak = 0;
    slow = mx >= 0x7fe00000u || !(fabs(S) < 1e300) || E > FX_EMAX || E < FX_EMIN;
    if (!slow) {
      kexp = (FX_BITS - E) << 20;
      scale = ldexp(-0.25 * inv_h, 2 * FX_LOW + 2 * (E - FX_BITS));
      if (s_out && tid == 0) sm.by_s = ldexp(-0.25 * inv_h * S, E - FX_BITS);
      const Fx s = s_out ? Fx{0, 0} : fx_from_double<FX_BITS, FX_LOW>(4.0 * S, kexp);
      // 4S to a multiple of four units, so that S and 2S are the same S
      const long long s4 = (((long long)s.h << FX_LOW) + s.l + 2) >> 2 << 2;
      const long long s2 = s4 >> 1;
      S4 = {(int)((s4 + (1 << (FX_LOW - 1))) >> FX_LOW), 0};
      S4.l = (int)(s4 - ((long long)S4.h << FX_LOW));
      S2 = {(int)((s2 + (1 << (FX_LOW - 1))) >> FX_LOW), 0};
      S2.l = (int)(s2 - ((long long)S2.h << FX_LOW));
      below = Sf < __int_as_float((E - FX_WEAK + 127) << 23) ? (unsigned)(E - FX_WEAK + 1023) << 20 : 0u;
      choose(m);
#pragma unroll 1
      for (int b = 0; b < 3; ++b) convert_plane(b);
    }
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    __syncthreads();
    if (!slow) keep(0);
    __syncthreads();  // buffer 0 is refilled by the first prefetch
    cur = 1;
    nxt = 2;
    pre = 0;
  };
  // The planes from another one on.  sm.red and the plane buffers belong to every
  // warp until the last one has read this plane's values and maxima, and what was
  // written to the buffers is ordered before the copies that come next.
  auto restart = [&](int z) {
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    __syncthreads();
    start(z);
  };
  start(z0);
  int walked = 0;  // planes of the block behind
  const int gx = x0 + tx;
  for (int kz = 0; kz < ptz; ++kz) {
    const int z = z0 + kz;
    if (z >= n) break;  // uniform across the CTA
    const bool more = kz + 1 < ptz && z + 1 < n;
    if (more && !slow) load_plane(pre, wrapm(z + 2));
    auto cells = [&](auto s_outside) {
      constexpr bool S_OUT = decltype(s_outside)::value;
      const Fx s2 = S_OUT ? Fx{0, 0} : S2, s4 = S_OUT ? Fx{0, 0} : S4;
#pragma unroll
      for (int i = 0; i < NC; ++i) {
        const int r = NC * ty + 1 + i, gy = y0 + NC * ty + i;
        const Fx a = fxat(cur, 0, r, col), b = fxat(cur, 1, r, col), c = fxat(cur, 2, r, col);
        double o1 = 0, o2 = 0, o3 = 0;
        const bool direct = slow || max(abs(a.h), max(abs(b.h), abs(c.h))) < tiny;
        if (!slow) {
          // u1: neighbours along x, y, z and (-x, +y), (-x, +z)
          const Fx axp = fxat(cur, 0, r, col + 1), axm = fxat(cur, 0, r, col - 1);
          const Fx ayp = fxat(cur, 0, r + 1, col), aym = fxat(cur, 0, r - 1, col);
          const Fx axmyp = fxat(cur, 0, r + 1, col - 1);
          const Fx azp = fxat(nxt, 0, r, col), axmzp = fxat(nxt, 0, r, col - 1);
          // u2: along x, y, z and (+x, -y), (-y, +z)
          const Fx bxp = fxat(cur, 1, r, col + 1), bxm = fxat(cur, 1, r, col - 1);
          const Fx byp = fxat(cur, 1, r + 1, col), bym = fxat(cur, 1, r - 1, col);
          const Fx bxpym = fxat(cur, 1, r - 1, col + 1);
          const Fx bzp = fxat(nxt, 1, r, col), bymzp = fxat(nxt, 1, r - 1, col);
          // u3: along x, y, z
          const Fx cxp = fxat(cur, 2, r, col + 1), cxm = fxat(cur, 2, r, col - 1);
          const Fx cyp = fxat(cur, 2, r + 1, col), cym = fxat(cur, 2, r - 1, col);
          const Fx czp = fxat(nxt, 2, r, col);
          // the linear term's group common to the components
          FxSum s0{0, 0, 0};
          fx_mac(s0, (a - axm) + (b - bym), s4);
          const Fx dz3 = c - pw3[i];
          const Fx A12 = a + ayp - s2, B12 = b + bxp - s2;
          const Fx A13 = a + azp - s2, B13 = c + cxp - s2;
          const Fx A23 = b + bzp - s2, B23 = c + cyp - s2;
          if (!S_OUT || !(weak & 1)) {
            FxSum s = s0;
            fx_mac(s, dz3 + (a - axm), s4);
            fx_mac(s, (a - aym) + (a - pw1[i]), s4);
            fx_mac(s, axp - axm, (axp + axm) + (a + a) - s4);
            fx_mac(s, A12, B12);
            fx_mac(s, s2 - a - aym, bym + bxpym - s2);
            fx_mac(s, A13, B13);
            fx_mac(s, s2 - a - pw1[i], pb13[i]);
            o1 = fx_to_double<FX_LOW>(s, scale);
            if constexpr (S_OUT)
              o1 = fma(sm.by_s, linear((a - axm) + (b - bym), dz3 + (a - axm), (a - aym) + (a - pw1[i]), axp - axm,
                       (ayp - aym) + (b + bxp) - (bym + bxpym), (azp - pw1[i]) + (c + cxp) - (pb13[i] + s2)), o1);
          }
          if (!S_OUT || !(weak & 2)) {
            FxSum s = s0;
            fx_mac(s, dz3 + (b - bxm), s4);
            fx_mac(s, (b - bym) + (b - pw2[i]), s4);
            fx_mac(s, byp - bym, (byp + bym) + (b + b) - s4);
            fx_mac(s, A12, B12);
            fx_mac(s, s2 - axm - axmyp, bxm + b - s2);
            fx_mac(s, A23, B23);
            fx_mac(s, s2 - b - pw2[i], pb23[i]);
            o2 = fx_to_double<FX_LOW>(s, scale);
            if constexpr (S_OUT)
              o2 = fma(sm.by_s, linear((a - axm) + (b - bym), dz3 + (b - bxm), (b - bym) + (b - pw2[i]), byp - bym,
                       (a + ayp) - (axm + axmyp) + (bxp - bxm), (bzp - pw2[i]) + (c + cyp) - (pb23[i] + s2)), o2);
          }
          if (!S_OUT || !(weak & 4)) {
            FxSum s = s0;
            fx_mac(s, dz3 + (c - cxm), s4);
            fx_mac(s, (c - cym) + dz3, s4);
            fx_mac(s, czp - pw3[i], (czp + pw3[i]) + (c + c) - s4);
            fx_mac(s, A13, B13);
            fx_mac(s, s2 - axm - axmzp, cxm + c - s2);
            fx_mac(s, A23, B23);
            fx_mac(s, s2 - bym - bymzp, cym + c - s2);
            o3 = fx_to_double<FX_LOW>(s, scale);
            if constexpr (S_OUT)
              o3 = fma(sm.by_s, linear((a - axm) + (b - bym), dz3 + (c - cxm), (c - cym) + dz3, czp - pw3[i],
                       (a + azp) - (axm + axmzp) + (cxp - cxm), (b + bzp) - (bym + bymzp) + (cyp - cym)), o3);
          }
          pw1[i] = a;
          pw2[i] = b;
          pw3[i] = c;
          pb13[i] = B13;
          pb23[i] = B23;
        }
        if (gx < n && gy < n) {
          if (weak & 1) o1 = rhs_cell_f64<0, true>(u, n, gx, gy, z, inv_h, visc);
          if (weak & 2) o2 = rhs_cell_f64<1, true>(u, n, gx, gy, z, inv_h, visc);
          if (weak & 4) o3 = rhs_cell_f64<2, true>(u, n, gx, gy, z, inv_h, visc);
          if (direct) {
            o1 = rhs_cell_f64<0, false>(u, n, gx, gy, z, inv_h, visc);
            o2 = rhs_cell_f64<1, false>(u, n, gx, gy, z, inv_h, visc);
            o3 = rhs_cell_f64<2, false>(u, n, gx, gy, z, inv_h, visc);
          }
          double* const d = du + ((long long)z * n + gy) * n + gx;
          if (DOADD) {
            d[0] += o1;
            d[N] += o2;
            d[2 * N] += o3;
          } else {
            d[0] = o1;
            d[N] = o2;
            d[2 * N] = o3;
          }
        }
      }
    };
    // two copies: the linear term by itself would cost the usual one registers
    if (s_out) cells(std::true_type());
    else cells(std::false_type());
    if (!more) break;
    if (slow) {
      if (++walked == block) walked = 0;
      restart(z + 1);
      continue;
    }
    wait_plane(pre);
    scan_plane(pre);
    __syncthreads();
    const unsigned m[3] = {held_max(0), held_max(1), held_max(2)};
    const unsigned mx = max(m[0], max(m[1], m[2]));
    const int En = exponent_for(mx, s_out);
    bool other = En > E || En < E - 2;
    if (++walked == block) {  // a block starts with its own scale
      bool out;
      walked = 0;
      other = fresh(mx, out) != E || out != s_out;
    }
    if (mx >= 0x7fe00000u || other) {
      restart(z + 1);
      continue;
    }
    choose(m);
    convert_plane(pre);
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    __syncthreads();
    const int freed = cur;
    cur = nxt;
    nxt = pre;
    pre = freed;
  }
}

// ---------------------------------------------------------------------------
// FP32 sweep with 2 x 2 cells per thread (64 x 16 tiles, the last ones ragged, of
// rows of 16-byte multiples): each thread reads its u rows as aligned float pairs, takes
// the x and y neighbour stresses of its own cells from registers and stores
// float pairs, which halves the shared-memory and global instructions per
// cell.  Same stress and divergence arithmetic, in the same order, as
// rhs_kernel: the results are bit-identical.
// ---------------------------------------------------------------------------
constexpr int QX = 64, QY = 16, QBX = QX + 2, QBY = QY + 2;
constexpr int QROW = 72;  // box x b at b + 3: left piece [0, 4), interior [4, 68), right piece [68, 72)
constexpr int QPLANE = QBY * QROW;                 // words of one component plane
constexpr int QCOMP = (QPLANE + 31) / 32 * 32;     // padded to 128 bytes (TMA destinations)

struct QuadComp {
  float r[QBY][QROW];
  float pad[QCOMP - QPLANE];
};
struct QuadSmem {
  QuadComp u[3][3];      // [plane buffer][component]
  float s[5][QBY][QBX];  // s11, s22, s12, s13, s23 of the current plane
  unsigned long long bar[3];  // TMA completion of each plane buffer
};
// dynamic shared memory of rhs_quad_kernel: the struct plus room to align it
// to 128 bytes
constexpr size_t QUAD_SMEM = sizeof(QuadSmem) + 128;



__device__ __forceinline__ float qdiag(float a, float b, float rv2) {
  const float s = a + b, d = a - b;
  return s * s - rv2 * d;
}
__device__ __forceinline__ float qoff(float a, float b, float c, float d, float rv) {
  return (a + b) * (c + d) - rv * ((b - a) + (d - c));
}

template <bool DOADD>
__global__ void __launch_bounds__(256, 3)
rhs_quad_kernel(int n, float inv_h, float visc, const float* __restrict__ u, float* __restrict__ du, SlotBatch sb,
                int zblocks, int ptz, const __grid_constant__ CUtensorMap umap, int have_map) {
  chain_wait();
  extern __shared__ __align__(128) unsigned char quad_smem[];
  QuadSmem& sm = *reinterpret_cast<QuadSmem*>(quad_smem + ((128u - (smem_u32(quad_smem) & 127u)) & 127u));
  const long long N = (long long)n * n * n;
  const int slot = blockIdx.z / zblocks;
  const int zb = blockIdx.z - slot * zblocks;
  if (sb.active && !sb.active[slot]) return;
  u += slot * sb.ustride;
  du += slot * sb.ustride;
  if (sb.visc) visc = reinterpret_cast<const float*>(sb.visc)[slot];
  const int tx = threadIdx.x, ty = threadIdx.y, lane = tx, warp = ty;
  const int x0 = blockIdx.x * QX, y0 = blockIdx.y * QY, z0 = zb * ptz;
  const float kd = 0.25f * inv_h, rv = 4.0f * visc * inv_h, rv2 = 2.0f * rv;  // 4 sigma kept, as above
  auto wrap = [n](int g) { return g < 0 ? g + n : (g >= n ? g - n : g); };
  // 16-byte copy pieces of a plane: 18 pieces per box row (left, 16 interior,
  // right), offsets computed once
  constexpr int NPQ = 3 * QBY * 18, NSQ = (NPQ + 255) / 256;
  const int tid = ty * 32 + tx;
  long long goff[NSQ];
  int soff[NSQ];
#pragma unroll
  for (int i = 0; i < NSQ; ++i) {
    const int t = tid + i * 256;
    goff[i] = -1;
    soff[i] = 0;
    if (t < NPQ) {
      const int c = t / (QBY * 18), rem = t - c * (QBY * 18);
      const int rr = rem / 18, j = rem - rr * 18;
      const int gy = wrap(y0 - 1 + rr);
      const int gx = wrap(x0 + 4 * (j - 1));
      goff[i] = c * N + (long long)gy * n + gx;
      soff[i] = c * QCOMP + rr * QROW + 4 * j;
    }
  }
  const long long nn = (long long)n * n;
  // tiles whose box (x0 - 4 .. x0 + 67, y0 - 1 .. y0 + 16) lies inside the
  // grid take each component plane as one TMA box, completed on the
  // buffer's mbarrier; the others (their halo wraps around the periodic
  // boundary) use the cp.async pieces
  const bool tma = have_map && x0 >= 4 && x0 + QX + 4 <= n && y0 >= 1 && y0 + QY + 1 <= n;
  unsigned parity = 0;  // bit b: phase of buffer b's mbarrier to wait for
  const bool drill = tma && g_rhs_drill != 0;
  const int poll_limit = drill ? RHS_DRILL_POLLS : RHS_POLLS;
  if (tma) {
    if (tid == 0) {
#pragma unroll
      for (int b = 0; b < 3; ++b) mbar_init(&sm.bar[b], 1);
      asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncthreads();
  }
  auto load_plane = [&](int buf, int gz) {
    if (tma) {
      if (tid == 0 && !drill) {
        mbar_expect_tx(&sm.bar[buf], 3u * QPLANE * sizeof(float));
#pragma unroll
        for (int c = 0; c < 3; ++c)
          tma_load_3d(&sm.u[buf][c].r[0][0], &umap, x0 - 4, y0 - 1, (slot * 3 + c) * n + gz, &sm.bar[buf]);
      }
      return;
    }
    float* const s0 = &sm.u[buf][0].r[0][0];
    const float* const ub = u + gz * nn;
#pragma unroll
    for (int i = 0; i < NSQ; ++i)
      if (goff[i] >= 0) cp_async_16(s0 + soff[i], ub + goff[i]);
    cp_async_commit();
  };
  // completion of the loads of buffer buf (its mbarrier phase, or every
  // cp.async of this thread); a TMA wait gives up after about 2^20 polls
  // (RHS_DRILL_POLLS in the wait drill), records the fault and goes on
  auto wait_plane = [&](int buf) {
    if (!tma) {
      cp_async_wait_all();
      return;
    }
    int polls = 0;
    while (!mbar_try_wait(&sm.bar[buf], (parity >> buf) & 1u)) {
      if (++polls > poll_limit) {
        if (tid == 0) atomicExch(&g_rhs_tma_fault, 1);
        break;
      }
    }
    parity ^= 1u << buf;
  };
  // this thread: box columns c0 = 2 tx + 1, c0 + 1 and rows r0 = 2 ty + 1, r0 + 1
  const int c0 = 2 * tx + 1, r0 = 2 * ty + 1;
  const int sc = c0 + 3;  // smem column of c0 (even: float2 aligned)
  auto f2 = [&](const float* row) { return *reinterpret_cast<const float2*>(row + sc); };
  load_plane(0, wrap(z0 - 1));
  load_plane(1, wrap(z0));
  load_plane(2, wrap(z0 + 1));
  wait_plane(0);
  wait_plane(1);
  wait_plane(2);
  __syncthreads();
  float p13[2][2], p23[2][2], p33[2][2];  // [row j][col i]
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const auto& ua = sm.u[0];  // plane z0 - 1
    const auto& ub = sm.u[1];  // plane z0
    const int r = r0 + j;
    const float2 a1 = f2(ua[0].r[r]), b1 = f2(ub[0].r[r]), a3 = f2(ua[2].r[r]), a2 = f2(ua[1].r[r]), b2 = f2(ub[1].r[r]);
    const float a3r = ua[2].r[r][sc + 2];
    const float2 a3u = f2(ua[2].r[r + 1]);
    const float2 b3 = f2(ub[2].r[r]);
    p13[j][0] = qoff(a1.x, b1.x, a3.x, a3.y, rv);
    p13[j][1] = qoff(a1.y, b1.y, a3.y, a3r, rv);
    p23[j][0] = qoff(a2.x, b2.x, a3.x, a3u.x, rv);
    p23[j][1] = qoff(a2.y, b2.y, a3.y, a3u.y, rv);
    p33[j][0] = qdiag(b3.x, a3.x, rv2);
    p33[j][1] = qdiag(b3.y, a3.y, rv2);
  }
  __syncthreads();  // buffer 0 is refilled by the first prefetch
  int cur = 1, nxt = 2, pre = 0;
  const int gx = x0 + 2 * tx, gy = y0 + 2 * ty;
  float* const du1 = du;
  float* const du2 = du + N;
  float* const du3 = du + 2 * N;
  for (int kz = 0; kz < ptz; ++kz) {
    const int z = z0 + kz;
    if (z >= n) break;  // uniform across the CTA
    if (kz + 1 < ptz && z + 1 < n) load_plane(pre, wrap(z + 2));
    const auto& uc = sm.u[cur];
    const auto& un = sm.u[nxt];
    // register patch: u1 rows r0, r0+1, r0+2 and column c0-1; u2 rows r0-1,
    // r0, r0+1 and column c0+2; u3 rows r0, r0+1, r0+2 and column c0+2; the
    // next plane's u1, u2, u3 on the thread's rows
    float2 u1r[3], u2r[3], u3r[3], u1n[2], u2n[2], u3n[2];
    float u1l[2], u2r2[2], u3r2[2];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      u1r[k] = f2(uc[0].r[r0 + k]);
      u2r[k] = f2(uc[1].r[r0 - 1 + k]);
      u3r[k] = f2(uc[2].r[r0 + k]);
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      u1l[j] = uc[0].r[r0 + j][sc - 1];
      u2r2[j] = uc[1].r[r0 + j][sc + 2];
      u3r2[j] = uc[2].r[r0 + j][sc + 2];
      u1n[j] = f2(un[0].r[r0 + j]);
      u2n[j] = f2(un[1].r[r0 + j]);
      u3n[j] = f2(un[2].r[r0 + j]);
    }
    float v11[2][2], v22[2][2], v12[2][2], v13[2][2], v23[2][2], v33[2][2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const float2 a1 = u1r[j], a1u = u1r[j + 1];
      const float2 a2 = u2r[j + 1], a2d = u2r[j];
      const float2 a3 = u3r[j], a3u = u3r[j + 1];
      v11[j][0] = qdiag(a1.x, u1l[j], rv2);
      v11[j][1] = qdiag(a1.y, a1.x, rv2);
      v22[j][0] = qdiag(a2.x, a2d.x, rv2);
      v22[j][1] = qdiag(a2.y, a2d.y, rv2);
      v12[j][0] = qoff(a1.x, a1u.x, a2.x, a2.y, rv);
      v12[j][1] = qoff(a1.y, a1u.y, a2.y, u2r2[j], rv);
      v13[j][0] = qoff(a1.x, u1n[j].x, a3.x, a3.y, rv);
      v13[j][1] = qoff(a1.y, u1n[j].y, a3.y, u3r2[j], rv);
      v23[j][0] = qoff(a2.x, u2n[j].x, a3.x, a3u.x, rv);
      v23[j][1] = qoff(a2.y, u2n[j].y, a3.y, a3u.y, rv);
      v33[j][0] = qdiag(u3n[j].x, a3.x, rv2);
      v33[j][1] = qdiag(u3n[j].y, a3.y, rv2);
    }
    // stresses other threads read: s11 of column c0 (left neighbour), s12 of
    // column c0+1 and of row r0+1 (right neighbour, row above), s13 of column
    // c0+1, s22 of row r0 (row below), s23 of row r0+1 (row above)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      sm.s[0][r0 + j][c0] = v11[j][0];
      sm.s[3][r0 + j][c0 + 1] = v13[j][1];
    }
    sm.s[2][r0][c0 + 1] = v12[0][1];
    sm.s[2][r0 + 1][c0] = v12[1][0];
    sm.s[2][r0 + 1][c0 + 1] = v12[1][1];
    sm.s[1][r0][c0] = v22[0][0];
    sm.s[1][r0][c0 + 1] = v22[0][1];
    sm.s[4][r0 + 1][c0] = v23[1][0];
    sm.s[4][r0 + 1][c0 + 1] = v23[1][1];
    // halo stresses, one task per warp (box row 0, row QY+1, column 0,
    // column QX+1)
    if (warp == 0) {
      for (int c = lane + 1; c <= QX; c += 32)
        sm.s[2][0][c] = qoff(uc[0].r[0][c + 3], uc[0].r[1][c + 3], uc[1].r[0][c + 3], uc[1].r[0][c + 4], rv);
    } else if (warp == 1) {
      for (int c = lane + 1; c <= QX; c += 32)
        sm.s[4][0][c] = qoff(uc[1].r[0][c + 3], un[1].r[0][c + 3], uc[2].r[0][c + 3], uc[2].r[1][c + 3], rv);
    } else if (warp == 2) {
      for (int c = lane + 1; c <= QX; c += 32)
        sm.s[1][QY + 1][c] = qdiag(uc[1].r[QY + 1][c + 3], uc[1].r[QY][c + 3], rv2);
    } else if (warp == 3) {
      if (lane <= QY) sm.s[2][lane][0] = qoff(uc[0].r[lane][3], uc[0].r[lane + 1][3], uc[1].r[lane][3], uc[1].r[lane][4], rv);
    } else if (warp == 4) {
      if (lane < QY) {
        const int r = lane + 1;
        sm.s[3][r][0] = qoff(uc[0].r[r][3], un[0].r[r][3], uc[2].r[r][3], uc[2].r[r][4], rv);
      }
    } else if (warp == 5) {
      if (lane < QY) {
        const int r = lane + 1;
        sm.s[0][r][QX + 1] = qdiag(uc[0].r[r][QX + 4], uc[0].r[r][QX + 3], rv2);
      }
    }
    __syncthreads();
    const auto& S = sm.s;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int r = r0 + j;
      float d1[2], d2[2], d3[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int c = c0 + i;
        const float s11_right = i == 0 ? v11[j][1] : S[0][r][c + 1];
        const float s12_below = j == 1 ? v12[0][i] : S[2][r - 1][c];
        const float s12_left = i == 1 ? v12[j][0] : S[2][r][c - 1];
        const float s22_above = j == 0 ? v22[1][i] : S[1][r + 1][c];
        const float s13_left = i == 1 ? v13[j][0] : S[3][r][c - 1];
        const float s23_below = j == 1 ? v23[0][i] : S[4][r - 1][c];
        d1[i] = (s11_right - v11[j][i]) + (v12[j][i] - s12_below) + (v13[j][i] - p13[j][i]);
        d2[i] = (v12[j][i] - s12_left) + (s22_above - v22[j][i]) + (v23[j][i] - p23[j][i]);
        d3[i] = (v13[j][i] - s13_left) + (v23[j][i] - s23_below) + (v33[j][i] - p33[j][i]);
        p13[j][i] = v13[j][i];
        p23[j][i] = v23[j][i];
        p33[j][i] = v33[j][i];
      }
      if (gx >= n || gy + j >= n) continue;  // outside a ragged tile's cells
      const long long g = ((long long)z * n + gy + j) * n + gx;
      float2* o1 = reinterpret_cast<float2*>(du1 + g);
      float2* o2 = reinterpret_cast<float2*>(du2 + g);
      float2* o3 = reinterpret_cast<float2*>(du3 + g);
      if (DOADD) {
        float2 a = *o1, b = *o2, c = *o3;
        a.x -= kd * d1[0]; a.y -= kd * d1[1];
        b.x -= kd * d2[0]; b.y -= kd * d2[1];
        c.x -= kd * d3[0]; c.y -= kd * d3[1];
        *o1 = a; *o2 = b; *o3 = c;
      } else {
        *o1 = make_float2(-kd * d1[0], -kd * d1[1]);
        *o2 = make_float2(-kd * d2[0], -kd * d2[1]);
        *o3 = make_float2(-kd * d3[0], -kd * d3[1]);
      }
    }
    if (kz + 1 < ptz && z + 1 < n) wait_plane(pre);
    __syncthreads();
    const int freed = cur;
    cur = nxt;
    nxt = pre;
    pre = freed;
  }
}

// Cells per thread along y: two (16-row tiles: the halo stresses are
// recomputed for fewer cells and adjacent rows share their u reads); four ran
// slower in FP32 (94 registers, two CTAs per SM).
template <typename T> constexpr int CYT = 2;

// The driver's tensor-map encoder, reached through the runtime (no link to
// the driver library); null when the driver does not provide it.
using TensorMapEncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                          const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                          CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                          CUtensorMapFloatOOBfill);
static TensorMapEncodeTiled tensor_map_encoder() {
  static std::once_flag once;
  static TensorMapEncodeTiled fn = nullptr;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<TensorMapEncodeTiled>(p);
  });
  return fn;
}

// Tiled tensor map, no interleave or swizzle, 128-byte L2 promotion, zero
// fill; false when the encoder is unavailable or rejects the arguments.
bool encode_tiled_map(CUtensorMap* map, CUtensorMapDataType dt, unsigned rank, const void* base,
                      const cuuint64_t* dims, const cuuint64_t* strides, const cuuint32_t* box) {
  std::memset(map, 0, sizeof(*map));
  TensorMapEncodeTiled enc = tensor_map_encoder();
  if (!enc) return false;
  cuuint32_t es[5] = {1, 1, 1, 1, 1};
  return enc(map, dt, rank, const_cast<void*>(base), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Tensor map of the vector fields of nslots solves as one 3-D tensor
// (x, y, (slot * 3 + component) * n + z) with boxes of bx x by x 1 words;
// false when it cannot be made (the sweep then copies with cp.async).
template <typename T>
static bool field_tensor_map(const T* u, int n, int nslots, const SlotBatch& sb, unsigned bx, unsigned by,
                             CUtensorMap* map) {
  std::memset(map, 0, sizeof(*map));
  const long long N = (long long)n * n * n;
  if (nslots > 1 && sb.ustride != 3 * N) return false;
  if ((reinterpret_cast<uintptr_t>(u) & 15) != 0 || (n * sizeof(T)) % 16 != 0) return false;
  TensorMapEncodeTiled enc = tensor_map_encoder();
  if (!enc) return false;
  const cuuint64_t dims[3] = {(cuuint64_t)n, (cuuint64_t)n, (cuuint64_t)nslots * 3 * n};
  const cuuint64_t strides[2] = {(cuuint64_t)n * sizeof(T), (cuuint64_t)n * n * sizeof(T)};
  const cuuint32_t box[3] = {bx, by, 1};
  const cuuint32_t es[3] = {1, 1, 1};
  return enc(map, sizeof(T) == 8 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3,
             const_cast<T*>(u), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
             CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Planes per CTA (cmin to 32, a multiple of `mult`): the fewest waves of resident CTAs (`per_sm` per
// SM) times the planes each CTA walks plus `start` for its start (three planes
// loaded, the previous plane's part), ties to more planes -- so small grids and
// single solves still fill the GPU without a nearly empty last wave.  Returns
// the CTAs of the launch.
static long long zsplit(int n, int nslots, long long columns, int per_sm, int cmin, int start, int& ptz,
                        int& zblocks, int mult = 1) {
  const long long slots = (long long)per_sm * 152;
  long long best = -1;
  for (int c = 32 / mult * mult; c >= cmin; c -= mult) {
    const int zb = (n + c - 1) / c;
    const long long waves = (columns * zb * nslots + slots - 1) / slots;
    if (best < 0 || waves * (c + start) < best) {
      best = waves * (c + start);
      ptz = c;
      zblocks = zb;
    }
  }
  return columns * zblocks * nslots;
}

// FP64: the fixed-point sweep, one plane per CTA and up (a 32^3 grid takes 64
// CTAs of one plane: 10 us, 16 us with four).  A block of planes with one exponent
// is what a CTA has in a launch of one field, and the CTAs of a batch take
// multiples of it: a field's bits are the same alone and in any batch.
template <>
cudaError_t launch_rhs<double>(int n, double h, double visc, const double* u, double* du, bool doadd, cudaStream_t st,
                               const SlotBatch& sb, int nslots) {
  int block, ptz, zblocks;
  dim3 grid((n + PTX - 1) / PTX, (n + FXY - 1) / FXY, 1);
  zsplit(n, 1, (long long)grid.x * grid.y, FX_CTAS, 1, 2, block, zblocks);
  zsplit(n, nslots, (long long)grid.x * grid.y, FX_CTAS, block, 2, ptz, zblocks, block);
  grid.z = zblocks * nslots;
  // the field as (x, y, z, slot * 3 + component), boxes of one plane of the
  // three components
  CUtensorMap map{};
  const long long N = (long long)n * n * n;
  const cuuint64_t dims[4] = {(cuuint64_t)n, (cuuint64_t)n, (cuuint64_t)n, (cuuint64_t)nslots * 3};
  const cuuint64_t strides[3] = {(cuuint64_t)n * 8, (cuuint64_t)n * n * 8, (cuuint64_t)N * 8};
  const cuuint32_t box[4] = {FXROW, FXBY, 1, 3};
  const int have = (nslots == 1 || sb.ustride == 3 * N) && (reinterpret_cast<uintptr_t>(u) & 15) == 0 && n >= FXROW &&
                   encode_tiled_map(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 4, u, dims, strides, box);
  const dim3 threads(PTX, FXW);
  if (doadd)
    chain(rhs_fixed_kernel<true>, grid, threads, FIXED_SMEM, st)(n, 1.0 / h, visc, u, du, sb, zblocks, ptz, block, map, have);
  else
    chain(rhs_fixed_kernel<false>, grid, threads, FIXED_SMEM, st)(n, 1.0 / h, visc, u, du, sb, zblocks, ptz, block, map, have);
  return cudaGetLastError();
}

template <>
cudaError_t launch_rhs<float>(int n, float h, float visc, const float* u, float* du, bool doadd, cudaStream_t st,
                              const SlotBatch& sb, int nslots) {
  constexpr int NC = CYT<float>;
  int ptz, zblocks;
  // the 2 x 2 kernel for 16-byte aligned fields whose rows are 16-byte
  // multiples, its last tiles ragged.  Against the general kernel, which copies
  // the last tile of a row that is no multiple of 32 word by word: 100^3 18.0 /
  // 12.7 us, 180^3 56.3 / 38.1, 240^3 112 / 81, 500^3 704 / 583; not on fewer
  // than 228 CTAs (72^3 9.9 / 10.1).  Without such tiles it wants a full wave
  // (three CTAs per SM) and at most an eighth of padding: 128^3 16.7 / 15.5, 320^3
  // 179 / 162, 512^3 691 / 622, but 96^3 9.4 / 10.0, 224^3 68.9 / 69.4.
  const int qx = (n + QX - 1) / QX, qy = (n + QY - 1) / QY;
  const long long qctas = zsplit(n, nslots, (long long)qx * qy, 3, 4, 1, ptz, zblocks);
  const bool fits = n % PTX == 0 ? qctas >= 3LL * 152 && 8 * qx * QX <= 9 * n : qctas >= 228;
  if (n % 4 == 0 && n >= QROW && fits && (reinterpret_cast<uintptr_t>(u) & 15) == 0 &&
      (reinterpret_cast<uintptr_t>(du) & 15) == 0) {
    dim3 gq(qx, qy, zblocks * nslots);
    const float ih = (float)(1.0 / (double)h);
    CUtensorMap map;
    const int have = field_tensor_map<float>(u, n, nslots, sb, QROW, QBY, &map) ? 1 : 0;
    if (doadd)
      chain(rhs_quad_kernel<true>, gq, dim3(32, 8), QUAD_SMEM, st)(n, ih, visc, u, du, sb,
                                                                zblocks, ptz, map, have);
    else
      chain(rhs_quad_kernel<false>, gq, dim3(32, 8), QUAD_SMEM, st)(n, ih, visc, u, du, sb,
                                                                 zblocks, ptz, map, have);
    return cudaGetLastError();
  }
  const int gxb = (n + PTX - 1) / PTX, gyb = (n + PTYT<NC> - 1) / PTYT<NC>;
  zsplit(n, nslots, (long long)gxb * gyb, 4, 4, 1, ptz, zblocks);
  dim3 grid(gxb, gyb, zblocks * nslots);
  const size_t sh = plane_smem_bytes<float, NC>();
  CUtensorMap map;
  const int have = field_tensor_map<float>(u, n, nslots, sb, UROW<float>, PBYT<NC>, &map) ? 1 : 0;
  if (doadd)
    chain(rhs_kernel<float, NC, true>, grid, dim3(PTX, NWARP), sh, st, CHAIN_BLOCKS_FEW)(
        n, (float)(1.0 / (double)h), visc, u, du, sb, zblocks, ptz, map, have);
  else
    chain(rhs_kernel<float, NC, false>, grid, dim3(PTX, NWARP), sh, st, CHAIN_BLOCKS_FEW)(
        n, (float)(1.0 / (double)h), visc, u, du, sb, zblocks, ptz, map, have);
  return cudaGetLastError();
}

template <typename T>
static cudaError_t configure_rhs_t() {
  constexpr int NC = CYT<T>;
  const int sh = (int)plane_smem_bytes<T, NC>();
  cudaError_t e = cudaFuncSetAttribute(rhs_kernel<T, NC, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, sh);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(rhs_kernel<T, NC, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, sh);
  return e;
}

cudaError_t configure_stencil() {
  cudaError_t e = configure_rhs_t<float>();
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(rhs_quad_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)QUAD_SMEM);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(rhs_quad_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)QUAD_SMEM);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(rhs_fixed_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FIXED_SMEM);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(rhs_fixed_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FIXED_SMEM);
  return e;
}

}  // namespace exc

extern "C" int exc_debug_wait_drill(int flags) {
  if (flags < 0 || flags > 3) { exc::set_last_error("drill flags must be 0..3"); return EXC_ERR_ARG; }
  int rc = exc::configure_device();
  if (rc) return rc;
  const int rhs = flags & 1;
  cudaError_t e = cudaMemcpyToSymbol(exc::g_rhs_drill, &rhs, sizeof(int));
  if (e != cudaSuccess) { exc::set_last_error(cudaGetErrorString(e)); return EXC_ERR_CUDA; }
  return exc::learned_set_drill((flags >> 1) & 1);
}

extern "C" int exc_device_sync(void* stream, int* flags) {
  cudaError_t e = cudaStreamSynchronize((cudaStream_t)stream);
  if (e != cudaSuccess) { exc::set_last_error(cudaGetErrorString(e)); return EXC_ERR_CUDA; }
  int f = 0;
  int rc = exc_device_faults(&f);
  if (rc) return rc;
  if (flags) *flags = f;
  if (f) {
    exc::set_last_error(f & 1 ? (f & 2 ? "device waits gave up (RHS sweep TMA plane, tensor-core convolution)"
                                       : "a device wait gave up (RHS sweep TMA plane)")
                              : "a device wait gave up (tensor-core convolution)");
    return EXC_ERR_TIMEOUT;
  }
  return EXC_OK;
}

extern "C" int exc_device_faults(int* flags) {
  if (!flags) { exc::set_last_error("null argument"); return EXC_ERR_ARG; }
  int v = 0, zero = 0, lf = 0;
  cudaError_t e = cudaMemcpyFromSymbol(&v, exc::g_rhs_tma_fault, sizeof(int));
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(exc::g_rhs_tma_fault, &zero, sizeof(int));
  if (e != cudaSuccess) { exc::set_last_error(cudaGetErrorString(e)); return EXC_ERR_CUDA; }
  const int rc = exc::learned_fault_take(&lf);
  if (rc) return rc;
  *flags = (v ? 1 : 0) | (lf ? 2 : 0);
  return EXC_OK;
}
