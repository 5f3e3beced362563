// shells.cuh - contracted Gaussian shells evaluated on the grid (the device
// half of numint.eval_ao, interface/pyscf.py:849-852, and ao_grads,
// interface/pyscf.py:677-705).
//
//   phi(r) = E0(r2) * A(d),  d = r - R_shell,  r2 = |d|^2,
//   E0 = sum_p C_p exp(-alpha_p r2),  E1 = sum_p -2 alpha_p C_p exp(..),  E2 = sum_p 4 alpha_p^2 C_p exp(..),
//   A(d) = sum_(i,j,k) t_ijk x^i y^j z^k  (the component's row of cartesian coefficients, degree l),
// so that d_x phi = A_x E0 + A x E1 and d_xx phi = A_xx E0 + 2 A_x x E1 + A (E1 + x^2 E2).
//
// Work layout: a CTA evaluates a tile of 32 grid points x 32 AOs into shared
// memory, then a sink writes the tile to its destination with the AO index
// fastest (coalesced).  In the evaluation phase the lanes of a warp are the 32
// points and each warp takes the next whole shell, so the angular momentum and
// the primitive count are uniform across the warp (no divergence) and each
// exponential is computed once per point and shell, shared by all of the
// shell's contractions and components.
//
// What bounds it is the FP64 pipe (16 clocks a warp operation): s, p and d
// shells have their own angular forms, sharing P E1 and P E2 between the seven
// values, and the exponential is taken by table (expd.cuh).  Three tiles of 32
// AOs share an SM, so that one's output runs beside the others' evaluation (of
// 64 AOs only one fits with second derivatives).
// 506 AOs (s, p, d of 4, 3, 2 primitives) x 20,001 points: 2.66 -> 1.28 ms.
#pragma once

#include "common.cuh"
#include "expd.cuh"

namespace gdft {

constexpr int kMaxShellL = 6;
constexpr int kShellCols = 8;  // l, nprim, exp offset, coef offset, first AO, ncomp, nctr, row offset
constexpr int kTilePts = 32;
constexpr int kTileAo = 32;
constexpr int kTileLd = kTileAo + 1;  // padded row: lanes (points) land in different banks
constexpr int kTileThreads = 256;
constexpr int kCtrGroup = 4;  // contractions whose radial sums are carried together

struct ShellView {
  const int32_t *shell;  // (n_shell, 8)
  const double *centre;  // (n_shell, 3)
  const double *exps;
  const double *coef;    // shell s, contraction c, primitive p at coef offset + c * nprim + p
  const int32_t *ao;     // (n_ao, 4): shell, contraction, component, 0
  const double *trans;   // shell s, component k: ncart(l) values at row offset + k * ncart(l)
  int n_shell, n_ao;
  int64_t n_prim, n_coef, n_trans;
};

__device__ __forceinline__ double nan_value() { return __longlong_as_double(0x7ff8000000000000LL); }

namespace shells_detail {

// The angular polynomial and its first and diagonal second derivatives.
template <int L>
__device__ __forceinline__ void poly(const double *__restrict__ t, double x, double y, double z, double P[7]) {
  double xp[L + 1], yp[L + 1], zp[L + 1];
  xp[0] = yp[0] = zp[0] = 1.0;
#pragma unroll
  for (int i = 1; i <= L; ++i) {
    xp[i] = xp[i - 1] * x;
    yp[i] = yp[i - 1] * y;
    zp[i] = zp[i - 1] * z;
  }
#pragma unroll
  for (int q = 0; q < 7; ++q) P[q] = 0.0;
  int idx = 0;
#pragma unroll
  for (int lx = L; lx >= 0; --lx) {
#pragma unroll
    for (int ly = L - lx; ly >= 0; --ly) {
      const int lz = L - lx - ly;
      const double c = t[idx++];
      // the lanes of a warp evaluate the same AO row (warp-uniform branch): solid-harmonic
      // rows are mostly zero, and a zero term adds nothing
      if (c == 0.0) continue;
      const double X0 = xp[lx], Y0 = yp[ly], Z0 = zp[lz];
      const double X1 = lx > 0 ? lx * xp[lx > 0 ? lx - 1 : 0] : 0.0;
      const double Y1 = ly > 0 ? ly * yp[ly > 0 ? ly - 1 : 0] : 0.0;
      const double Z1 = lz > 0 ? lz * zp[lz > 0 ? lz - 1 : 0] : 0.0;
      const double X2 = lx > 1 ? lx * (lx - 1) * xp[lx > 1 ? lx - 2 : 0] : 0.0;
      const double Y2 = ly > 1 ? ly * (ly - 1) * yp[ly > 1 ? ly - 2 : 0] : 0.0;
      const double Z2 = lz > 1 ? lz * (lz - 1) * zp[lz > 1 ? lz - 2 : 0] : 0.0;
      const double YZ = Y0 * Z0;
      P[0] = fma(c, X0 * YZ, P[0]);
      P[1] = fma(c, X1 * YZ, P[1]);
      P[2] = fma(c, X0 * Y1 * Z0, P[2]);
      P[3] = fma(c, X0 * Y0 * Z1, P[3]);
      P[4] = fma(c, X2 * YZ, P[4]);
      P[5] = fma(c, X0 * Y2 * Z0, P[5]);
      P[6] = fma(c, X0 * Y0 * Z2, P[6]);
    }
  }
}

// exp(a) for the radial sums, a = -alpha r^2, by a whole warp: by table; where a
// lane is below -708, from a + 64 ln 2 and scaled back (denormal results), and
// zero below -745.25.  Only infinities and NaN reach the library: at many points
// some lane of a warp is that far out.
__device__ __forceinline__ double radial_exp(double a, const double2 *tab) {
  if (!__any_sync(0xffffffffu, !expd::tabled(a))) return expd::exp_of(expd::parts(a, tab));
  const unsigned hi = (unsigned)__double2hiint(a);
  const bool zero = hi >= 0xC0874A00u && hi < 0xFFF00000u, deep = hi >= 0xC0862000u && hi < 0xC0874A00u;
  double b = zero ? -1.0 : a;
  if (deep) b += 0x1.62e42fefa39efp+5;
  if (!expd::tabled(b)) return exp(a);
  double e = expd::exp_of(expd::parts(b, tab));
  if (deep) e *= 0x1p-64;
  return zero ? 0.0 : e;
}

// Radial sums at a point and what of them the components share.
struct Radial {
  double E0, E1, E2;
};

// The sums of N contractions from c on.  N is a constant (not a bound under which
// four are predicated): left-out FP64 operations take their slots too.
template <int N>
__device__ __forceinline__ void radial_sums(const double *__restrict__ exps, const double *__restrict__ coef, int np,
                                            double r2, const double2 *tab, Radial *E) {
#pragma unroll
  for (int j = 0; j < N; ++j) E[j].E0 = E[j].E1 = E[j].E2 = 0.0;
  for (int q = 0; q < np; ++q) {
    const double al = exps[q];
    const double e = radial_exp(-al * r2, tab);
#pragma unroll
    for (int j = 0; j < N; ++j) {
      const double ce = coef[(int64_t)j * np + q] * e, ae = al * ce;
      E[j].E0 += ce;
      E[j].E1 += ae;
      E[j].E2 = fma(al, ae, E[j].E2);
    }
  }
#pragma unroll
  for (int j = 0; j < N; ++j) {
    E[j].E1 *= -2.0;
    E[j].E2 *= 4.0;
  }
}

// The seven values of the component with angular row t at d = (x, y, z).  q: the
// squares x^2, y^2, z^2.  A row's zeros are the same for the whole warp and are
// left out (solid harmonics are mostly zeros).
__device__ __forceinline__ bool nonzero(double t) { return (__double_as_longlong(t) << 1) != 0; }

// From the polynomial P[0] and its derivatives: first P[1..3], diagonal second P[4..6].
template <bool SECOND>
__device__ __forceinline__ void combine(const double P[7], const double d[3], const Radial &r, double v[7]) {
  const double g1 = P[0] * r.E1, g2 = P[0] * r.E2, e1 = r.E1 + r.E1;
  v[0] = P[0] * r.E0;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    v[1 + i] = fma(g1, d[i], P[1 + i] * r.E0);
    v[4 + i] = fma(d[i], fma(g2, d[i], P[1 + i] * e1), g1);
    if (SECOND) v[4 + i] = fma(P[4 + i], r.E0, v[4 + i]);
  }
}

__device__ __forceinline__ void component(int l, const double *__restrict__ t, const double d[3], const double q[3],
                                          const Radial &r, double v[7]) {
  double P[7];
  if (l == 0) {
    const double c = t[0], e0 = c * r.E0, e1 = c * r.E1, e2 = c * r.E2;
    v[0] = e0;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      v[1 + i] = e1 * d[i];
      v[4 + i] = fma(q[i], e2, e1);
    }
  } else if (l == 1) {
    P[0] = 0.0;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      P[1 + i] = t[i];
      if (nonzero(t[i])) P[0] = fma(t[i], d[i], P[0]);
    }
    combine<false>(P, d, r, v);
  } else if (l == 2) {
#pragma unroll
    for (int k = 0; k < 7; ++k) P[k] = 0.0;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = i; j < 3; ++j) {  // xx, xy, xz, yy, yz, zz
        const double c = t[i == 0 ? j : i + j + 1];
        if (!nonzero(c)) continue;
        if (i == j) {
          P[0] = fma(c, q[i], P[0]);
          P[4 + i] = c + c;
          P[1 + i] = fma(c + c, d[i], P[1 + i]);
        } else {
          const double cj = c * d[j];
          P[0] = fma(cj, d[i], P[0]);
          P[1 + i] += cj;
          P[1 + j] = fma(c, d[i], P[1 + j]);
        }
      }
    combine<true>(P, d, r, v);
  } else {
    switch (l) {
      case 3: poly<3>(t, d[0], d[1], d[2], P); break;
      case 4: poly<4>(t, d[0], d[1], d[2], P); break;
      case 5: poly<5>(t, d[0], d[1], d[2], P); break;
      default: poly<6>(t, d[0], d[1], d[2], P); break;
    }
    combine<true>(P, d, r, v);
  }
}

// A shell's table entries, checked against the table sizes.
struct ShellRec {
  int l, np, aoff, ncomp, nctr, ncart;
  int64_t poff, coff, toff;
};

__device__ __forceinline__ bool load_shell(const ShellView &B, int s, ShellRec &r) {
  if (s < 0 || s >= B.n_shell) return false;
  const int32_t *e = B.shell + (size_t)kShellCols * s;
  r.l = e[0];
  r.np = e[1];
  r.poff = e[2];
  r.coff = e[3];
  r.aoff = e[4];
  r.ncomp = e[5];
  r.nctr = e[6];
  r.toff = e[7];
  if (r.l < 0 || r.l > kMaxShellL || r.np <= 0 || r.ncomp <= 0 || r.nctr <= 0) return false;
  r.ncart = (r.l + 1) * (r.l + 2) / 2;
  return r.poff >= 0 && r.poff + r.np <= B.n_prim && r.coff >= 0 && r.coff + (int64_t)r.nctr * r.np <= B.n_coef &&
         r.toff >= 0 && r.toff + (int64_t)r.ncomp * r.ncart <= B.n_trans && r.aoff >= 0 &&
         (int64_t)r.aoff + (int64_t)r.nctr * r.ncomp <= B.n_ao;
}

}  // namespace shells_detail

// Evaluation phase, by all threads of the block (the caller synchronises): the tile
// [kVals][kTilePts][kTileLd] of AOs [a0, a0 + kTileAo)
// at points [p0, p0 + 32).  kVals = 7 keeps the three diagonal second
// derivatives, kVals = 5 their sum (the Laplacian).  Entries no shell covers
// stay NaN; AOs at or beyond n_ao stay NaN too (sinks write zero padding there).
template <int kVals>
__device__ __forceinline__ void eval_tile(const ShellView &B, const double *__restrict__ coords, int64_t n_grid,
                                          int64_t p0, int a0, double *tile) {
  using namespace shells_detail;
  __shared__ double2 tab[expd::kTable];
  __shared__ int next;  // the next shell that a warp takes
  expd::build_table(tab);
  for (int i = threadIdx.x; i < kVals * kTilePts * kTileLd; i += blockDim.x) tile[i] = nan_value();
  const int a1 = min(a0 + kTileAo, B.n_ao);
  const int s_lo = a0 < B.n_ao ? B.ao[4 * a0] : 0, s_hi = a0 < B.n_ao ? B.ao[4 * (a1 - 1)] : -1;
  if (threadIdx.x == 0) next = s_lo;
  __syncthreads();
  if (s_lo < 0 || s_hi >= B.n_shell || s_hi < s_lo) return;
  const int lane = threadIdx.x & 31;
  const int64_t p = p0 + lane;
  double px = 0.0, py = 0.0, pz = 0.0;
  if (p < n_grid) {
    px = coords[3 * p + 0];
    py = coords[3 * p + 1];
    pz = coords[3 * p + 2];
  }
  for (;;) {
    int s = lane == 0 ? atomicAdd(&next, 1) : 0;
    s = __shfl_sync(0xffffffffu, s, 0);
    if (s > s_hi) break;
    ShellRec r;
    if (!load_shell(B, s, r)) continue;
    const int lo = max(a0, r.aoff), hi = min(a1, r.aoff + r.nctr * r.ncomp);
    if (lo >= hi) continue;
    const double d[3] = {px - B.centre[3 * s + 0], py - B.centre[3 * s + 1], pz - B.centre[3 * s + 2]};
    const double sq[3] = {d[0] * d[0], d[1] * d[1], d[2] * d[2]};
    const double r2 = sq[0] + sq[1] + sq[2];
    const int c_lo = (lo - r.aoff) / r.ncomp, c_hi = (hi - 1 - r.aoff) / r.ncomp;
    for (int cg = c_lo; cg <= c_hi; cg += kCtrGroup) {
      const int nc = min(kCtrGroup, c_hi - cg + 1);
      Radial E[kCtrGroup];
      const double *exps = B.exps + r.poff, *coef = B.coef + r.coff + (int64_t)cg * r.np;
      switch (nc) {
        case 1: radial_sums<1>(exps, coef, r.np, r2, tab, E); break;
        case 2: radial_sums<2>(exps, coef, r.np, r2, tab, E); break;
        case 3: radial_sums<3>(exps, coef, r.np, r2, tab, E); break;
        default: radial_sums<kCtrGroup>(exps, coef, r.np, r2, tab, E);
      }
#pragma unroll
      for (int j = 0; j < kCtrGroup; ++j) {
        if (j >= nc) break;
        for (int k = 0; k < r.ncomp; ++k) {
          const int a = r.aoff + (cg + j) * r.ncomp + k;
          if (a < lo || a >= hi) continue;
          double v[7];
          component(r.l, B.trans + r.toff + (int64_t)k * r.ncart, d, sq, E[j], v);
          double *t = tile + (size_t)lane * kTileLd + (a - a0);
#pragma unroll
          for (int q = 0; q < 4; ++q) t[q * kTilePts * kTileLd] = v[q];
          if (kVals == 7) {
#pragma unroll
            for (int q = 4; q < 7; ++q) t[q * kTilePts * kTileLd] = v[q];
          } else {
            t[4 * kTilePts * kTileLd] = (v[4] + v[5]) + v[6];
          }
        }
      }
    }
  }
}

// One tile per CTA: blockIdx.x = 32-point group, blockIdx.y = 32-AO chunk of
// the sink's AO extent.  The sink is called after the whole tile is written.
template <int kVals, class Sink>
__global__ void __launch_bounds__(kTileThreads, 3) eval_shells_tile_kernel(ShellView B, const double *__restrict__ coords,
                                                                        int64_t n_grid, Sink sink) {
  extern __shared__ double tile[];
  const int64_t p0 = (int64_t)blockIdx.x * kTilePts;
  const int a0 = blockIdx.y * kTileAo;
  eval_tile<kVals>(B, coords, n_grid, p0, a0, tile);
  __syncthreads();
  for (int i = threadIdx.x; i < kTilePts * kTileAo; i += blockDim.x) {
    const int pt = i / kTileAo, aa = i % kTileAo;
    sink(tile, pt * kTileLd + aa, kTilePts * kTileLd, p0 + pt, a0 + aa);
  }
}

constexpr size_t tile_smem_bytes(int vals) { return (size_t)vals * kTilePts * kTileLd * sizeof(double); }

// Launch over (points rounded to 32) x (AO extent rounded to 32).
template <int kVals, class Sink>
cudaError_t launch_shell_tiles(const ShellView &B, const double *coords, int64_t n_grid, int64_t n_points,
                               int ao_extent, const Sink &sink, cudaStream_t st) {
  const size_t smem = tile_smem_bytes(kVals);
  cudaError_t e = cudaFuncSetAttribute(eval_shells_tile_kernel<kVals, Sink>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const dim3 grid((unsigned)((n_points + kTilePts - 1) / kTilePts), (unsigned)((ao_extent + kTileAo - 1) / kTileAo));
  eval_shells_tile_kernel<kVals, Sink><<<grid, kTileThreads, smem, st>>>(B, coords, n_grid, sink);
  return cudaGetLastError();
}

}  // namespace gdft
