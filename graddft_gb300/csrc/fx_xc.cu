// fx_xc.cu - the FP64 form's density and V_xc contractions on fx_gemm.cu.
//
// Density: X_t = T_t D for the planes t = phi, d_x, d_y, d_z, 128 points x 64
// columns of both spins per tile, then one pass of row products with the planes
// (molecule.py:385-502; the sums dens_f64.cu states).  The d_j planes enter only
// through quadratic forms sum_ab d_j phi_a D_ab d_j phi_b, which need one
// triangle: column block b takes the row blocks a <= b of U = D + D^T (D itself
// on the diagonal blocks), (n + 64) / 2n of the products.  A point's row of AOs is fixed
// point on the largest, which may be one that D hardly occupies (a steep function near its
// nucleus): phi_a is taken times 2^t and D_ab times 2^-t, t half the exponent of the
// largest entry of D in row or column a, relative to D's largest (exact), so that rows are like
// phi_a sqrt(D_aa).  The spins share the digits of phi: the larger of their two t counts.
// s functions up to exponent 1e10, the two steepest not in D, errors relative to the sums of
// the terms' sizes: rho 5e-15 -> 3e-16, tau 8e-11 -> 4e-16.
//
// V_xc: V_s = phi^T Q_s + sum_j d_j phi^T (c_kin,s d_j phi), with
// Q_s = c_rho phi + sum_j c_gj d_j phi + c_lap lap phi (vxc_f64.cu).  The second
// sum is symmetric: only tiles that reach the diagonal are formed.  A row of this
// contraction is one AO over the points of a slab, in fixed point on its largest
// value, and phi and Q are graded against one another: a steep function is large
// where the weights, and so Q, are small.  Both are therefore taken times a power
// of two for each point that shares the coefficients out evenly (phi 2^t and
// Q 2^-t, t half the exponent of the point's largest coefficient, relative to the spin's
// largest in the slab, the larger of the spins' t; exact): rows are then
// like sqrt(|c|) phi, square-integrable, and the error is relative to the product of
// two such maxima instead of max |phi_a| max |Q_b|.  s functions of exponents A and 0.15
// on one centre, 300 radial points, error relative to sum |phi_a Q_b|: A = 6,665
// 8e-13 -> 2e-15, 1e6 3e-10 -> 3e-14, 1e8 1e-6 -> 5e-13 (an FP64 sum 7e-16).  What is left of
// the grading, and AOs that hardly meet (distant centres), are held to 2^-58 of that product.
//
// Both run over the grid in slabs whose digits and products fit a fixed
// workspace.  An operand that is not finite (or overflows its bound) sets a
// word on the device; the plain kernels of dens_f64.cu and vxc_f64.cu then
// compute the whole result, with IEEE's infinities and NaNs.  This path is the
// faster one at every size (E_xc + V_xc, B88+LYP, plain kernels -> here: 4 AOs x
// 128 points 779 -> 294 us, 24 x 3,600 928 -> 397 us, 100 x 10,000 5.4 -> 0.74 ms,
// 400 x 150,001 827 -> 27.6 ms; with the point kernel's and launches' later forms 24 x
// 3,600 146 us, 400 x 150,001 22.9 ms), and the more accurate one (features at 400 AOs
// against quadruple precision: 1.4e-16 .. 2.7e-16, before 2.7e-16 .. 6.0e-16).
#include "common.cuh"
#include "fx.cuh"
#include "kernels.cuh"

namespace gdft {
namespace fx {

namespace {

// Workspace of one slab, about.  A slab's GEMM ends in a wave that is not full and
// its sums are added to the slab before's, so few and large ones are faster (B88 115 x
// 65,536 at 512 MB, 1, 2 and 4 GB: 1,128, 1,108, 971, 971 us; BLYP 400 x 150,001 23.7,
// 22.4, 21.9, 21.7 ms); but every resident molecule holds its workspace, and a set of
// them should not take several times the memory of its tables.
constexpr size_t kSlabBytes = (size_t)1 << 30;
size_t align256(size_t x) { return (x + 255) / 256 * 256; }

// High word of |x|, kNone for a zero.
constexpr int kNone = -(1 << 30);
__device__ __forceinline__ int hi_of(double x) {
  const int h = __double2hiint(x) & 0x7FFFFFFF;
  return h ? h : kNone;
}
// Exponent field of a row's largest high word m, negative where the octaves have moved it there; 1 for a row without
// values (kNone, or a little above it).
constexpr int kNoRow = -(600 << 20);
__device__ __forceinline__ int field_at(int m) { return m < kNoRow ? 1 : m >> 20; }

// Largest high word of D in row or column a of either spin, mx[2][n_pad], a warp each; also clears the non-finite
// word, if any.
__global__ void __launch_bounds__(256) fx_rdm1_max_kernel(const double *__restrict__ D, int n, int n_pad,
                                                          int *__restrict__ mx, int *__restrict__ bad) {
  previous_done();
  if (blockIdx.x == 0 && threadIdx.x == 0 && bad != nullptr) *bad = 0;
  const int i = (blockIdx.x * 256 + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (i >= 2 * n_pad) return;
  const int a = i % n_pad;
  const double *Ds = D + (size_t)(i / n_pad) * n * n;
  int m = kNone;
  for (int b = lane; a < n && b < n; b += 32) m = max(m, max(hi_of(Ds[(size_t)a * n + b]), hi_of(Ds[(size_t)b * n + a])));
#pragma unroll
  for (int o = 16; o > 0; o /= 2) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (lane == 0) mx[i] = m;
}

// Octaves of the AOs from that, one block: half the exponent relative to the spin's
// largest, of both spins together (the larger one) or of each.  kEmpty where D has no entry
// (and past the last AO): the AO's digits are then below all others.
constexpr int kEmpty = -1200;
__global__ void __launch_bounds__(1024) fx_octaves_kernel(const int *__restrict__ mx, int n_pad, bool each,
                                                          int *__restrict__ oct) {
  previous_done();
  __shared__ int top[2];
  if (threadIdx.x < 2) top[threadIdx.x] = kNone;
  __syncthreads();
  for (int i = threadIdx.x; i < 2 * n_pad; i += blockDim.x) atomicMax(&top[i / n_pad], mx[i]);
  __syncthreads();
  for (int a = threadIdx.x; a < n_pad; a += blockDim.x) {
    int t[2];
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const int m = mx[s * n_pad + a];
      t[s] = m == kNone ? kEmpty : (m - top[s]) >> 21;
    }
    if (each) {
      oct[a] = t[0];
      oct[n_pad + a] = t[1];
    } else {
      oct[a] = max(t[0], t[1]);
    }
  }
}

// Digits of D as the B operand: tile nt = columns 64 nt .. of spin 0, then of
// spin 1; version 0 is D, version 1 the triangle U (chunks 0 .. nt).  A warp
// takes eight operand rows (columns of D), lane = (row, eight consecutive k).
__global__ void __launch_bounds__(128) fx_rdm1_kernel(const double *__restrict__ D, int n, int nb,
                                                      const int *__restrict__ oct, unsigned char *__restrict__ out,
                                                      int *__restrict__ exps, int *__restrict__ bad) {
  previous_done();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = blockIdx.x * 4 + warp;  // group of eight operand rows: 16 per tile
  if (g >= nb * 16) return;
  const int version = blockIdx.y;
  const int nt = g / 16, rt = (g % 16) * 8 + (lane & 7);
  const int s = rt >> 6, c = nt * 64 + (rt & 63);
  const double *Ds = D + (size_t)s * n * n;
  const int chunks = version ? nt + 1 : nb;
  const int kg = (lane >> 3) * 8;
  auto value = [&](int k) {
    if (c >= n || k >= n) return 0.0;
    const double d = Ds[(size_t)k * n + c];
    return version && k < nt * 64 ? d + Ds[(size_t)c * n + k] : d;
  };
  int m = kNone;
  for (int k = kg; k < chunks * kChunkK; k += 32)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int h = hi_of(value(k + j));
      if (h != kNone) m = max(m, h - oct[k + j] * (1 << 20));
    }
  m = max(m, __shfl_xor_sync(0xffffffffu, m, 8));
  m = max(m, __shfl_xor_sync(0xffffffffu, m, 16));
  const int emax = field_at(m);
  if (emax > kMaxField) atomicOr(bad, 1);
  if (lane < 8) exps[version * nb * kTile + nt * kTile + rt] = emax;
  unsigned char *base = out + ((size_t)version * nb + nt) * nb * kSetBytes;
  for (int k = kg; k < chunks * kChunkK; k += 32) {
    long long f[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = to_fixed(value(k + j), emax + oct[k + j]);
    uint4 d[kDigits];
    digits8(f, d);
    unsigned char *set = base + (size_t)(k / kChunkK) * kSetBytes + elem_off(rt, k % kChunkK);
#pragma unroll
    for (int i = 0; i < kDigits; ++i) *(uint4 *)(set + (size_t)i * kBlockBytes) = d[i];
  }
}

// Row products of X with the planes -> feat.  X is [plane][spin][column][slab
// point], the planes [point][ld]: a block takes 32 points and walks the columns
// in tiles of 16, the planes' tile through shared memory (rows in, columns out),
// X directly (lanes are points); both spins share a tile.  Bound by the FP64 pipe
// (16 FMA per point and column); the next tile is copied asynchronously while one
// is used, and at 43 KB four blocks share an SM: 9,376 x 400 148 -> 130 us (one tile
// of 32 at a time; two of 32 127, but 79.5 against 75.9 at 33,920 x 43), where the
// pipe needs 108.
constexpr int kFeatTile = 32;  // points
constexpr int kFeatCols = 16;
__global__ void __launch_bounds__(256, 4) fx_features_kernel(const double *__restrict__ tab, size_t pe, int64_t np, int ld,
                                                          int n, int64_t p0, int64_t slab,
                                                          const double *__restrict__ X, int cols, bool kin,
                                                          double *__restrict__ feat, const int *__restrict__ bad) {
  previous_done();
  if (*bad != 0) return;
  __shared__ double tile[2][kPlanes][kFeatTile][kFeatCols + 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t r0 = (int64_t)blockIdx.x * kFeatTile;
  const int planes = kin ? kPlanes : 4;
  const size_t xs = (size_t)slab * cols;
  double f[2][6];
#pragma unroll
  for (int s = 0; s < 2; ++s)
#pragma unroll
    for (int k = 0; k < 6; ++k) f[s][k] = 0.0;
  auto fetch = [&](int c0, int b) {  // the planes' columns c0 .. c0 + 15, 16 lanes a point
    const int l = threadIdx.x % kFeatCols;
    for (int i = threadIdx.x / kFeatCols; i < planes * kFeatTile; i += 256 / kFeatCols) {
      const unsigned dst = (unsigned)__cvta_generic_to_shared(&tile[b][i / kFeatTile][i % kFeatTile][l]);
      const double *src = tab + (size_t)(i / kFeatTile) * pe + (size_t)(p0 + r0 + i % kFeatTile) * ld + c0 + l;
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fetch(0, 0);
  for (int c0 = 0, b = 0; c0 < n; c0 += kFeatCols, b ^= 1) {  // ld, a multiple of 32, holds the last tile
    if (c0 + kFeatCols < n) {
      fetch(c0 + kFeatCols, b ^ 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    const auto &t = tile[b];
#pragma unroll
    for (int k = 0; k < kFeatCols / 8; ++k) {
      const int c = warp + 8 * k;
      if (c0 + c >= n) break;  // X has no columns from n on: whatever memory holds there times the planes' zeros
      const double phi = t[T_PHI][lane][c], dx = t[T_DX][lane][c], dy = t[T_DY][lane][c], dz = t[T_DZ][lane][c];
      const double *x = X + (size_t)(c0 + c) * slab + r0 + lane;
#pragma unroll
      for (int s = 0; s < 2; ++s, x += xs) {
        const double x0 = x[0];
        f[s][0] = fma(x0, phi, f[s][0]);
        f[s][1] = fma(x0, dx, f[s][1]);
        f[s][2] = fma(x0, dy, f[s][2]);
        f[s][3] = fma(x0, dz, f[s][3]);
        if (kin) {
          f[s][4] = fma(x0, t[T_LAP][lane][c], f[s][4]);
          f[s][5] = fma(x[2 * xs], dx, f[s][5]);
          f[s][5] = fma(x[4 * xs], dy, f[s][5]);
          f[s][5] = fma(x[6 * xs], dz, f[s][5]);
        }
      }
    }
    __syncthreads();
  }
  double *red = &tile[0][0][0][0];  // [warp][spin * 6 + feature][point]
#pragma unroll
  for (int k = 0; k < 12; ++k) red[(warp * 12 + k) * 32 + lane] = f[k / 6][k % 6];
  __syncthreads();
  for (int i = threadIdx.x; i < 12 * 32; i += 256) {
    double v = 0.0;
#pragma unroll
    for (int w = 0; w < 8; ++w) v += red[w * 12 * 32 + i];
    red[i] = v;  // only this thread reads entry i of warp 0's block
  }
  __syncthreads();
  if (warp < 2) {
    const int64_t p = p0 + r0 + lane;
    const double *v = red + warp * 6 * 32 + lane;
    double *fs = feat + (size_t)warp * kFeat * np;
    fs[F_RHO * np + p] = v[0];
    fs[F_GX * np + p] = 2.0 * v[32];
    fs[F_GY * np + p] = 2.0 * v[64];
    fs[F_GZ * np + p] = 2.0 * v[96];
    fs[F_LAP * np + p] = 2.0 * v[160] + 2.0 * v[128];
    fs[F_TAU * np + p] = 0.5 * v[160];
  }
}

// ---------------------------------------------------------------- V_xc operands
// High words add like logarithms: hi(x) + hi(y) - hi(1) is at most the product's, and
// below it by at most 3 - 2 sqrt 2 = 0.172 of an octave (both mantissas sqrt 2), for which field_of adds 1/4.
constexpr int kOneHi = 0x3FF00000;
static_assert((int)T_PHI == (int)C_RHO && (int)T_DX == (int)C_GX && (int)T_DY == (int)C_GY && (int)T_DZ == (int)C_GZ &&
                  (int)T_LAP == (int)C_LAP,
              "Q pairs plane p with coefficient p");
// Exponent field bound of a sum of `terms` products whose largest has the (approximate) high word m.
__device__ __forceinline__ int field_of(int m, int octaves) {
  if (m < kNoRow) return 1;
  const int f = ((m + (1 << 18)) >> 20) + octaves;
  return f > 0x7FE ? 0x7FE : f;
}

// Largest high words of a slab's coefficients: g[0][s] of those of Q_s, g[1][s] of c_kin,s.
__global__ void __launch_bounds__(256) fx_coef_max_kernel(const double *__restrict__ coef, int64_t np, int64_t p0,
                                                          int64_t rows, int *__restrict__ g) {
  previous_done();
  __shared__ int sg[4];
  if (threadIdx.x < 4) sg[threadIdx.x] = kNone;
  __syncthreads();
  const int64_t p = (int64_t)blockIdx.x * 256 + threadIdx.x;
  const int warp_lane = threadIdx.x & 31;
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    int m[2] = {kNone, kNone};
    if (p < rows)
#pragma unroll
      for (int k = 0; k < kFeat; ++k)
        m[k == C_KIN] = max(m[k == C_KIN], hi_of(coef[((size_t)s * kFeat + k) * np + p0 + p]));
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int w = __reduce_max_sync(0xffffffffu, m[i]);
      if (warp_lane == 0) atomicMax(&sg[2 * i + s], w);
    }
  }
  __syncthreads();
  if (threadIdx.x < 4) atomicMax(g + threadIdx.x, sg[threadIdx.x]);
}

// The non-finite word, and n maxima below every high word (a kernel, not a
// memset: launches before and after it stay chained).
__global__ void fx_clear_kernel(int *bad, int *mx, int n) {
  previous_done();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0 && bad != nullptr) *bad = 0;
  if (i < n) mx[i] = kNone;
}

// Largest high words over a slab of points: [0] phi, [1] d_j phi (one for the
// three), [2 + s] the terms of Q_s, [4 + s] c_kin,s d_j phi, each with its point's
// octaves, which go to oct[2][oct_stride] (phi's and Q's, then the kinetic part's).
// Lanes are AOs, a block takes 32 AOs and `per` points, its warps every eighth point.
__global__ void __launch_bounds__(256) fx_vmax_kernel(const double *__restrict__ tab, size_t pe, int64_t np, int ld,
                                                      const double *__restrict__ coef, int64_t p0, int64_t rows,
                                                      int per, bool kin, int n_max, const int *__restrict__ g,
                                                      int *__restrict__ mx, int *__restrict__ oct, int64_t oct_stride,
                                                      int *__restrict__ bad) {
  previous_done();
  __shared__ int sc[2][kFeat][128], so[2][128];  // high words over 1 (2^-t, for the octaves), octaves
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int a = blockIdx.x * 32 + lane;
  int m[6] = {kNone, kNone, kNone, kNone, kNone, kNone};
  const int64_t r_begin = (int64_t)blockIdx.y * per, r_end = r_begin + per < rows ? r_begin + per : rows;
  for (int64_t q0 = r_begin; q0 < r_end; q0 += 128) {
    const int cnt = (int)(r_end - q0 < 128 ? r_end - q0 : 128);
    __syncthreads();
    for (int i = threadIdx.x; i < 2 * kFeat * 128; i += blockDim.x) {
      const int p = i % 128;
      const int h = p < cnt ? hi_of(coef[(size_t)(i / 128) * np + p0 + q0 + p]) : kNone;
      if (h > (kMaxField << 20)) atomicOr(bad, 1);
      (&sc[0][0][0])[i] = h == kNone ? kNone : h - kOneHi;
    }
    __syncthreads();
    {
      const int p = threadIdx.x % 128, part = threadIdx.x / 128;  // part 1: the kinetic rows
      const int k0 = part ? C_KIN : 0, k1 = part ? C_KIN + 1 : C_KIN;
      int t = kDead;
      for (int s = 0; s < 2; ++s) {
        int m = kNone;
        for (int k = k0; k < k1; ++k) m = max(m, sc[s][k][p]);
        if (m != kNone) t = max(t, (m - (g[2 * part + s] - kOneHi)) >> 21);
      }
      so[part][p] = t;
      for (int k = k0; k < k1; ++k)
        for (int s = 0; s < 2; ++s)  // kept at or above kNone: two of them still add without overflow
          if (sc[s][k][p] != kNone) sc[s][k][p] = max(sc[s][k][p] - (t << 20), kNone);
      if (blockIdx.x == 0 && p < cnt) oct[part * oct_stride + q0 + p] = t;
    }
    __syncthreads();
    if (a < ld)
      for (int p = warp; p < cnt; p += 8) {
        const double *t = tab + (size_t)(p0 + q0 + p) * ld + a;
        const int phi = hi_of(t[0]), dx = hi_of(t[pe]), dy = hi_of(t[2 * pe]), dz = hi_of(t[3 * pe]),
                  lp = hi_of(t[4 * pe]);
        const int dm = max(dx, max(dy, dz));
        if (max(phi, max(dm, lp)) > (kMaxField << 20)) atomicOr(bad, 1);
        if (so[0][p] != kDead) m[0] = max(m[0], phi + (so[0][p] << 20));
        if (so[1][p] != kDead) m[1] = max(m[1], dm + (so[1][p] << 20));
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          int v = sc[s][C_RHO][p] + phi;
          v = max(v, sc[s][C_GX][p] + dx);
          v = max(v, sc[s][C_GY][p] + dy);
          v = max(v, sc[s][C_GZ][p] + dz);
          v = max(v, sc[s][C_LAP][p] + lp);
          m[2 + s] = max(m[2 + s], v);
          if (kin) m[4 + s] = max(m[4 + s], sc[s][C_KIN][p] + dm);
        }
      }
  }
  if (a < ld) {
#pragma unroll
    for (int k = 0; k < 6; ++k) atomicMax(mx + (size_t)k * n_max + a, m[k]);
  }
}

// Digits of the operands for 64 points (one K chunk) and 32 AOs: warp = eight
// consecutive points, lane = AO.  blockIdx.x = 0: A sets [mt][4 npc] (the planes),
// 1 and 2: B sets [nb][4 npc] of spin 0 and 1 (Q and c_kin d_j phi), chunk t npc + pc
// for plane t.  One plane's values live at a time (the planes are read again from
// L1): with all five in registers one block of 168 registers a thread fitted an SM
// and the kernel ran at 3 TB/s, bound by its latencies (6,800 points x 400 AOs 187 us,
// then 139; 72 bytes are spilled at 64 registers, and one block less an SM costs more).  The three blocks of a tile are neighbours in the launch, so that its
// planes come from HBM once (128 us).  The blocks of chunk 0 write
// the exponent fields of the operand rows: ea [2][128 mt] (phi, kinetic), eb
// [2][128 nb] (Q, kinetic; tile rows 64 of each spin).
__global__ void __launch_bounds__(256, 4) fx_vdigits_kernel(const double *__restrict__ tab, size_t pe, int64_t np, int ld,
                                                            const double *__restrict__ coef, int64_t p0, int64_t rows,
                                                            int npc, bool kin, int mt, int nb, int n8,
                                                            const int *__restrict__ mx,
                                                            const int *__restrict__ oct, int64_t oct_stride,
                                                            int *__restrict__ ea, int *__restrict__ eb,
                                                            unsigned char *__restrict__ va,
                                                            unsigned char *__restrict__ vb, int *__restrict__ bad) {
  previous_done();
  if (*bad != 0) return;
  __shared__ double sc[kFeat][64];
  __shared__ int so[2][64];  // the points' octaves, for B with the other sign
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int pc = blockIdx.z, a = blockIdx.y * 32 + lane, s = (int)blockIdx.x - 1;
  const int64_t q0 = (int64_t)pc * kChunkK;
  if (s >= 0) {
    for (int i = threadIdx.x; i < kFeat * 64; i += blockDim.x) {
      const int p = i % 64;
      sc[i / 64][p] = q0 + p < rows ? coef[((size_t)s * kFeat + i / 64) * np + p0 + q0 + p] : 0.0;
    }
  }
  if (threadIdx.x < 128) {
    const int p = threadIdx.x % 64, t = q0 + p < rows ? oct[threadIdx.x / 64 * oct_stride + q0 + p] : 0;
    so[threadIdx.x / 64][p] = s < 0 ? t : -t;
  }
  __syncthreads();
  if (a >= n8) return;  // n8 <= ld
  const int k0 = warp * 8, n_max = mt * kTile;
  const int64_t left = rows - q0 - k0;  // points of these eight that there are
  const double *t0 = tab + (size_t)(p0 + q0 + k0) * ld + a;
  const size_t chunks = (size_t)(kin ? 4 : 1) * npc;
  bool over = false;
  auto load = [&](int p, double (&v)[8]) {
    const double *t = t0 + (size_t)p * pe;
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = j < left ? t[(size_t)j * ld] : 0.0;
  };
  auto emit = [&](unsigned char *set, int row, const double (&x)[8], int emax, const int *octaves) {
    over = over || emax > kMaxField;
    long long f[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int e = emax - octaves[k0 + j];
      if (s >= 0) {  // A's maxima are exact, and have been looked at
        const int ef = exp_field((uint32_t)__double2hiint(x[j]));
        over = over || (ef != 0 && ef > e);
      }
      f[j] = to_fixed(x[j], e);
    }
    uint4 d[kDigits];
    digits8(f, d);
    unsigned char *o = set + elem_off(row, k0);
#pragma unroll
    for (int i = 0; i < kDigits; ++i) *(uint4 *)(o + (size_t)i * kBlockBytes) = d[i];
  };
  double v[8];
  if (s < 0) {
    const int e0 = field_at(mx[a]), e1 = field_at(mx[n_max + a]);
    if (pc == 0 && warp == 0) {
      ea[a] = e0;
      ea[n_max + a] = e1;
    }
    unsigned char *A = va + ((size_t)(a / kTile) * chunks + pc) * kSetBytes;
#pragma unroll 1
    for (int t = 0; t < (kin ? 4 : 1); ++t) {
      load(t, v);
      emit(A + (size_t)t * npc * kSetBytes, a % kTile, v, t ? e1 : e0, so[t ? 1 : 0]);
    }
  } else {
    const int row = s * 64 + a % 64, at = a / 64 * kTile + row;
    const int e0 = field_of(mx[(size_t)(2 + s) * n_max + a], 3);  // five terms
    const int e1 = field_of(mx[(size_t)(4 + s) * n_max + a], 0);
    if (pc == 0 && warp == 0) {
      eb[at] = e0;
      eb[nb * kTile + at] = e1;
    }
    unsigned char *B = vb + ((size_t)(a / 64) * chunks + pc) * kSetBytes;
    double q[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) q[j] = 0.0;
#pragma unroll 1
    for (int p = 0; p < kPlanes; ++p) {  // C_RHO phi + C_GX d_x + C_GY d_y + C_GZ d_z + C_LAP lap: same order
      load(p, v);
#pragma unroll
      for (int j = 0; j < 8; ++j) q[j] = fma(sc[p][k0 + j], v[j], q[j]);
    }
    emit(B, row, q, e0, so[0]);
    if (kin)
#pragma unroll 1
      for (int t = 1; t < 4; ++t) {
        load(t, v);
#pragma unroll
        for (int j = 0; j < 8; ++j) q[j] = sc[C_KIN][k0 + j] * v[j];
        emit(B + (size_t)t * npc * kSetBytes, row, q, e1, so[1]);
      }
  }
  if (over) atomicOr(bad, 1);
}

// V[s][a][b] = sum of the phi part's splits at (a, b) and of the kinetic part's
// at (a, b) or, left of the diagonal tile, (b, a).  part: [split][spin][b][a].
// A block takes one b, 32 a (lanes) and spreads the splits over its eight warps:
// with few AOs there are hundreds of splits and few elements.
__global__ void __launch_bounds__(256) fx_vreduce_kernel(const double *__restrict__ part, int s0, int s1, int n,
                                                         int rows, int cols, double *__restrict__ out,
                                                         const int *__restrict__ bad) {
  previous_done();
  if (*bad != 0) return;
  __shared__ double sm[8][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int a = blockIdx.x * 32 + lane, b = blockIdx.y, s = blockIdx.z;
  const size_t split = (size_t)2 * rows * cols, spin = (size_t)s * rows * cols;
  double v = 0.0;
  if (a < n) {
    const double *p = part + spin + (size_t)b * rows + a;
    for (int k = warp; k < s0; k += 8) v += p[(size_t)k * split];
    p = part + (size_t)s0 * split + spin + (b >= a / kTile * kTile ? (size_t)b * rows + a : (size_t)a * rows + b);
    for (int k = warp; k < s1; k += 8) v += p[(size_t)k * split];
  }
  sm[warp][lane] = v;
  __syncthreads();
  if (warp == 0 && a < n) {
#pragma unroll
    for (int w = 1; w < 8; ++w) v += sm[w][lane];
    out[((size_t)s * n + a) * n + b] = v;
  }
}

}  // namespace

XcWs xc_ws(int64_t np, int n_ao) {
  XcWs w{};
  w.nb = (n_ao + 63) / 64;
  w.mt = (n_ao + kTile - 1) / kTile;
  const int64_t n64 = (int64_t)w.nb * 64, n128 = (int64_t)w.mt * kTile;
  auto slab = [&](int64_t per_point) {
    int64_t p = (int64_t)kSlabBytes / per_point / 128 * 128;
    p = p < 1024 ? 1024 : p;
    return p < np ? p : round_up(np, 128);
  };
  w.dens_slab = slab(n64 * (4 * 2 * kDigits + 64));
  w.v_slab = slab((n128 + n64 * 2) * 4 * 2 * kDigits);
  // V_xc items: about two rounds of one CTA per SM, at least four chunks each.
  const int64_t npc = w.v_slab / kChunkK;
  int64_t upper = 0;
  for (int m = 0; m < w.mt; ++m) upper += w.nb - 2 * m > 0 ? w.nb - 2 * m : 0;
  const int64_t work = npc * ((int64_t)w.mt * w.nb + 3 * upper);
  int64_t per = (work + 2 * 148 - 1) / (2 * 148);
  per = per < 4 ? 4 : per;
  w.v_chunks = (int)per;
  w.s0 = (int)((npc + per - 1) / per);
  w.s1 = (int)((3 * npc + per - 1) / per);
  size_t off = 0;
  w.off_bad = off;
  off = 256;
  const size_t shared = off;
  w.off_dset = off;
  off = align256(off + (size_t)2 * w.nb * w.nb * kSetBytes);
  w.off_dexp = off;
  off = align256(off + (size_t)2 * w.nb * kTile * sizeof(int));
  w.off_doct = off;
  off = align256(off + (size_t)3 * octaves_len(n_ao) * sizeof(int));  // and the maxima they come from
  w.off_a = off;
  off = align256(off + (size_t)4 * (w.dens_slab / kTile) * w.nb * kSetBytes);
  w.off_ea = off;
  off = align256(off + (size_t)4 * w.dens_slab * sizeof(int));
  w.off_x = off;
  off = align256(off + (size_t)8 * w.dens_slab * n64 * sizeof(double));
  const size_t dens_end = off;
  off = shared;
  w.off_va = off;
  off = align256(off + (size_t)w.mt * 4 * npc * kSetBytes);
  w.off_vb = off;
  off = align256(off + (size_t)w.nb * 4 * npc * kSetBytes);
  w.off_vexp = off;
  off = align256(off + (size_t)(2 * w.mt * kTile + 2 * w.nb * kTile + 6 * n128 + 4 + 2 * w.v_slab) * sizeof(int));
  w.off_vpart = off;
  // s0 + s1 is at most this for any grid, so a shorter grid never needs more than a longer one.
  const int64_t most = 4 * 2 * 148 / ((int64_t)w.mt * w.nb + 3 * upper) + 2;
  off = align256(off + (size_t)most * 2 * n128 * n64 * sizeof(double));
  w.bytes = off > dens_end ? off : dens_end;
  return w;
}

cudaError_t launch_octaves(const double *D, int n, bool each, int *mx, int *oct, int *bad, cudaStream_t st) {
  const int len = octaves_len(n);
  launch_next(fx_rdm1_max_kernel, 2 * len / 8, 256, 0, st, D, n, len, mx, bad);
  launch_next(fx_octaves_kernel, 1, len < 1024 ? len : 1024, 0, st, mx, len, each, oct);
  return cudaGetLastError();
}

cudaError_t launch_density(const double *tab, int64_t np, int ld, int n_ao, const double *rdm1, bool kin, double *feat,
                           unsigned char *ws, int *err, cudaStream_t st) {
  const XcWs w = xc_ws(np, n_ao);
  const size_t pe = (size_t)np * ld;
  int *bad = bad_word(ws, w);
  unsigned char *dset = ws + w.off_dset;
  int *dexp = (int *)(ws + w.off_dexp), *ea = (int *)(ws + w.off_ea), *oct = (int *)(ws + w.off_doct);
  double *X = (double *)(ws + w.off_x);
  cudaError_t e;
  if ((e = launch_octaves(rdm1, n_ao, false, oct + octaves_len(n_ao), oct, bad, st)) != cudaSuccess) return e;
  launch_next(fx_rdm1_kernel, dim3((unsigned)(w.nb * 4), kin ? 2 : 1), 128, 0, st, rdm1, n_ao, w.nb, oct, dset, dexp,
              bad);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  for (int64_t p0 = 0; p0 < np; p0 += w.dens_slab) {
    const int64_t rows = np - p0 < w.dens_slab ? np - p0 : w.dens_slab;
    const int planes = kin ? 4 : 1;
    if ((e = launch_rows(tab + (size_t)p0 * ld, (int64_t)pe, planes, rows, ld, ld, w.nb, oct, ws + w.off_a, ea, bad,
                         st)) !=
        cudaSuccess)
      return e;
    GemmArgs g{};
    g.a = ws + w.off_a;
    g.b = dset;
    g.b1 = dset + (size_t)w.nb * w.nb * kSetBytes;
    g.ea = ea;
    g.eb = dexp;
    g.eb1 = dexp + w.nb * kTile;
    g.mode = kDensity;
    g.m_tiles = (int)(rows / kTile);
    g.n_tiles = w.nb;
    g.planes = planes;
    g.chunks = g.a_stride = g.b_stride = w.nb;
    g.out = X;
    g.ldc = w.dens_slab;
    g.half_stride = (int64_t)w.nb * 64 * g.ldc;
    g.plane_stride = 2 * g.half_stride;
    g.nt_stride = 64 * g.ldc;
    g.m_valid = rows;
    g.n_valid = n_ao;
    g.bad = bad;
    g.err = err;
    if ((e = launch_gemm(g, st)) != cudaSuccess) return e;
    // Not chained: its blocks would be placed while the GEMM still holds most SMs, and crowd on the rest (24 AOs x
    // 3,600 points: 8 us, chained 24).
    fx_features_kernel<<<(unsigned)(rows / kFeatTile), 256, 0, st>>>(tab, pe, np, ld, n_ao, p0, w.dens_slab, X,
                                                                     w.nb * 64, kin, feat, bad);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t launch_vxc(const double *tab, int64_t np, int ld, int n_ao, const double *coef, bool kin,
                       unsigned char *ws, double *vxc, int *err, cudaStream_t st) {
  const XcWs w = xc_ws(np, n_ao);
  const size_t pe = (size_t)np * ld;
  int *bad = bad_word(ws, w);
  const int n_max = w.mt * kTile;
  int *ea = (int *)(ws + w.off_vexp), *eb = ea + 2 * n_max, *mx = eb + 2 * w.nb * kTile, *g = mx + 6 * n_max, *oct = g + 4;
  unsigned char *va = ws + w.off_va, *vb = ws + w.off_vb;
  double *part = (double *)(ws + w.off_vpart);
  cudaError_t e;
  for (int64_t p0 = 0; p0 < np; p0 += w.v_slab) {
    const int64_t rows = np - p0 < w.v_slab ? np - p0 : w.v_slab;
    const int npc = (int)((rows + kChunkK - 1) / kChunkK);
    launch_next(fx_clear_kernel, (6 * n_max + 4 + 255) / 256, 256, 0, st, p0 == 0 ? bad : nullptr, mx, 6 * n_max + 4);
    launch_next(fx_coef_max_kernel, (unsigned)((rows + 255) / 256), 256, 0, st, coef, np, p0, rows, g);
    const int blocks_a = (ld + 31) / 32;
    int64_t segs = (8 * 148 + blocks_a - 1) / blocks_a;
    int64_t per = (rows + segs - 1) / segs;
    per = per < 64 ? 64 : per;
    segs = (rows + per - 1) / per;
    launch_next(fx_vmax_kernel, dim3(blocks_a, (unsigned)segs), 256, 0, st, tab, pe, np, ld, coef, p0, rows, (int)per,
                kin, n_max, g, mx, oct, w.v_slab, bad);
    launch_next(fx_vdigits_kernel, dim3(3, ld / 32, npc), 256, 0, st, tab, pe, np, ld, coef, p0, rows, npc, kin, w.mt,
                w.nb, (n_ao + 7) / 8 * 8, mx, oct, w.v_slab, ea, eb, va, vb, bad);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    GemmArgs g{};
    g.a = va;
    g.b = g.b1 = vb;
    g.ea = ea;
    g.eb = eb;
    g.eb1 = eb + w.nb * kTile;
    g.mode = kVxc;
    g.m_tiles = w.mt;
    g.n_tiles = w.nb;
    g.planes = kin ? 2 : 1;
    g.chunks = npc;
    g.a_stride = g.b_stride = (kin ? 4 : 1) * npc;
    g.chunks_per_split = w.v_chunks;
    g.ldc = n_max;
    g.half_stride = (int64_t)w.nb * 64 * g.ldc;
    g.split_stride = 2 * g.half_stride;
    g.nt_stride = 64 * g.ldc;
    g.plane_stride = w.s0 * g.split_stride;
    g.m_valid = g.n_valid = n_ao;
    g.out = part;
    g.add = p0 > 0 ? part : nullptr;
    g.bad = bad;
    g.err = err;
    if ((e = launch_gemm(g, st)) != cudaSuccess) return e;
  }
  // The first slab, the longest, writes all s0 + s1 splits.
  launch_next(fx_vreduce_kernel, dim3((n_ao + 31) / 32, n_ao, 2), 256, 0, st, part, w.s0, kin ? w.s1 : 0, n_ao, n_max,
              w.nb * 64, vxc, bad);
  return cudaGetLastError();
}

}  // namespace fx
}  // namespace gdft
