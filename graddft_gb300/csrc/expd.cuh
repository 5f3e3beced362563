// expd.cuh - FP64 exp and expm1 by table for the network's row kernels.
//
// The FP64 pipe issues a warp's operation every 16 clocks an SM, so a row
// kernel's time is its count of FP64 operations, and the library's functions
// were half of it.  Here (the table-driven scheme of P. T. P. Tang, ACM TOMS 15
// (1989) and 18 (1992)) a = (256 k' + j) ln2 / 256 + r with |r| <= ln2 / 512,
// exp(a) = 2^k T_j (1 + p(r)), T_j = 2^(j/256) to twice FP64, p the Taylor
// polynomial of degree 5 (the next term is below 2^-57 of r): 11 operations for
// exp and 12 for expm1, the exponent and index work in integers.  Errors over
// [-707, 0] against quad precision: exp 0.502 ulp at most, expm1 1.40 (1.0 below -ln 2).
#pragma once

namespace gdft {
namespace expd {

// 2^(a/16) and 2^(b/256), a, b = 0..15, as sums of two FP64 numbers.
__constant__ double kCoarse[16][2] = {
    {0x1.0000000000000p+0, 0x0.0p+0},
    {0x1.0b5586cf9890fp+0, 0x1.8a62e4adc610bp-54},
    {0x1.172b83c7d517bp+0, -0x1.19041b9d78a76p-55},
    {0x1.2387a6e756238p+0, 0x1.9b07eb6c70573p-54},
    {0x1.306fe0a31b715p+0, 0x1.6f46ad23182e4p-55},
    {0x1.3dea64c123422p+0, 0x1.ada0911f09ebcp-55},
    {0x1.4bfdad5362a27p+0, 0x1.d4397afec42e2p-56},
    {0x1.5ab07dd485429p+0, 0x1.6324c054647adp-54},
    {0x1.6a09e667f3bcdp+0, -0x1.bdd3413b26456p-54},
    {0x1.7a11473eb0187p+0, -0x1.41577ee04992fp-55},
    {0x1.8ace5422aa0dbp+0, 0x1.6e9f156864b27p-54},
    {0x1.9c49182a3f090p+0, 0x1.c7c46b071f2bep-56},
    {0x1.ae89f995ad3adp+0, 0x1.7a1cd345dcc81p-54},
    {0x1.c199bdd85529cp+0, 0x1.11065895048ddp-55},
    {0x1.d5818dcfba487p+0, 0x1.2ed02d75b3707p-55},
    {0x1.ea4afa2a490dap+0, -0x1.e9c23179c2893p-54},
};
__constant__ double kFine[16][2] = {
    {0x1.0000000000000p+0, 0x0.0p+0},
    {0x1.00b1afa5abcbfp+0, -0x1.4f6b2a7609f71p-55},
    {0x1.0163da9fb3335p+0, 0x1.b61299ab8cdb7p-54},
    {0x1.02168143b0281p+0, -0x1.2bf310fc54eb6p-55},
    {0x1.02c9a3e778061p+0, -0x1.19083535b085dp-56},
    {0x1.037d42e11bbccp+0, 0x1.56811eeade11ap-57},
    {0x1.04315e86e7f85p+0, -0x1.0a31c1977c96ep-54},
    {0x1.04e5f72f654b1p+0, 0x1.4c3793aa0d08dp-55},
    {0x1.059b0d3158574p+0, 0x1.d73e2a475b465p-55},
    {0x1.0650a0e3c1f89p+0, -0x1.5cb7b5799c397p-54},
    {0x1.0706b29ddf6dep+0, -0x1.c91dfe2b13c27p-55},
    {0x1.07bd42b72a836p+0, 0x1.3233454458700p-55},
    {0x1.0874518759bc8p+0, 0x1.186be4bb284ffp-57},
    {0x1.092bdf66607e0p+0, -0x1.68063800a3fd1p-54},
    {0x1.09e3ecac6f383p+0, 0x1.1487818316136p-54},
    {0x1.0a9c79b1f3919p+0, 0x1.5d16c873d1d38p-55},
};

constexpr int kTable = 256;

// Entry j: T_j and the part of 2^(j/256) below it, over T_j.
__device__ __forceinline__ double2 table_entry(int j) {
  const double h1 = kCoarse[j >> 4][0], l1 = kCoarse[j >> 4][1], h2 = kFine[j & 15][0], l2 = kFine[j & 15][1];
  const double p = h1 * h2;
  const double l = fma(h1, h2, -p) + fma(h1, l2, l1 * h2);
  const double t = p + l;
  return make_double2(t, (double)((float)(l - (t - p)) / (float)t));  // 24 of the bits past 2^-53 are plenty
}

// By all threads of a block, which then synchronises.
__device__ __forceinline__ void build_table(double2 *tab) {
  for (int j = threadIdx.x; j < kTable; j += blockDim.x) tab[j] = table_entry(j);
}

// exp(a) = t (1 + r + tail) for |a| < 708; r is exact, tail carries what the
// reduction and the table left over and the polynomial from its square on.
struct Parts {
  double t, r, tail;
};
__device__ __forceinline__ Parts parts(double a, const double2 *tab) {
  constexpr double kMagic = 6755399441055744.0;  // 1.5 2^52: the sum's low word is the rounded integer
  const double s = fma(a, 0x1.71547652b82fep+8, kMagic);  // 256 / ln 2
  const int n = __double2loint(s);
  const double kd = s - kMagic;
  const double2 e = tab[n & (kTable - 1)];
  const double rh = fma(kd, -0x1.62e42fef00000p-9, a);  // ln 2 / 256: 33 bits (exact product), then the rest
  const double c = fma(kd, -0x1.473de6af278edp-42, e.y);
  const double r = rh + c, r2 = r * r;
  double q = fma(r, 1.0 / 120.0, 1.0 / 24.0);
  q = fma(r, q, 1.0 / 6.0);
  q = fma(r, q, 0.5);
  return Parts{__hiloint2double(__double2hiint(e.x) + ((n >> 8) << 20), __double2loint(e.x)), rh, fma(r2, q, c)};
}
__device__ __forceinline__ double exp_of(const Parts &e) { return fma(e.t, e.r + e.tail, e.t); }
// t - 1 is exact from t = 1/2 on, where r is added on its own (the sum may be
// as small as r); below, r + tail loses nothing that t - 1 did not.
__device__ __forceinline__ double expm1_of(const Parts &e) {
  const double w = e.t - 1.0;
  const bool half = __double2hiint(e.t) >= 0x3fe00000;
  return fma(e.t, half ? e.tail : e.r + e.tail, half ? fma(e.t, e.r, w) : w);
}

// Arguments from 708 on (2^k would not be a normal number), infinities and NaN: the caller's.
__device__ __forceinline__ bool tabled(double a) {
  return (unsigned)(__double2hiint(a) & 0x7fffffff) < 0x40862000u;
}
// True for 0 < a < infinity, by the high word (a denormal may read as zero).
__device__ __forceinline__ bool positive(double a) { return (unsigned)(__double2hiint(a) - 1) < 0x7fefffffu; }

// elu(a) and elu'(a) where a is not positive().
__device__ __forceinline__ double elu(double a, const double2 *tab) {
  if (!tabled(a)) return a > 0.0 ? a : expm1(a);
  return expm1_of(parts(a, tab));
}
__device__ __forceinline__ double elu_slope(double a, const double2 *tab) {
  if (!tabled(a)) return a > 0.0 ? 1.0 : exp(a);
  return exp_of(parts(a, tab));
}
__device__ __forceinline__ double2 elu_both(double a, const double2 *tab) {
  if (!tabled(a)) return a > 0.0 ? make_double2(a, 1.0) : make_double2(expm1(a), exp(a));
  const Parts e = parts(a, tab);
  return make_double2(expm1_of(e), exp_of(e));
}

}  // namespace expd
}  // namespace gdft
