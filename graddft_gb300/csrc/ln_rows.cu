// ln_rows.cu - LayerNorm + ELU passes of the FP64 network (first order, and with tangents).
//
//   z = zW + b + h_prev;  xh = (z - mean) rs,  rs = (var + eps)^-1/2,  var = max(0, E[z^2] - mean^2) as flax forms it;
//   a = gamma xh + beta;  h = elu(a)
//
// A row of the hidden width W = 32 PL belongs to one warp, R rows at a time.
// These passes are bound by the FP64 pipe (16 clocks a warp operation on an
// SM; their memory traffic takes a fifth of that), so they are laid out to
// issue as few FP64 operations as there are:
//  - the exponential is taken by table (expd.cuh) and only where a <= 0: a
//    warp lists those elements in shared memory and works through the list 32
//    at a time, the integer work beside the FP64 pipe;
//  - a lane's sums over R rows are folded together (fold_sums: 2 R sums take
//    2 R + 2 additions a lane at R = 4, not 10 R), and a row's root and
//    division are taken once for all R rows;
//  - the forward pass leaves xh where z was, and rs beside it, so the reverse
//    pass starts from them.
// One row a warp and turn, with the library's functions and z read again, took
// 34 and 41 FP64 operations an element; now it is 15 and 16.  16,400 rows of 256:
// forward 250 -> 140 us, reverse 297 -> 148; with tangents, 8,192 rows: 214 ->
// 114 and 256 -> 141.  The pipe is busy for 80 % of the forward pass.
#include "common.cuh"
#include "expd.cuh"
#include "mlp.cuh"

namespace gdft {

namespace {

constexpr int kWarps = 4;
constexpr int kFwdBlocks = 608;  // 4 x 152 SMs

// Sums of NV values over the warp's lanes: the returned value is the total of
// s[lane / (32 / NV)].  Each step halves the values a lane still adds up.
template <int NV>
__device__ __forceinline__ double fold_sums(double (&s)[NV], int lane) {
  int o = 16;
#pragma unroll
  for (int n = NV / 2; n >= 1; n /= 2, o /= 2) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < n; ++i) {
      const double give = up ? s[i] : s[i + n], keep = up ? s[i + n] : s[i];
      s[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
  }
  for (; o >= 1; o /= 2) s[0] += __shfl_xor_sync(0xffffffffu, s[0], o);
  return s[0];
}
// Total i of fold_sums<NV>.
template <int NV>
__device__ __forceinline__ double folded(double x, int i) {
  return __shfl_sync(0xffffffffu, x, i * (32 / NV));
}

// Groups of rows go round the blocks before a block's next warp gets one, so
// that a last round is spread over all SMs.
__device__ __forceinline__ int64_t first_group() { return (int64_t)(threadIdx.x >> 5) * gridDim.x + blockIdx.x; }

// A warp's working elements: E values a lane, element e of lane l at 32 e + l.
template <int E, int OUT>
struct Rows {
  double v[OUT][32 * E];
  uint16_t list[32 * E];
};

// put(j, f(v[0][j])) for every element j that the lanes take.
template <int E, int OUT, class F, class P>
__device__ __forceinline__ void for_listed(Rows<E, OUT> &w, const bool (&take)[E], int lane, F f, P put) {
  int n = 0;
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const unsigned m = __ballot_sync(0xffffffffu, take[e]);
    if (take[e]) w.list[n + __popc(m & ((1u << lane) - 1u))] = (uint16_t)(32 * e + lane);
    n += __popc(m);
  }
  __syncwarp();
  int i = lane;
#pragma unroll 1
  for (; i - lane + 32 < n; i += 64) {  // two chains in flight
    const int j0 = w.list[i], j1 = i + 32 < n ? w.list[i + 32] : j0;
    const auto y0 = f(w.v[0][j0]), y1 = f(w.v[0][j1]);
    put(j0, y0);
    if (j1 != j0) put(j1, y1);
  }
  if (i < n) put(w.list[i], f(w.v[0][w.list[i]]));
  __syncwarp();
}

template <int PL, int R>
__global__ void __launch_bounds__(32 * kWarps, 4)
    ln_elu_fwd_kernel(double *__restrict__ z, const double *__restrict__ b, const double *__restrict__ hprev,
                      const double *__restrict__ gam, const double *__restrict__ bet, double eps, int64_t rows,
                      double *__restrict__ h, double *__restrict__ rs) {
  previous_done();
  constexpr int W = 32 * PL, E = R * PL;
  __shared__ double2 tab[expd::kTable];
  __shared__ Rows<E, 1> work[kWarps];
  expd::build_table(tab);
  __syncthreads();
  const int lane = threadIdx.x & 31;
  Rows<E, 1> &w = work[threadIdx.x >> 5];
  for (int64_t r0 = first_group() * R; r0 < rows;
       r0 += (int64_t)gridDim.x * kWarps * R) {
    const int live = rows - r0 < R ? (int)(rows - r0) : R;
    double v[E], st[2 * R];
#pragma unroll
    for (int q = 0; q < R; ++q) {
      st[q] = st[R + q] = 0.0;
#pragma unroll
      for (int k = 0; k < PL; ++k) {
        const int c = lane + 32 * k;
        const size_t o = (size_t)(r0 + q) * W + c;
        const double x = q < live ? (z[o] + b[c]) + hprev[o] : 0.0;
        v[q * PL + k] = x;
        st[q] += x;
        st[R + q] += x * x;
      }
    }
    const double s = fold_sums<2 * R>(st, lane), o = __shfl_xor_sync(0xffffffffu, s, 16);
    const double mean = (lane < 16 ? s : o) / W;
    const double var = fmax(0.0, (lane < 16 ? o : s) / W - mean * mean);
    const double rsq = rsqrt(var + eps);
    constexpr int kSpan = 32 / (2 * R);  // lanes that hold a row's statistics
    if (lane < 16 && lane % kSpan == 0 && lane / kSpan < live) rs[r0 + lane / kSpan] = rsq;
    bool take[E];
#pragma unroll
    for (int q = 0; q < R; ++q) {
      const double mq = folded<2 * R>(mean, q), rq = folded<2 * R>(rsq, q);
#pragma unroll
      for (int k = 0; k < PL; ++k) {
        const int c = lane + 32 * k, e = q * PL + k;
        const double xh = (v[e] - mq) * rq;
        if (q < live) z[(size_t)(r0 + q) * W + c] = xh;
        const double a = fma(gam[c], xh, bet[c]);
        take[e] = !expd::positive(a);
        w.v[0][32 * e + lane] = a;
      }
    }
    for_listed<E, 1>(w, take, lane, [&](double a) { return expd::elu(a, tab); },
                     [&](int j, double y) { w.v[0][j] = y; });
#pragma unroll
    for (int q = 0; q < R; ++q)
#pragma unroll
      for (int k = 0; k < PL; ++k)
        if (q < live) h[(size_t)(r0 + q) * W + lane + 32 * k] = w.v[0][32 * (q * PL + k) + lane];
  }
}

// Parameter-gradient partials of a block: part[block][0][W] = dL/dgamma, part[block][1][W] = dL/dbeta,
// summed over its warps in warp order.
template <int PL>
__device__ __forceinline__ void store_partials(const double (&pg)[PL], const double (&pb)[PL], double *sacc,
                                               double *__restrict__ part) {
  constexpr int W = 32 * PL;
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();  // sacc lies over the rows' working memory
#pragma unroll
  for (int k = 0; k < PL; ++k) {
    sacc[(wid * 2 + 0) * W + lane + 32 * k] = pg[k];
    sacc[(wid * 2 + 1) * W + lane + 32 * k] = pb[k];
  }
  __syncthreads();
  for (int c = threadIdx.x; c < 2 * W; c += blockDim.x) {
    double s = 0.0;
    for (int w = 0; w < kWarps; ++w) s += sacc[w * 2 * W + c];
    part[(size_t)blockIdx.x * 2 * W + c] = s;
  }
}

// dh (row) -> dz in place: g = dh elu'(a) gamma, dz = rs (g - mean(g) - xh mean(g xh)).
template <int PL, int R>
__global__ void __launch_bounds__(32 * kWarps, 3)
    ln_elu_bwd_kernel(double *__restrict__ dh, const double *__restrict__ xhat, const double *__restrict__ rs,
                      const double *__restrict__ gam, const double *__restrict__ bet, int64_t rows,
                      double *__restrict__ part) {
  previous_done();
  constexpr int W = 32 * PL, E = R * PL;
  __shared__ double2 tab[expd::kTable];
  __shared__ union {
    Rows<E, 1> work[kWarps];
    double sacc[kWarps * 2 * W];
  } sm;
  expd::build_table(tab);
  __syncthreads();
  const int lane = threadIdx.x & 31;
  Rows<E, 1> &w = sm.work[threadIdx.x >> 5];
  double pg[PL], pb[PL];
#pragma unroll
  for (int k = 0; k < PL; ++k) pg[k] = pb[k] = 0.0;
  for (int64_t r0 = first_group() * R; r0 < rows;
       r0 += (int64_t)gridDim.x * kWarps * R) {
    const int live = rows - r0 < R ? (int)(rows - r0) : R;
    double xh[E], d[E], st[2 * R];
    bool take[E];
#pragma unroll
    for (int q = 0; q < R; ++q)
#pragma unroll
      for (int k = 0; k < PL; ++k) {
        const int c = lane + 32 * k, e = q * PL + k;
        const size_t o = (size_t)(r0 + q) * W + c;
        xh[e] = q < live ? xhat[o] : 0.0;
        d[e] = q < live ? dh[o] : 0.0;
        const double a = fma(gam[c], xh[e], bet[c]);
        take[e] = !expd::positive(a);
        w.v[0][32 * e + lane] = take[e] ? a : 1.0;
      }
    for_listed<E, 1>(w, take, lane, [&](double a) { return expd::elu_slope(a, tab); },
                     [&](int j, double y) { w.v[0][j] = y; });
#pragma unroll
    for (int q = 0; q < R; ++q) {
      st[q] = st[R + q] = 0.0;
#pragma unroll
      for (int k = 0; k < PL; ++k) {
        const int e = q * PL + k;
        const double da = d[e] * w.v[0][32 * e + lane];
        pg[k] += da * xh[e];
        pb[k] += da;
        d[e] = da * gam[lane + 32 * k];
        st[q] += d[e];
        st[R + q] += d[e] * xh[e];
      }
    }
    const double s = fold_sums<2 * R>(st, lane) / W;
#pragma unroll
    for (int q = 0; q < R; ++q) {
      const double m1 = folded<2 * R>(s, q), m2 = folded<2 * R>(s, R + q);
      if (q < live) {
        const double rq = rs[r0 + q];
#pragma unroll
        for (int k = 0; k < PL; ++k) {
          const int e = q * PL + k;
          dh[(size_t)(r0 + q) * W + lane + 32 * k] = rq * (d[e] - m1 - xh[e] * m2);
        }
      }
    }
  }
  store_partials<PL>(pg, pb, sm.sacc, part);
}

// With tangents: z~ = z~W + h~_prev, xh~ = rs (z~ - m1 - xh m2) with m1 = mean(z~),
// m2 = mean(xh z~), h~ = elu'(a) gamma xh~.  [xh; xh~] go where Z was, rs and
// rs m2 to st[2][rows].
template <int PL, int R>
__global__ void __launch_bounds__(32 * kWarps, 4)
    ln_elu_tan_fwd_kernel(double *__restrict__ Z, const double *__restrict__ b, const double *__restrict__ Hp,
                          const double *__restrict__ gam, const double *__restrict__ bet, double eps, int64_t rows,
                          double *__restrict__ H, double *__restrict__ stat) {
  previous_done();
  constexpr int W = 32 * PL, E = R * PL;
  __shared__ double2 tab[expd::kTable];
  __shared__ Rows<E, 2> work[kWarps];
  expd::build_table(tab);
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const size_t act = (size_t)rows * W;
  Rows<E, 2> &w = work[threadIdx.x >> 5];
  constexpr int kSpan = 32 / (2 * R);
  for (int64_t r0 = first_group() * R; r0 < rows;
       r0 += (int64_t)gridDim.x * kWarps * R) {
    const int live = rows - r0 < R ? (int)(rows - r0) : R;
    double v[E], t[E], st[2 * R];
#pragma unroll
    for (int q = 0; q < R; ++q) {
      st[q] = st[R + q] = 0.0;
#pragma unroll
      for (int k = 0; k < PL; ++k) {
        const int c = lane + 32 * k, e = q * PL + k;
        const size_t o = (size_t)(r0 + q) * W + c;
        v[e] = q < live ? (Z[o] + b[c]) + Hp[o] : 0.0;
        t[e] = q < live ? Z[act + o] + Hp[act + o] : 0.0;
        st[q] += v[e];
        st[R + q] += v[e] * v[e];
      }
    }
    const double s = fold_sums<2 * R>(st, lane), o = __shfl_xor_sync(0xffffffffu, s, 16);
    const double mean = (lane < 16 ? s : o) / W;
    const double var = fmax(0.0, (lane < 16 ? o : s) / W - mean * mean);
    const double rsq = rsqrt(var + eps);
#pragma unroll
    for (int q = 0; q < R; ++q) {
      const double mq = folded<2 * R>(mean, q), rq = folded<2 * R>(rsq, q);
      st[q] = st[R + q] = 0.0;
#pragma unroll
      for (int k = 0; k < PL; ++k) {
        const int e = q * PL + k;
        v[e] = (v[e] - mq) * rq;
        st[q] += t[e];
        st[R + q] += v[e] * t[e];
      }
    }
    const double m = fold_sums<2 * R>(st, lane) / W, om = __shfl_xor_sync(0xffffffffu, m, 16);
    if (lane < 16 && lane % kSpan == 0 && lane / kSpan < live) {
      stat[r0 + lane / kSpan] = rsq;
      stat[rows + r0 + lane / kSpan] = rsq * om;
    }
    bool take[E];
#pragma unroll
    for (int q = 0; q < R; ++q) {
      const double rq = folded<2 * R>(rsq, q), m1 = folded<2 * R>(m, q), m2 = folded<2 * R>(m, R + q);
#pragma unroll
      for (int k = 0; k < PL; ++k) {
        const int c = lane + 32 * k, e = q * PL + k;
        const double xt = rq * (t[e] - m1 - v[e] * m2);
        if (q < live) {
          Z[(size_t)(r0 + q) * W + c] = v[e];
          Z[act + (size_t)(r0 + q) * W + c] = xt;
        }
        t[e] = gam[c] * xt;
        const double a = fma(gam[c], v[e], bet[c]);
        take[e] = !expd::positive(a);
        w.v[0][32 * e + lane] = a;
        w.v[1][32 * e + lane] = 1.0;
      }
    }
    for_listed<E, 2>(w, take, lane, [&](double a) { return expd::elu_both(a, tab); },
                     [&](int j, double2 y) {
                       w.v[0][j] = y.x;
                       w.v[1][j] = y.y;
                     });
#pragma unroll
    for (int q = 0; q < R; ++q)
#pragma unroll
      for (int k = 0; k < PL; ++k)
        if (q < live) {
          const int e = q * PL + k;
          const size_t oo = (size_t)(r0 + q) * W + lane + 32 * k;
          H[oo] = w.v[0][32 * e + lane];
          H[act + oo] = w.v[1][32 * e + lane] * t[e];
        }
  }
}

// Reverse of that: D = [dL/dh; dL/dh~] -> [dL/dz; dL/dz~] in place.  With
// g = g_a gamma, g~ = g_a~ gamma, means over the row and m' = rs m2:
//   dz~ = rs (g~ - <g~> - xh <g~ xh>)
//   dz  = rs (g - <g> - xh <g xh> - xh (<g~ xh~> - 2 m' <g~ xh>) - <g~ xh> (xh~ + m' xh) - m' (g~ - <g~>))
template <int PL>
__global__ void __launch_bounds__(32 * kWarps, 3)
    ln_elu_tan_bwd_kernel(double *__restrict__ D, const double *__restrict__ X, const double *__restrict__ stat,
                          const double *__restrict__ gam, const double *__restrict__ bet, int64_t rows,
                          double *__restrict__ part) {
  previous_done();
  constexpr int W = 32 * PL;
  __shared__ double2 tab[expd::kTable];
  __shared__ union {
    Rows<PL, 1> work[kWarps];
    double sacc[kWarps * 2 * W];
  } sm;
  expd::build_table(tab);
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const size_t act = (size_t)rows * W;
  Rows<PL, 1> &w = sm.work[threadIdx.x >> 5];
  double pg[PL], pb[PL];
#pragma unroll
  for (int k = 0; k < PL; ++k) pg[k] = pb[k] = 0.0;
  for (int64_t r = first_group(); r < rows; r += (int64_t)gridDim.x * kWarps) {
    double xh[PL], xt[PL], d[PL], dt[PL];
    bool take[PL];
#pragma unroll
    for (int k = 0; k < PL; ++k) {
      const int c = lane + 32 * k;
      const size_t o = (size_t)r * W + c;
      xh[k] = X[o];
      xt[k] = X[act + o];
      d[k] = D[o];
      dt[k] = D[act + o];
      const double a = fma(gam[c], xh[k], bet[c]);
      take[k] = !expd::positive(a);
      w.v[0][c] = take[k] ? a : 1.0;
    }
    for_listed<PL, 1>(w, take, lane, [&](double a) { return expd::elu_slope(a, tab); },
                      [&](int j, double y) { w.v[0][j] = y; });
    double st[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};  // g, g xh, g~, g~ xh, g~ xh~
#pragma unroll
    for (int k = 0; k < PL; ++k) {
      const int c = lane + 32 * k;
      const double e1 = w.v[0][c];
      // elu'' = elu' where a <= 0, else 0 (elu' = 1 there).
      const double ga = (take[k] ? fma(dt[k], gam[c] * xt[k], d[k]) : d[k]) * e1;
      const double gat = dt[k] * e1;
      pg[k] += ga * xh[k] + gat * xt[k];
      pb[k] += ga;
      d[k] = ga * gam[c];
      dt[k] = gat * gam[c];
      st[0] += d[k];
      st[1] += d[k] * xh[k];
      st[2] += dt[k];
      st[3] += dt[k] * xh[k];
      st[4] += dt[k] * xt[k];
    }
    const double s = fold_sums<8>(st, lane) / W;
    const double rq = stat[r], mp = stat[rows + r];
    const double mgt = folded<8>(s, 2), mgtx = folded<8>(s, 3);
    const double c0 = folded<8>(s, 0) - mp * mgt;                    // constant of dz
    const double cx = folded<8>(s, 1) + folded<8>(s, 4) - mp * mgtx;  // factor of xh
#pragma unroll
    for (int k = 0; k < PL; ++k) {
      const size_t o = (size_t)r * W + lane + 32 * k;
      D[o] = rq * (d[k] - c0 - xh[k] * cx - mgtx * xt[k] - mp * dt[k]);
      D[act + o] = rq * (dt[k] - mgt - xh[k] * mgtx);
    }
  }
  store_partials<PL>(pg, pb, sm.sacc, part);
}

unsigned blocks_for(int64_t rows, int group) {  // a block for every group of rows as long as all are resident
  const int64_t n = (rows + group - 1) / group;
  return (unsigned)(n < kFwdBlocks ? n : kFwdBlocks);
}

}  // namespace

#define GDFT_WIDTHS(CALL)          \
  switch (width) {                 \
    case 32: CALL(1); break;       \
    case 64: CALL(2); break;       \
    case 128: CALL(4); break;      \
    case 256: CALL(8); break;      \
    default: return cudaErrorInvalidValue; \
  }                                \
  return cudaGetLastError()

cudaError_t launch_ln_elu_fwd(int width, double *z, const double *b, const double *hprev, const double *gam,
                              const double *bet, double eps, int64_t rows, double *h, double *rs, cudaStream_t st) {
#define GDFT_FWD(PL) \
  launch_next(ln_elu_fwd_kernel<PL, 4>, blocks_for(rows, 4), 32 * kWarps, 0, st, z, b, hprev, gam, bet, eps, rows, h, \
              rs)
  GDFT_WIDTHS(GDFT_FWD);
#undef GDFT_FWD
}

cudaError_t launch_ln_elu_bwd(int width, double *dh, const double *xhat, const double *rs, const double *gam,
                              const double *bet, int64_t rows, double *part, cudaStream_t st) {
#define GDFT_BWD(PL) \
  launch_next(ln_elu_bwd_kernel<PL, 2>, kLnRowBlocks, 32 * kWarps, 0, st, dh, xhat, rs, gam, bet, rows, part)
  GDFT_WIDTHS(GDFT_BWD);
#undef GDFT_BWD
}

cudaError_t launch_ln_elu_tan_fwd(int width, double *Z, const double *b, const double *Hp, const double *gam,
                                  const double *bet, double eps, int64_t rows, double *H, double *stat,
                                  cudaStream_t st) {
#define GDFT_FWD(PL) \
  launch_next(ln_elu_tan_fwd_kernel<PL, 2>, blocks_for(rows, 2), 32 * kWarps, 0, st, Z, b, Hp, gam, bet, eps, rows, H, \
              stat)
  GDFT_WIDTHS(GDFT_FWD);
#undef GDFT_FWD
}

cudaError_t launch_ln_elu_tan_bwd(int width, double *D, const double *X, const double *stat, const double *gam,
                                  const double *bet, int64_t rows, double *part, cudaStream_t st) {
#define GDFT_BWD(PL) \
  launch_next(ln_elu_tan_bwd_kernel<PL>, kLnRowBlocks, 32 * kWarps, 0, st, D, X, stat, gam, bet, rows, part)
  GDFT_WIDTHS(GDFT_BWD);
#undef GDFT_BWD
}

#undef GDFT_WIDTHS

}  // namespace gdft
