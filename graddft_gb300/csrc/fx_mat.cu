// fx_mat.cu - general FP64 GEMMs on the digit products of fx_gemm.cu: the network's
// layers and weight gradients, the exact-exchange and chi contractions.
//
// gemm_rows: C = A op(B) for a tall A (points x width).  The tall operand takes
// the kernel's column side and the small one its row side, so that a drain's
// lanes write consecutive entries of a row of C.  gemm_cols: C = A^T B over many
// rows, split over the SMs, partials summed in order.  Operands that are not
// finite go to the plain kernel, slab by slab.
//
// Measured (plain FP64 GEMM -> here, with the digits' kernels): a layer of the
// network, 16,512 x 256 x 256, 1,430 -> 95 us; its weight gradient (K 16,512),
// which ran on 16 CTAs, 17,800 -> 95 us.  A DM21 training step on 16,400 points:
// 177.3 -> 7.9 ms, the second-order pass on 8,192: 260 -> 11.6 ms (5.6 and 8.3
// with the row passes of ln_rows.cu and chained launches).
#include "common.cuh"
#include "fx.cuh"
#include "kernels.cuh"
#include "mlp_gemm.cuh"

namespace gdft {
namespace fx {

namespace {

constexpr size_t kSlabBytes = (size_t)512 << 20;  // digits held at a time, about
constexpr uint32_t kInfHi = 0x7FF00000u;  // high word of an infinity
constexpr size_t align256(size_t x) { return (x + 255) / 256 * 256; }
constexpr int64_t tiles_of(int64_t n) { return (n + kTile - 1) / kTile; }
constexpr int64_t chunks_of(int64_t k) { return (k + kChunkK - 1) / kChunkK; }

// Columns of a short row-major matrix X [k_rows][cols] as operand rows (weights,
// density matrices), with oct row k times 2^-oct[k]: a warp takes eight columns, lane =
// (column, eight k), both passes over k in one kernel.
__global__ void __launch_bounds__(128) fx_short_cols_kernel(const double *__restrict__ X, int k_rows, int cols,
                                                            int64_t ld, int chunks, const int *__restrict__ oct,
                                                            unsigned char *__restrict__ out, int *__restrict__ exps,
                                                            int *__restrict__ bad) {
  previous_done();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c0 = (blockIdx.x * 4 + warp) * 8;
  if (c0 >= cols) return;
  const int c = c0 + (lane & 7), kg = (lane >> 3) * 8;
  auto value = [&](int k) { return c < cols && k < k_rows ? X[(size_t)k * ld + c] : 0.0; };
  int m = 0;
  for (int k = kg; k < k_rows; k += 32)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int h = __double2hiint(value(k + j)) & 0x7FFFFFFF;
      if (h != 0) m = max(m, oct != nullptr ? h - oct[k + j] * (1 << 20) : h);
    }
  m = max(m, __shfl_xor_sync(0xffffffffu, m, 8));
  m = max(m, __shfl_xor_sync(0xffffffffu, m, 16));
  int emax = m >> 20;
  if (emax > kMaxField) atomicOr(bad, 1);
  if (emax < 1) emax = 1;
  if (lane < 8 && c < cols) exps[c] = emax;
  unsigned char *base = out + (size_t)(c / kTile) * chunks * kSetBytes;
  for (int k = kg; k < chunks * kChunkK; k += 32) {
    long long f[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = to_fixed(value(k + j), oct != nullptr ? emax + oct[k + j] : emax);
    uint4 d[kDigits];
    digits8(f, d);
    unsigned char *set = base + (size_t)(k / kChunkK) * kSetBytes + elem_off(c % kTile, k % kChunkK);
#pragma unroll
    for (int i = 0; i < kDigits; ++i) *(uint4 *)(set + (size_t)i * kBlockBytes) = d[i];
  }
}

// Largest high words of the columns of X [rows][cols], with OCT those of row r times 2^(sign oct[r]): lanes are
// columns, a block takes 32 of them and `per` rows.
template <bool OCT>
__global__ void __launch_bounds__(256) fx_colmax_kernel(const double *__restrict__ X, int64_t rows, int cols,
                                                        int64_t ld, int64_t per, const int *__restrict__ oct, int sign,
                                                        uint32_t *__restrict__ mx) {
  previous_done();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c = blockIdx.x * 32 + lane;
  const int64_t r0 = (int64_t)blockIdx.y * per, r1 = r0 + per < rows ? r0 + per : rows;
  uint32_t m = 0;
  if (c < cols)
    for (int64_t r = r0 + warp; r < r1; r += 8) {
      uint32_t h = (uint32_t)__double2hiint(X[(size_t)r * ld + c]) & 0x7FFFFFFFu;
      if (OCT && h < kInfHi && h != 0) {  // infinities and NaN stay what they are
        const int t = oct[r];
        const long long v = t == kDead ? 0 : (long long)h + (long long)(sign * t) * (1 << 20);
        h = v < 0 ? 0u : v > kInfHi ? kInfHi : (uint32_t)v;
      }
      m = max(m, h);
    }
  __shared__ uint32_t sm[8][32];
  sm[warp][lane] = m;
  __syncthreads();
  if (warp == 0 && c < cols) {
#pragma unroll
    for (int w = 1; w < 8; ++w) m = max(m, sm[w][lane]);
    atomicMax(mx + c, m);
  }
}

// Columns of a tall X as operand rows, K = its rows (times 2^(sign oct)): a block takes 64
// rows (one chunk) and 32 columns, a warp eight consecutive rows.
template <bool OCT>
__global__ void __launch_bounds__(256) fx_tall_cols_kernel(const double *__restrict__ X, int64_t rows, int cols,
                                                           int64_t ld, int chunks, const int *__restrict__ oct,
                                                           int sign, const uint32_t *__restrict__ mx,
                                                           unsigned char *__restrict__ out, int *__restrict__ exps,
                                                           int *__restrict__ bad) {
  previous_done();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c = blockIdx.y * 32 + lane, chunk = blockIdx.x;
  int emax = c < cols ? exp_field(mx[c]) : 1;
  if (emax > kMaxField) atomicOr(bad, 1);
  if (emax < 1) emax = 1;
  if (chunk == 0 && warp == 0 && c < cols) exps[c] = emax;
  const int64_t r0 = (int64_t)chunk * kChunkK + warp * 8;
  long long f[8];
#pragma unroll
  for (int j = 0; j < 8; ++j)
    f[j] = c < cols && r0 + j < rows
               ? to_fixed(X[(size_t)(r0 + j) * ld + c], OCT ? emax - sign * oct[r0 + j] : emax)
               : 0;
  uint4 d[kDigits];
  digits8(f, d);
  unsigned char *set = out + ((size_t)(c / kTile) * chunks + chunk) * kSetBytes + elem_off(c % kTile, warp * 8);
#pragma unroll
  for (int i = 0; i < kDigits; ++i) *(uint4 *)(set + (size_t)i * kBlockBytes) = d[i];
}

// C[i] = sum over splits of part[split][i].
__global__ void fx_sum_kernel(const double *__restrict__ part, int nsplit, size_t total, size_t stride,
                              double *__restrict__ C, const int *__restrict__ bad) {
  previous_done();
  if (*bad != 0) return;
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= total) return;
  double s = 0.0;
  for (int k = 0; k < nsplit; ++k) s += part[(size_t)k * stride + i];
  C[i] = s;
}

struct RowsWs {
  int64_t slab;  // rows of A at a time
  size_t off_b, off_eb, off_a, off_ea, bytes;
};
RowsWs rows_ws(int64_t M, int N, int K) {
  RowsWs w;
  const int64_t ch = chunks_of(K);
  w.slab = (int64_t)kSlabBytes / ((int64_t)kSetBytes * ch) * kTile;
  w.slab = w.slab < kTile ? kTile : w.slab;
  if (w.slab > tiles_of(M) * kTile) w.slab = tiles_of(M) * kTile;
  size_t off = 256;  // the bad word
  w.off_b = off;
  off = align256(off + (size_t)tiles_of(N) * ch * kSetBytes);
  w.off_eb = off;
  off = align256(off + (size_t)tiles_of(N) * kTile * sizeof(int));
  w.off_a = off;
  off = align256(off + (size_t)(w.slab / kTile) * ch * kSetBytes);
  w.off_ea = off;
  off = align256(off + (size_t)w.slab * sizeof(int));
  w.bytes = off;
  return w;
}

struct ColsWs {
  int64_t slab;  // rows (K) at a time
  int per, splits;
  size_t off_mx, off_exp, off_a, off_b, off_part, bytes;
};
ColsWs cols_ws(int M, int N, int64_t K) {
  ColsWs w;
  const int64_t tm = tiles_of(M), tn = tiles_of(N);
  w.slab = (int64_t)kSlabBytes / ((int64_t)kSetBytes * (tm + tn)) * kChunkK;
  w.slab = w.slab < 16 * kChunkK ? 16 * kChunkK : w.slab;
  if (w.slab > chunks_of(K) * kChunkK) w.slab = chunks_of(K) * kChunkK;
  // One round of one CTA per SM, at least four chunks an item.
  const int64_t ch = w.slab / kChunkK;
  int64_t per = (ch * tm * tn + 147) / 148;
  per = per < 4 ? 4 : per;
  w.per = (int)per;
  w.splits = (int)((ch + per - 1) / per);
  size_t off = 256;
  w.off_mx = off;
  off = align256(off + (size_t)(tm + tn) * kTile * sizeof(uint32_t));
  w.off_exp = off;
  off = align256(off + (size_t)(tm + tn) * kTile * sizeof(int));
  w.off_a = off;
  off = align256(off + (size_t)tm * ch * kSetBytes);
  w.off_b = off;
  off = align256(off + (size_t)tn * ch * kSetBytes);
  w.off_part = off;
  // splits is at most 148 / (tm tn) + 1 for any K: a shorter K never needs more.
  off = align256(off + (size_t)(148 / (tm * tn) + 1) * M * N * sizeof(double));
  w.bytes = off;
  return w;
}

}  // namespace

// Callers' workspaces may be aligned to 8 bytes only; the copies need 16.
static unsigned char *aligned(unsigned char *ws) { return (unsigned char *)(((uintptr_t)ws + 255) & ~(uintptr_t)255); }
size_t gemm_rows_bytes(int64_t M, int N, int K) { return rows_ws(M, N, K).bytes + 256; }
size_t gemm_cols_bytes(int M, int N, int64_t K) { return cols_ws(M, N, K).bytes + 256; }

cudaError_t gemm_rows(int64_t M, int N, int K, const double *A, int64_t lda, const double *B, int64_t ldb, bool b_rows,
                      const int *oct, double *C, int64_t ldc, const double *add, unsigned char *ws, int *err,
                      cudaStream_t st) {
  if (b_rows && oct != nullptr) return cudaErrorInvalidValue;
  const RowsWs w = rows_ws(M, N, K);
  const int ch = (int)chunks_of(K);
  ws = aligned(ws);
  int *bad = (int *)ws, *ew = (int *)(ws + w.off_eb), *ex = (int *)(ws + w.off_ea);
  unsigned char *sw = ws + w.off_b, *sx = ws + w.off_a;
  cudaError_t e;
  for (int64_t m0 = 0; m0 < M; m0 += w.slab) {
    const int64_t rows = M - m0 < w.slab ? M - m0 : w.slab;
    if ((e = cudaMemsetAsync(bad, 0, sizeof(int), st)) != cudaSuccess) return e;
    if (b_rows)
      e = launch_rows(B, 0, 1, N, ldb, K, ch, nullptr, sw, ew, bad, st);
    else {
      launch_next(fx_short_cols_kernel, (N + 31) / 32, 128, 0, st, B, K, N, ldb, ch, oct, sw, ew, bad);
      e = cudaGetLastError();
    }
    if (e != cudaSuccess) return e;
    if ((e = launch_rows(A + m0 * lda, 0, 1, rows, lda, K, ch, oct, sx, ex, bad, st)) != cudaSuccess) return e;
    GemmArgs g{};
    g.a = sw;
    g.b = g.b1 = sx;
    g.ea = ew;
    g.eb = g.eb1 = ex;
    g.mode = kFull;
    g.m_tiles = (int)tiles_of(N);
    g.n_tiles = (int)tiles_of(rows);
    g.planes = 1;
    g.chunks = g.a_stride = g.b_stride = g.chunks_per_split = ch;
    g.out = C + m0 * ldc;
    g.ldc = ldc;
    g.half_stride = 64 * ldc;
    g.nt_stride = kTile * ldc;
    g.m_valid = N;
    g.n_valid = rows;
    g.add = add != nullptr ? add + m0 * ldc : nullptr;
    g.bad = bad;
    g.err = err;
    if ((e = launch_gemm(g, st)) != cudaSuccess) return e;
    e = b_rows ? plain_gemm<kNT>((int)rows, N, K, A + m0 * lda, (int)lda, B, (int)ldb, C + m0 * ldc, (int)ldc,
                                 g.add, bad, st)
               : plain_gemm<kNN>((int)rows, N, K, A + m0 * lda, (int)lda, B, (int)ldb, C + m0 * ldc, (int)ldc,
                                 g.add, bad, st);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t gemm_cols(int M, int N, int64_t K, const double *A, int64_t lda, const double *B, int64_t ldb,
                      const int *oct, double *C, unsigned char *ws, int *err, int nsplit, double *part,
                      cudaStream_t st) {
  const ColsWs w = cols_ws(M, N, K);
  const int64_t tm = tiles_of(M), tn = tiles_of(N);
  ws = aligned(ws);
  int *bad = (int *)ws, *ea = (int *)(ws + w.off_exp), *eb = ea + tm * kTile;
  uint32_t *ma = (uint32_t *)(ws + w.off_mx), *mb = ma + tm * kTile;
  double *fpart = (double *)(ws + w.off_part);
  cudaError_t e = cudaMemsetAsync(bad, 0, sizeof(int), st);
  if (e != cudaSuccess) return e;
  for (int64_t k0 = 0; k0 < K; k0 += w.slab) {
    const int64_t rows = K - k0 < w.slab ? K - k0 : w.slab;
    const int ch = (int)chunks_of(rows);
    if ((e = cudaMemsetAsync(ma, 0, (size_t)(tm + tn) * kTile * sizeof(uint32_t), st)) != cudaSuccess) return e;
    const int *o = oct != nullptr ? oct + k0 : nullptr;
    auto digits = [&](const double *X, int64_t ld, int cols, int sign, uint32_t *mx, unsigned char *set, int *exps) {
      const int bc = (cols + 31) / 32;
      int64_t segs = (4 * 148 + bc - 1) / bc, per = (rows + segs - 1) / segs;
      per = per < 64 ? 64 : per;
      segs = (rows + per - 1) / per;
      launch_next(o != nullptr ? fx_colmax_kernel<true> : fx_colmax_kernel<false>, dim3(bc, (unsigned)segs), 256, 0,
                  st, X + k0 * ld, rows, cols, ld, per, o, sign, mx);
      launch_next(o != nullptr ? fx_tall_cols_kernel<true> : fx_tall_cols_kernel<false>, dim3(ch, bc), 256, 0, st,
                  X + k0 * ld, rows, cols, ld, ch, o, sign, mx, set, exps, bad);
      return cudaGetLastError();
    };
    if ((e = digits(A, lda, M, 1, ma, ws + w.off_a, ea)) != cudaSuccess) return e;
    if ((e = digits(B, ldb, N, -1, mb, ws + w.off_b, eb)) != cudaSuccess) return e;
    GemmArgs g{};  // rows of the tiles: columns n of B (consecutive in C); columns: m
    g.a = ws + w.off_b;
    g.b = g.b1 = ws + w.off_a;
    g.ea = eb;
    g.eb = g.eb1 = ea;
    g.mode = kFull;
    g.m_tiles = (int)tn;
    g.n_tiles = (int)tm;
    g.planes = 1;
    g.chunks = g.a_stride = g.b_stride = ch;
    g.chunks_per_split = w.per;
    g.out = fpart;
    g.ldc = N;
    g.half_stride = (int64_t)64 * N;
    g.nt_stride = (int64_t)kTile * N;
    g.split_stride = (int64_t)M * N;
    g.m_valid = N;
    g.n_valid = M;
    g.add = k0 > 0 ? fpart : nullptr;
    g.bad = bad;
    g.err = err;
    if ((e = launch_gemm(g, st)) != cudaSuccess) return e;
  }
  const size_t total = (size_t)M * N;
  launch_next(fx_sum_kernel, (unsigned)((total + 255) / 256), 256, 0, st, fpart, w.splits, total, total, C, bad);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  return plain_gemm_tn_split(M, N, K, A, (int)lda, B, (int)ldb, C, nsplit, part, bad, st);
}

}  // namespace fx
}  // namespace gdft
