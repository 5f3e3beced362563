// fx.cuh - FP64 contractions as exact sums of 9-bit digit products on the tensor cores.
//
// GB300 runs FP64 at 2 FMAs per clock and SM but BF16 tensor products at 4096.
// An FP64 operand row x_k is written as fixed point on the row's own exponent
// (|x_k| < 2^e, the largest at least 2^(e-1)):
//   x_k = 2^e * sum_{i<7} d_i 2^(-7-9i) + r,   d_i integers, |d_0| <= 128, |d_i| <= 256,
// |r| <= 2^(e-62): every value within 2^9 of the row's largest keeps all its 53
// bits.  The product of two rows is then sum_{i,j} 2^(-9(i+j)) sum_k a_i b_j, and
// the pairs i + j <= 6 (28 of 49; the rest is below 2^-58 of the product of the rows' 2^e, in the mean
// below 2^-60) are BF16 tensor-core GEMMs whose operands hold d_i 2^(-9i) exactly (the
// splitting of Ozaki, Ogita, Oishi and Rump, "Error-free transformations of
// matrix multiplication", 2012).  For i + j <= 4 a 64-term chunk's sum is an
// integer multiple of 2^(-9(i+j)) of at most 2^24, so FP32 accumulation is exact
// whatever the tensor core's alignment; the chunk sums are added as integers.  The thirteen pairs of i + j = 5, 6 (below
// 2^-45 of the result) share one FP32 accumulator.
//
// The error is therefore relative to the product of the rows' largest values, where an
// FP64 sum's is relative to the sum of the terms' sizes.  The two are close for rows of values that are
// alike.  Where operands are graded against one another, exact powers of two for each k level them first
// (octaves: a_k 2^t, b_k 2^-t; fx_xc.cu), in the density, V_xc, exact exchange and chi.  The network's do
// without: its hidden values are of order one, and max |h| max |dz| was at most 2.3
// times sum |h dz| in the weight gradients of 16,400 points with densities over 20 decades.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace gdft {
namespace fx {

constexpr int kDigits = 7;
constexpr int kChunkK = 64;                          // contraction length of one chunk
constexpr int kTile = 128;                           // operand rows of one block
constexpr uint32_t kBlockBytes = kTile * kChunkK * 2;  // one digit of a 128 x 64 block, 16 KB
constexpr uint32_t kSetBytes = kDigits * kBlockBytes;  // all digits of a block, 112 KB

// Byte offset of element (row, k) in a digit block: core matrices of 8 rows x
// 16 bytes, adjacent along k at 128 bytes and along rows at 1024.
__host__ __device__ constexpr uint32_t elem_off(int row, int k) {
  return (uint32_t)(((row >> 3) * 8 + (k >> 3)) * 128 + (row & 7) * 16 + (k & 7) * 2);
}

// Biased exponent field of |x| from the high word (0 for zeros and denormals).
__device__ __forceinline__ int exp_field(uint32_t hi) { return (int)((hi >> 20) & 0x7FFu); }

// x as fixed point on a row whose largest biased exponent field is emax (of x, so less
// its octaves; fields of 0 count as 1): an integer of magnitude <= 2^61, unit 2^(emax - 1083).
__device__ __forceinline__ long long to_fixed(double x, int emax) {
  const long long b = __double_as_longlong(x);
  const int ef = (int)((unsigned long long)b >> 52) & 0x7FF;
  unsigned long long m = (unsigned long long)b & 0xFFFFFFFFFFFFFull;
  if (ef) m |= 1ull << 52;
  m <<= 8;
  int sh = emax - (ef ? ef : 1);
  sh = sh > 63 ? 63 : sh;
  if (sh > 0) m = (m + (1ull << (sh - 1))) >> sh;
  return b < 0 ? -(long long)m : (long long)m;
}

// Octaves t of a term k that is taken as (a_k 2^t)(b_k 2^-t), where b_k is zero: a_k 2^t has no digits.
constexpr int kDead = -(1 << 14);

// The digits of a row's fixed-point values, eight consecutive k at a time:
// out[i] holds digit i times 2^(-9i) of the eight values as BF16.
__device__ __forceinline__ void digits8(const long long (&f)[8], uint4 (&out)[kDigits]) {
  constexpr long long kBias =
      256ll + (256ll << 9) + (256ll << 18) + (256ll << 27) + (256ll << 36) + (256ll << 45);
  constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23: integers become mantissa bits
#pragma unroll
  for (int h = 0; h < 4; ++h) {
    const unsigned long long u0 = (unsigned long long)(f[2 * h] + kBias), u1 = (unsigned long long)(f[2 * h + 1] + kBias);
#pragma unroll
    for (int i = 0; i < kDigits; ++i) {
      const float scale = __uint_as_float((uint32_t)(127 - 9 * i) << 23);
      float a, b;
      if (i == 0) {  // top digit, signed, -128 .. 128
        a = __int_as_float(0x4B400000 + (int)((long long)u0 >> 54)) - kMagic;
        b = __int_as_float(0x4B400000 + (int)((long long)u1 >> 54)) - kMagic;
      } else {
        const int s = 9 * (kDigits - 1 - i);
        const float off = -(kMagic + 256.0f) * scale;
        a = fmaf(__uint_as_float(0x4B400000u | ((uint32_t)(u0 >> s) & 511u)), scale, off);
        b = fmaf(__uint_as_float(0x4B400000u | ((uint32_t)(u1 >> s) & 511u)), scale, off);
      }
      // Exact in BF16: the upper halves of the FP32 words.
      (&out[i].x)[h] = __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);
    }
  }
}

// Largest exponent field of an operand row: beyond it (2^450, or not finite) the
// plain kernels take over, which also keeps the products within range.
constexpr int kMaxField = 1023 + 450;

// v 2^scale as a double, rounded to nearest (halves away from zero), by integer
// operations: conversions run at the FP64 rate.  Below 2^-1022 the result is 0.
__device__ __forceinline__ double fixed_to_double(long long v, int scale) {
  const unsigned long long m = v < 0 ? (unsigned long long)(-v) : (unsigned long long)v;
  const int lz = __clzll((long long)m);
  const unsigned long long n = m << (lz & 63);               // leading one at bit 63
  const unsigned long long r = (n >> 11) + ((n >> 10) & 1);  // 53 bits, may carry to 2^53
  const int e = 63 - lz + scale;                             // exponent of the leading one
  unsigned long long d = ((unsigned long long)(e + 1022) << 52) + r;
  if (e < -1022 || v == 0) return 0.0;
  return __longlong_as_double((long long)(d | ((unsigned long long)v & 0x8000000000000000ull)));
}

// What the items (output tiles over a range of K chunks) of a launch are.
enum Mode {
  kFull = 0,     // out[split][m tile][n tile] of A B^T, the K chunks split evenly
  kDensity = 1,  // A planes 0..3: plane 0 over all chunks against b, planes 1..3 over chunks 0..n tile against b1
  kVxc = 2,      // "plane" 0: chunks 0..chunks-1 of every tile; "plane" 1: the 3 chunks after them, only the tiles
                 // whose 64-column block reaches the diagonal (64 nt + 63 >= 128 mt; the product is symmetric)
};

struct GemmArgs {
  const unsigned char *a, *b;  // digit sets [tile][chunk][7][16 KB]
  const unsigned char *b1;     // kDensity: operand of planes 1..3
  const int *ea, *eb, *eb1;    // exponent field of each operand row (emax of to_fixed)
  int mode;
  int m_tiles, n_tiles;
  int planes;                  // kDensity: 1 or 4; kVxc: 1 or 2
  int chunks;                  // K chunks of a tile (kVxc: of plane 0; plane 1 has three times as many)
  int a_stride, b_stride;      // sets between consecutive tiles
  int chunks_per_split;
  double *out;                 // row r, column c of half h (columns 64 h .. of a tile): out + split_stride split
  int64_t ldc;                 //   + plane_stride plane + half_stride h + nt_stride nt + ldc c + r (lanes are rows)
  int64_t half_stride, nt_stride, split_stride, plane_stride;
  int64_t m_valid, n_valid;    // rows of A and of B (kDensity, kVxc: B's per spin) with values; only their products
                               // are formed and written, and only their digits need to be there (to a multiple of 8)
  const double *add;           // added to the result, laid out like out (may be out itself), or null
  const int *bad;              // non-zero: an operand is not finite, nothing to do
  int *err;
};

cudaError_t launch_gemm(const GemmArgs &a, cudaStream_t st);

// Row-major FP64 rows (planes of them, k_valid values each) -> digit sets [plane][row tile][chunk], exponents
// [plane][rows].  Rows past the last are left as they are: they only reach outputs that are not written.  oct, or
// null: 64 chunks octaves t <= 0, aligned to 16 bytes; column k is taken times 2^t.
cudaError_t launch_rows(const double *src, int64_t plane_elems, int planes, int64_t rows, int64_t ld, int k_valid,
                        int chunks, const int *oct, unsigned char *out, int *exps, int *bad, cudaStream_t st);

// FP64 GEMMs of fx_mat.cu, on row-major operands.  ws: scratch of gemm_rows_bytes / gemm_cols_bytes; err: the device
// word that an expired wait is recorded in (it also leaves NaN in the output); part: partials of the plain kernel that
// takes over where an operand is not finite (nsplit x M x N doubles).
size_t gemm_rows_bytes(int64_t M, int N, int K);
size_t gemm_cols_bytes(int M, int N, int64_t K);
// C[m][n] = sum_k A[m][k] B[k][n] (B stored N x K when b_rows) + add[m][n] (laid out like C; null: nothing).  oct, or
// null (it has to be with b_rows): octaves_len(K) octaves t <= 0, aligned to 16 bytes; A's columns are taken times 2^t, B's
// rows times 2^-t.
cudaError_t gemm_rows(int64_t M, int N, int K, const double *A, int64_t lda, const double *B, int64_t ldb, bool b_rows,
                      const int *oct, double *C, int64_t ldc, const double *add, unsigned char *ws, int *err, cudaStream_t st);
// C[m][n] = sum_k A[k][m] B[k][n], C contiguous (M x N).  oct, or null: K octaves t; A's rows are taken times 2^t and
// B's times 2^-t, for operands that are graded against one another (fx_xc.cu).
cudaError_t gemm_cols(int M, int N, int64_t K, const double *A, int64_t lda, const double *B, int64_t ldb,
                      const int *oct, double *C, unsigned char *ws, int *err, int nsplit, double *part,
                      cudaStream_t st);

// Octaves of the AOs for products of AO values with D (2, n, n), fx_xc.cu: octaves_len(n) for both spins together, or
// (each) for either.  mx: 2 octaves_len(n) integers of scratch; bad: a word to clear, or null.
inline int octaves_len(int n) { return (n + 63) / 64 * 64; }
cudaError_t launch_octaves(const double *D, int n, bool each, int *mx, int *oct, int *bad, cudaStream_t st);

// Feature sets of fx_xc.cu: the FP64 form's density and V_xc contractions.
struct XcWs {
  int nb, mt;              // 64-column blocks, 128-row tiles of the AOs
  int64_t dens_slab, v_slab;  // grid points per pass (multiples of 128)
  int v_chunks;            // K chunks of one V_xc item
  int s0, s1;              // splits of the phi and kinetic parts of a full slab
  size_t off_bad, off_dset, off_dexp, off_doct, off_a, off_ea, off_x;  // density
  size_t off_va, off_vb, off_vexp, off_vpart;                          // V_xc
  size_t bytes;
};
XcWs xc_ws(int64_t np, int n_ao);
// kin: the Laplacian and tau are wanted (planes d_x, d_y, d_z contracted too); otherwise they are set to 0.
cudaError_t launch_density(const double *tab, int64_t np, int ld, int n_ao, const double *rdm1, bool kin, double *feat,
                           unsigned char *ws, int *err, cudaStream_t st);
// kin: coef's C_KIN rows may be non-zero.
cudaError_t launch_vxc(const double *tab, int64_t np, int ld, int n_ao, const double *coef, bool kin,
                       unsigned char *ws, double *vxc, int *err, cudaStream_t st);
// The word that says an operand of the last density / V_xc was not finite.
inline int *bad_word(unsigned char *ws, const XcWs &w) { return (int *)(ws + w.off_bad); }

}  // namespace fx
}  // namespace gdft
