// fx_gemm.cu - the digit-product GEMM of fx.cuh on tcgen05 (kind::f16, BF16 operands).
//
// One CTA per SM walks 128 x 128 output tiles (items) with one continuous
// pipeline.  A K chunk of 64 is seven 16 KB digit blocks of A and seven of B, one
// slot each; a slot is refilled for the next chunk as soon as its digit's last
// product is issued and done.  B's blocks are adjacent, so one MMA of N 256 forms
// A_i B_j and A_i B_(j+1), two neighbouring orders i + j, in adjacent TMEM
// columns: 72 MMAs a chunk instead of 112, reading 12 KB of shared memory in
// 128 clocks where N 128 reads 8 KB in 64 (the limit is 128 B per clock).
// TMEM: orders (0, 1), (2, 3) and then 4 pass through the accumulators L and H,
// which the drain warps read as integers; orders 5 and 6 stay in Z5 and Z6 for up
// to 16 chunks (450 truncations of 2^-24 of a part below 2^-45 of the result).
// The products of orders 5 and 6 are issued between those of L and H, which gives
// a drain about 1,300 clocks (float-to-integer conversions run at 16 per clock:
// 1,024 for one order), and in an order that frees the digits a chunk starts with
// six pairs before its end.  Few waits: each leaves the tensor core idle for some 110
// clocks, so a chunk's blocks arrive in three groups and the drains' releases count
// towards two of them.
//
// What bounds it: 28 digit pairs take 7,168 clocks a chunk at the dense BF16 rate.
// Measured with 38,912 rows, K 1,024, N 128 (A read from HBM): 11,020 clocks a
// chunk (12,400 while the copies were issued in a loop, 11,200 with eight waits a
// chunk instead of four), of which the copies take
// about 1,500, the drains 1,300 and an item's output 1,200; 55 TFLOP/s of FP64
// products, where the FP64 pipe gives 1.1.  An item's output costs some 16,000
// clocks whatever its K (24 bytes a thread are spilled, outside the chunk's loop).  Error against quadruple
// precision 4.7e-17 (a sequential FP64 sum: 1.1e-15).
//
// Warp roles (384 threads): warp 0 producer (one thread), warp 1 TMEM owner and
// MMA issuer (one thread), warps 4-11 drains, one per (lane quadrant, 64 columns).
// A drain thread holds 64 64-bit sums: the two drain warpgroups take 216 registers
// a thread, the first gives up all but 72 (72 + 2 x 216 = 3 x 168).  Every wait is
// bounded (umma::mbar_wait); on expiry the CTA records an error word, lets its
// copies and MMAs land and releases TMEM.
#include "common.cuh"
#include "fx.cuh"
#include "umma.cuh"

namespace gdft {
namespace fx {

namespace {

constexpr int kThreads = 384;
constexpr int kDrains = 8;  // drain warps
constexpr int kCols = 64;   // columns of one
constexpr uint32_t kTmemCols = 512;  // L [0,128), H [128,256), Z5 [256,384), Z6 [384,512)
constexpr uint32_t kZcol = 256;
constexpr int kSmemBytes = 2 * kSetBytes + 1024;  // digits of A, then of B
constexpr int kRowsPerWarp = 4;  // of fx_rows_kernel
constexpr int kSumChunks = 16;  // chunks of one 64-bit sum, then it is added to the output

// A chunk's blocks (0-6: A's digits, 7-13: B's) arrive in groups, in the order in
// which they are first read; a group's slots are free again together.
constexpr int kGroups = 3;
__device__ constexpr int kGroupOf[2 * kDigits] = {0, 7, 8, 1, 5, 6, 12, 13, 9, 10, 2, 3, 4, 11};
__device__ constexpr int kGroupAt[kGroups + 1] = {0, 4, 8, 14};

struct Item {
  int plane, mt, nt, c0, c1, split, base;  // base: set of chunk 0 within the tile's sets
};

// Tiles of the upper triangle (kVxc).
__host__ __device__ inline int upper_of(int m_tiles, int n_tiles) {
  int u = 0;
  for (int mt = 0; mt < m_tiles; ++mt) u += n_tiles - 2 * mt > 0 ? n_tiles - 2 * mt : 0;
  return u;
}

__host__ __device__ inline int splits_of(int chunks, int per) { return (chunks + per - 1) / per; }

__host__ __device__ inline int64_t n_items(const GemmArgs &A, int upper) {
  const int64_t tiles = (int64_t)A.m_tiles * A.n_tiles;
  if (A.mode == kDensity) return tiles * A.planes;
  const int64_t all = tiles * splits_of(A.chunks, A.chunks_per_split);
  if (A.mode == kVxc && A.planes == 2) return all + (int64_t)upper * splits_of(3 * A.chunks, A.chunks_per_split);
  return all;
}

__device__ __forceinline__ Item item_of(const GemmArgs &A, int upper, int i) {
  Item t;
  if (A.mode == kDensity) {
    // All products of a row tile one after another (its digits stay in L2), the
    // full-length ones first and the triangular ones from long to short.
    const int per = A.planes * A.n_tiles;
    t.mt = i / per;
    int r = i % per;
    t.c0 = t.split = t.base = 0;
    if (r < A.n_tiles) {
      t.plane = 0;
      t.nt = r;
      t.c1 = A.chunks;
    } else {
      r -= A.n_tiles;
      t.plane = 1 + r % (A.planes - 1);
      t.nt = A.n_tiles - 1 - r / (A.planes - 1);
      t.c1 = t.nt + 1;
    }
    return t;
  }
  // Split-major: the tiles of one K range run together and share its digits in L2.
  const int kin = A.mode == kVxc && A.planes == 2 ? upper * splits_of(3 * A.chunks, A.chunks_per_split) : 0;
  int chunks = A.chunks;
  if (i < kin) {
    t.plane = 1;
    t.base = A.chunks;
    t.split = i / upper;
    int r = i % upper;
    t.mt = 0;
    while (r >= A.n_tiles - 2 * t.mt) {
      r -= A.n_tiles - 2 * t.mt;
      ++t.mt;
    }
    t.nt = 2 * t.mt + r;
    chunks = 3 * A.chunks;
  } else {
    i -= kin;
    t.plane = t.base = 0;
    const int tiles = A.m_tiles * A.n_tiles;
    t.split = i / tiles;
    t.nt = i % tiles / A.m_tiles;
    t.mt = i % tiles % A.m_tiles;
  }
  t.c0 = t.split * A.chunks_per_split;
  t.c1 = t.c0 + A.chunks_per_split < chunks ? t.c0 + A.chunks_per_split : chunks;
  return t;
}

// Rows of a tile (of `most`) that hold values when `left` are left, to a multiple of 8.
__device__ __forceinline__ uint32_t valid8(int64_t left, int most) {
  return left >= most ? (uint32_t)most : (uint32_t)(left + 7) / 8 * 8;
}

__device__ __forceinline__ void flag(int *err, int code) { atomicCAS(err, 0, code); }

// D (+)= A B^T on BF16 operands, K 16, issued by one thread.  a, b: the low
// words of the operands' descriptors; the high word is the same for all.
constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14);  // SBO 1024, version 1
__device__ __forceinline__ void mma_bf16(uint32_t d, uint32_t a, uint32_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      ".reg .b64 da, db;\n"
      "mov.b64 da, {%1, %5};\n"
      "mov.b64 db, {%2, %5};\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n"
      "}\n" ::"r"(d),
      "r"(a), "r"(b), "r"(idesc), "r"(accumulate), "r"(kDescHi)
      : "memory");
}
// FP32 accumulator (bits 4-5 = 1), BF16 A and B (bits 7-9, 10-12 = 1), both K-major.
constexpr uint32_t idesc_of(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((128u >> 4) << 24);
}

// sum += v << sh, rsh = 32 - sh, 0 <= sh < 32.
__device__ __forceinline__ void add_shifted(long long &sum, int v, int sh, int rsh) {
  asm("{\n"
      ".reg .b32 lo, hi, a, b;\n"
      "mov.b64 {lo, hi}, %0;\n"
      "shl.b32 a, %1, %2;\n"
      "shr.s32 b, %1, %3;\n"  // a shift by 32 leaves the sign
      "add.cc.u32 lo, lo, a;\n"
      "addc.u32 hi, hi, b;\n"
      "mov.b64 %0, {lo, hi};\n"
      "}\n"
      : "+l"(sum)
      : "r"(v), "r"(sh), "r"(rsh));
}

// v 2^e: the conversion, then the exponent field.  Below 2^-1022 the result is 0, as
// fixed_to_double's (kMaxField keeps products from the other end).
__device__ __forceinline__ double scaled(long long v, int e) {
  const double d = (double)v;
  const int hi = __double2hiint(d);
  return exp_field((uint32_t)hi) + e < 1 || v == 0 ? 0.0 : __hiloint2double(hi + e * (1 << 20), __double2loint(d));
}

__global__ void __launch_bounds__(kThreads, 1) fx_gemm_kernel(const GemmArgs A, const int upper) {
  previous_done();
  if (A.bad != nullptr && *A.bad != 0) return;
  extern __shared__ unsigned char smem_raw[];
  unsigned char *smem = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t full[kGroups], empty[kGroups], yfull[2], yempty, zfull, zempty, drain;
  __shared__ uint32_t tmem_base;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int items = (int)n_items(A, upper);

  if (threadIdx.x == 0) {
    for (int s = 0; s < kGroups; ++s) {
      umma::mbar_init(&full[s], s == 0 || s == 2 ? 1 + kDrains : 1);  // the copies, and accumulators drained
      umma::mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) umma::mbar_init(&yfull[b], 1);
    umma::mbar_init(&yempty, kDrains);
    umma::mbar_init(&zfull, 1);
    umma::mbar_init(&zempty, kDrains);
    umma::mbar_init(&drain, 1);
    umma::fence_barrier_init();
  }
  if (warp == 1) umma::tmem_alloc(&tmem_base, kTmemCols);
  umma::tc_fence_before();
  __syncthreads();
  umma::tc_fence_after();
  const uint32_t tbase = tmem_base;

  if (warp < 4) {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
  if (warp == 0) {
    // ------------------------------------------------------------ producer
    if (lane == 0) {
      uint32_t chunk = 0;
      int o = 0;
      bool ok = true;
      for (int i = blockIdx.x; i < items && ok; i += gridDim.x) {
        const Item t = item_of(A, upper, i);
        const int at = A.mode == kDensity ? t.plane * A.m_tiles + t.mt : t.mt;
        const unsigned char *a = A.a + ((size_t)at * A.a_stride + t.base + t.c0) * kSetBytes;
        const unsigned char *b = (t.plane ? A.b1 : A.b) + ((size_t)t.nt * A.b_stride + t.base + t.c0) * kSetBytes;
        // A block's first rows are its first bytes (128 each): rows without values are not copied.
        const uint32_t a_bytes = valid8(A.m_valid - (int64_t)t.mt * kTile, kTile) * 128u;
        const uint32_t b_valid = A.mode == kFull ? valid8(A.n_valid - (int64_t)t.nt * kTile, kTile)
                                                 : valid8(A.n_valid - (int64_t)t.nt * 64, 64);
        // Both halves of B in one copy where the first is full.
        const uint32_t b_bytes = (A.mode == kFull ? b_valid : 2 * b_valid) * 128u;
        const uint32_t b_first = A.mode != kFull && b_valid < 64 ? b_valid * 128u : b_bytes;
        for (int c = t.c0; c < t.c1 && ok; ++c, a += kSetBytes, b += kSetBytes) {
          // Straight-line code: the issue of a chunk's copies is on the critical path.
#pragma unroll
          for (int g = 0; g < kGroups; ++g) {
            o = g;
            if (!umma::mbar_wait(&empty[g], (chunk & 1) ^ 1)) {
              flag(A.err, 71);
              ok = false;
              break;
            }
            uint32_t bytes = 0;
#pragma unroll
            for (int k = kGroupAt[g]; k < kGroupAt[g + 1]; ++k) bytes += kGroupOf[k] < kDigits ? a_bytes : b_bytes;
            umma::mbar_arrive_expect_tx(&full[g], bytes);
#pragma unroll
            for (int k = kGroupAt[g]; k < kGroupAt[g + 1]; ++k) {
              const int s = kGroupOf[k];
              if (s < kDigits) {
                umma::bulk_g2s(smem + s * kBlockBytes, a + s * kBlockBytes, a_bytes, &full[g]);
              } else {
                umma::bulk_g2s(smem + s * kBlockBytes, b + (s - kDigits) * kBlockBytes, b_first, &full[g]);
                if (b_first != b_bytes)  // the valid rows of the second half
                  umma::bulk_g2s(smem + s * kBlockBytes + kBlockBytes / 2,
                                 b + (s - kDigits) * kBlockBytes + kBlockBytes / 2, b_first, &full[g]);
              }
            }
          }
          if (ok) o = kGroups;
          if (ok) ++chunk;
        }
      }
      // The last copies into every slot land before the CTA can retire.
      for (int k = 0; k < kGroups; ++k) {
        const uint32_t fills = chunk + (!ok && k < o ? 1 : 0);
        if (fills > 0 && !umma::mbar_wait(&full[k], (fills - 1) & 1)) flag(A.err, 72);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ---------------------------------------------------------- MMA issuer
    if (lane == 0) {
      // Low descriptor word of A's digit 0: address / 16, LBO 128.
      const uint32_t d0 = ((umma::smem_u32(smem) & 0x3FFFFu) >> 4) | ((128u >> 4) << 16);
      uint32_t chunk = 0, group = 0;
      bool ok = true;
      auto check = [&](bool done, int code) {
        if (!done) {
          flag(A.err, code);
          ok = false;
        }
        umma::tc_fence_after();
      };
      auto ready = [&](int g) { check(umma::mbar_wait(&full[g], chunk & 1), 73); };
      auto done = [&](int g) { umma::mma_commit(&empty[g]); };
      // Digit i of A times digit j of B (n 128) or digits j and j + 1 (n 256) into TMEM columns d.
      auto mul = [&](uint32_t d, int n, int i, int j, bool first) {
        const uint32_t a = d0 + i * (kBlockBytes >> 4), b = d0 + (kDigits + j) * (kBlockBytes >> 4);
#pragma unroll
        for (int kk = 0; kk < kChunkK / 16; ++kk)
          mma_bf16(d, a + 16 * kk, b + 16 * kk, idesc_of(n), (first && kk == 0) ? 0u : 1u);
      };
      const uint32_t l = tbase, h = tbase + 128, z5 = tbase + kZcol, z6 = z5 + 128;
      for (int i = blockIdx.x; i < items && ok; i += gridDim.x) {
        const Item t = item_of(A, upper, i);
        for (int c = t.c0; c < t.c1 && ok; ++c, ++chunk) {
          const bool zfirst = (c - t.c0) % kSumChunks == 0;
          const bool zlast = (c - t.c0) % kSumChunks == kSumChunks - 1 || c + 1 == t.c1;
          // L is filled three times a chunk (orders 0, 2, 4), H twice (1, 3).  The drains take them in order, so the
          // last one needed stands for both; the release of order 4 counts towards the next chunk's group 0, that of
          // order 1 towards group 2: one wait for both.
          ready(0);
          if (!ok) break;
          mul(l, 256, 0, 0, true);
          umma::mma_commit(&yfull[0]);
          mul(h, 128, 1, 0, false);
          umma::mma_commit(&yfull[1]);
          ready(1);
          if (zfirst) check(umma::mbar_wait(&zempty, (group & 1) ^ 1), 75);
          if (!ok) break;
          mul(z5, 256, 5, 0, zfirst);
          mul(z6, 128, 6, 0, false);
          mul(z5, 256, 0, 5, false);
          ready(2);
          if (!ok) break;
          mul(l, 256, 0, 2, true);
          mul(l, 256, 1, 1, false);
          mul(l, 256, 2, 0, false);
          umma::mma_commit(&yfull[0]);
          mul(h, 128, 3, 0, false);
          umma::mma_commit(&yfull[1]);
          mul(z5, 256, 4, 1, false);
          mul(z5, 256, 1, 4, false);
          done(1);
          check(umma::mbar_wait(&yempty, chunk & 1), 74);  // order 2 is drained
          if (!ok) break;
          mul(l, 128, 0, 4, true);
          mul(l, 128, 4, 0, false);
          mul(l, 128, 3, 1, false);
          mul(l, 128, 1, 3, false);
          done(0);
          mul(l, 128, 2, 2, false);
          umma::mma_commit(&yfull[0]);
          mul(z5, 256, 2, 3, false);
          mul(z5, 256, 3, 2, false);
          done(2);
          if (zlast) {
            umma::mma_commit(&zfull);
            ++group;
          }
        }
      }
      umma::mma_commit(&drain);
      if (!umma::mbar_wait(&drain, 0)) flag(A.err, 76);
    }
    __syncwarp();
  }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
    // -------------------------------------------------------------- drains
    const int q = warp & 3, col = ((warp - 4) >> 2) * kCols;
    const uint32_t tl = tbase + ((uint32_t)(q * 32) << 16) + col;
    uint32_t group = 0, chunk = 0;
    // After a wait has expired the rest of the launch runs through without waiting
    // (its results are invalid): leaving the loops early instead costs registers.
    bool ok = true;
    auto wait = [&](uint64_t *bar, uint32_t parity, int code) {
      if (ok && !umma::warp_wait(bar, parity)) {
        if (lane == 0) flag(A.err, code);
        ok = false;
      }
      umma::tc_fence_after();
    };
    // Columns of accumulator b to `take`; once the last are in registers, `freed` (if any) hears of it.
    auto drain = [&](int b, int cols, uint64_t *freed, auto &&take) {
      auto release = [&]() {
        umma::tc_fence_before();
        __syncwarp();
        if (lane == 0 && freed != nullptr) umma::mbar_arrive(freed);
      };
      if (cols == 0) {
        release();
        return;
      }
#pragma unroll
      for (int h = 0; h < kCols; h += 16) {
        uint32_t y[16];
        umma::tmem_ld16_nowait(tl + b * 128 + h, y);
        umma::tmem_ld_wait(y);
        if (h + 16 == kCols) release();
#pragma unroll
        for (int k = 0; k < 16; ++k) take(h + k, y[k]);
      }
      __syncwarp();
    };
    if (lane == 0) umma::mbar_arrive(&full[0]);  // L and H are free
    long long sum[kCols];  // orders 0..4 of this thread's row, unit 2^-36 (below 2^59 a chunk)
    for (int i = blockIdx.x; i < items; i += gridDim.x) {
      const Item t = item_of(A, upper, i);
#pragma unroll
      for (int k = 0; k < kCols; ++k) sum[k] = 0;
      int n = 0;  // chunks in the sums
      const int *eb = (t.plane ? A.eb1 : A.eb) + (size_t)t.nt * kTile + col;
      const int eb0 = __ldg(eb + lane), eb1 = __ldg(eb + 32 + lane);  // the columns' exponents, two a lane
      const int64_t row = (int64_t)t.mt * kTile + q * 32 + lane;
      // Columns of these 64 that are wanted; none where no row of the warp is.
      const int64_t left = A.mode == kFull ? A.n_valid - ((int64_t)t.nt * kTile + col) : A.n_valid - (int64_t)t.nt * 64;
      const int cols = row - lane >= A.m_valid || left <= 0 ? 0 : left < kCols ? (int)left : kCols;
      for (int c = t.c0; c < t.c1; ++c, ++chunk) {
        // Orders 0 and 1 are at most 2^20 and 2^22 units: the integer sits in the mantissa of v + 1.5 2^23 units
        // (the offsets are taken out below).  The others go through conversions, in one copy of the code: the
        // kernel's loops have to fit the instruction cache.
#pragma unroll
        for (int d = 0; d < 2; ++d) {
          wait(&yfull[d], (d ? 2 * chunk : 3 * chunk) & 1, 77);
          drain(d, cols, d ? &full[2] : nullptr, [&](int k, uint32_t y) {
            const int v = __float_as_int(__uint_as_float(y) + (d ? 24576.0f : 12582912.0f));
            sum[k] += (long long)v << (36 - 9 * d);
          });
        }
#pragma unroll 1
        for (int d = 2; d < 5; ++d) {
          const int b = d & 1, sh = 36 - 9 * d;
          const float f = __uint_as_float((uint32_t)(127 + 9 * d) << 23);
          wait(&yfull[b], (b ? 2 * chunk + 1 : 3 * chunk + d / 2) & 1, 77);
          drain(b, cols, d == 2 ? &yempty : d == 4 ? &full[0] : nullptr, [&](int k, uint32_t y) {
            add_shifted(sum[k], __float2int_rn(__uint_as_float(y) * f), sh, 32 - sh);
          });
        }
        ++n;
        if (c + 1 < t.c1 && n < kSumChunks) continue;
        // The sums of n chunks and Z into the output.
        wait(&zfull, group & 1, 78);
        ++group;
        // Bits below the unit 2^-36 that the result keeps: as far as 62 bits and Z's integer (|Z| < n 2^-20) allow.
        const int up_max = 14 - (n > 1 ? 32 - __clz(n - 1) : 0);
        // Offsets of orders 0 and 1: the words of 1.5 2^23 and of 1.5 2^14.
        const long long off = (long long)((unsigned long long)n * ((0x4B400000ull << 36) + (0x46C00000ull << 27)));
        const bool live = row < A.m_valid;
        const int *ea = A.ea + (size_t)t.plane * A.m_tiles * kTile;
        const int e0 = (live ? ea[row] : 0) - 2 * 1022 - 14 - 36;
        const int64_t at = (int64_t)t.split * A.split_stride + (int64_t)t.plane * A.plane_stride +
                           (col >> 6) * A.half_stride + (int64_t)t.nt * A.nt_stride + (col & 63) * A.ldc + row;
        double *out = A.out + at;
        const double *add = c - t.c0 >= kSumChunks ? out : A.add != nullptr ? A.add + at : nullptr;
        // 16 columns a turn, the sums moved down by 16 after each: unrolled, the code (some 60 KB, run once an
        // item) is fetched at the pace of instruction-cache misses.
#pragma unroll 1
        for (int h = 0; h < cols; h += 16) {
          uint32_t z5[16], z6[16];
          double v[16];
          __syncwarp();  // per-lane code above, warp-collective loads below
          umma::tmem_ld16_nowait(tl + kZcol + h, z5);
          umma::tmem_ld16_nowait(tl + kZcol + 128 + h, z6);
          umma::tmem_ld_wait(z5, z6);
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            const float z = __uint_as_float(z5[k]) + __uint_as_float(z6[k]);
            const long long x = sum[k] - off;
            const int top = (int)(x >> 32);  // up is below 15: the upper word says enough
            const int up = max(0, min(up_max, __clz(top ^ (top >> 31)) - 3));
            const float zs = __uint_as_float((uint32_t)(127 + 36 + up) << 23);
            const int e = e0 - up + __shfl_sync(0xffffffffu, h < 32 ? eb0 : eb1, (h & 31) + k);
            const long long y = (x << up) + (long long)__float2int_rn(z * zs);
            v[k] = k & 1 ? scaled(y, e) : fixed_to_double(y, e);  // the FP64 pipe takes half of the conversions
            if (!ok) v[k] = __longlong_as_double(0x7FF8000000000000ll);
          }
          if (h + 16 >= cols) {  // Z is read
            umma::tc_fence_before();
            __syncwarp();
            if (lane == 0) umma::mbar_arrive(&zempty);
          }
          // Stores apart from the arithmetic: a branch a column would serialise it.
          if (live) {
            double *o = out + (int64_t)h * A.ldc;
            if (add != nullptr) {
              const double *w = add + (int64_t)h * A.ldc;
              double was[16];
#pragma unroll
              for (int k = 0; k < 16; ++k) was[k] = h + k < cols ? w[(int64_t)k * A.ldc] : 0.0;
#pragma unroll
              for (int k = 0; k < 16; ++k) v[k] += was[k];
            }
#pragma unroll
            for (int k = 0; k < 16; ++k)
              if (h + k < cols) o[(int64_t)k * A.ldc] = v[k];
          }
#pragma unroll
          for (int k = 0; k < kCols; ++k) sum[k] = k + 16 < kCols ? sum[k + 16 < kCols ? k + 16 : 0] : 0;
        }
        if (cols <= kCols - 16) {  // turns left out: the sums they would have moved out
#pragma unroll
          for (int k = 0; k < kCols; ++k) sum[k] = 0;
        }
        n = 0;
        if (cols == 0) {
          umma::tc_fence_before();
          __syncwarp();
          if (lane == 0) umma::mbar_arrive(&zempty);
        }
      }
    }
  }
  umma::tc_fence_before();
  __syncthreads();
  if (warp == 1) umma::tmem_dealloc(tbase, kTmemCols);
}

// Four rows per warp: lane = (row, eight consecutive k), 64 of k (a chunk) a
// turn; the row's largest exponent first, then the digits.  The second read has
// to find the rows in L2: 40 warps an SM with four rows of 400 are 78 MB, with
// eight (as it was) 156 MB, which came from HBM twice.  Eight k in two 32-byte
// loads, so that no sector is asked for twice (L1 was busy for 75 % of the time).
// 9,376 x 400, four planes: 96 -> 77 us.
enum Load { kScalar, k16, k32 };  // bytes of a load
template <Load LOAD, bool OCT>
__global__ void __launch_bounds__(256) fx_rows_kernel(const double *__restrict__ src, int64_t plane_elems, int64_t rows,
                                                      int64_t ld, int k_valid, int chunks,
                                                      const int *__restrict__ oct, unsigned char *__restrict__ out,
                                                      int *__restrict__ exps, int *__restrict__ bad) {
  previous_done();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t tiles = (rows + kTile - 1) / kTile;
  const int64_t r0 = ((int64_t)blockIdx.x * 8 + warp) * kRowsPerWarp;
  if (r0 >= rows) return;
  const int plane = blockIdx.y;
  const int64_t row = r0 + lane % kRowsPerWarp;
  const bool in = row < rows;
  const double *x = src + (size_t)plane * plane_elems + (size_t)(in ? row : r0) * ld;
  const int kg = (lane / kRowsPerWarp) * 8;
  auto load8 = [&](int k, double (&v)[8]) {
    if (LOAD != kScalar && k + 8 <= k_valid) {
#pragma unroll
      for (int j = 0; j < 8; j += 4) {
        if (LOAD == k32) {
          asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
                       : "=d"(v[j]), "=d"(v[j + 1]), "=d"(v[j + 2]), "=d"(v[j + 3])
                       : "l"(x + k + j));
        } else {
          const double2 t = *(const double2 *)(x + k + j), u = *(const double2 *)(x + k + j + 2);
          v[j] = t.x;
          v[j + 1] = t.y;
          v[j + 2] = u.x;
          v[j + 3] = u.y;
        }
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = k + j < k_valid ? x[k + j] : 0.0;
    }
  };
  auto load_octaves = [&](int k, int (&t)[8]) {
    const int4 a = *(const int4 *)(oct + k), b = *(const int4 *)(oct + k + 4);
    t[0] = a.x, t[1] = a.y, t[2] = a.z, t[3] = a.w, t[4] = b.x, t[5] = b.y, t[6] = b.z, t[7] = b.w;
  };
  uint32_t m = 0;
  int mt = -(1 << 30);  // with the octaves; a zero counts as 2^(t - 1023)
  for (int k = kg; k < k_valid; k += kChunkK) {
    double v[8];
    int t[8];
    load8(k, v);
    if (OCT) load_octaves(k, t);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const uint32_t h = (uint32_t)__double2hiint(v[j]) & 0x7FFFFFFFu;
      m = max(m, h);
      if (OCT) mt = max(mt, (int)h + t[j] * (1 << 20));
    }
  }
#pragma unroll
  for (int o = kRowsPerWarp; o < 32; o *= 2) {
    m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (OCT) mt = max(mt, __shfl_xor_sync(0xffffffffu, mt, o));
  }
  int emax = exp_field(m);
  if (OCT) {
    if (max(emax, mt >> 20) > kMaxField) atomicOr(bad, 1);
    emax = mt >> 20;
  } else {
    if (emax > kMaxField) atomicOr(bad, 1);
    if (emax < 1) emax = 1;
  }
  if (lane < kRowsPerWarp && in) exps[(size_t)plane * rows + row] = emax;
  unsigned char *set = out + ((size_t)plane * tiles + (size_t)(row / kTile)) * chunks * kSetBytes +
                       elem_off((int)(row % kTile), kg);
  for (int k = kg; k < chunks * kChunkK; k += kChunkK, set += kSetBytes) {
    double v[8];
    int t[8];
    load8(k, v);
    if (OCT) load_octaves(k, t);
    long long f[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = to_fixed(v[j], OCT ? emax - t[j] : emax);
    uint4 d[kDigits];
    digits8(f, d);
#pragma unroll
    for (int i = 0; i < kDigits; ++i) *(uint4 *)(set + (size_t)i * kBlockBytes) = d[i];
  }
}

}  // namespace

cudaError_t launch_gemm(const GemmArgs &a, cudaStream_t st) {
  if (a.mode != kDensity && a.chunks_per_split < 1) return cudaErrorInvalidValue;
  cudaError_t e = cudaFuncSetAttribute(fx_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
  if (e != cudaSuccess) return e;
  int dev = 0, sms = 0;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  const int upper = a.mode == kVxc ? upper_of(a.m_tiles, a.n_tiles) : 0;
  const int64_t items = n_items(a, upper);
  if (items < 1) return cudaSuccess;
  if (items > 0x3FFFFFFF) return cudaErrorInvalidValue;
  const unsigned grid = (unsigned)(items < sms ? items : sms);
  // Chained (common.cuh) where few CTAs share an operand tile.  CTAs placed as SMs fall free do not start side by side,
  // and with more tiles in both directions those on one tile then miss each other in L2 (BLYP 400 x 150,001, 4 x 7 and
  // 74 x 7 tiles, 24.8 ms, chained 25.6; features of 187 AOs x 100,003 2.59 and 2.73; B88 115 x 65,536, two tiles, 1,191 us and
  // 1,177).
  if (a.m_tiles <= 2 || a.n_tiles <= 2)
    launch_next(fx_gemm_kernel, grid, kThreads, kSmemBytes, st, a, upper);
  else
    fx_gemm_kernel<<<grid, kThreads, kSmemBytes, st>>>(a, upper);
  return cudaGetLastError();
}

cudaError_t launch_rows(const double *src, int64_t plane_elems, int planes, int64_t rows, int64_t ld, int k_valid,
                        int chunks, const int *oct, unsigned char *out, int *exps, int *bad, cudaStream_t st) {
  const dim3 grid((unsigned)((rows + 8 * kRowsPerWarp - 1) / (8 * kRowsPerWarp)), planes);
  // The widest load that every row and plane starts on a boundary of.
  const uintptr_t at = (uintptr_t)src | (uintptr_t)(ld * sizeof(double)) | (uintptr_t)(plane_elems * sizeof(double));
  auto kernel = at % 32 == 0   ? oct != nullptr ? fx_rows_kernel<k32, true> : fx_rows_kernel<k32, false>
                : at % 16 == 0 ? oct != nullptr ? fx_rows_kernel<k16, true> : fx_rows_kernel<k16, false>
                               : oct != nullptr ? fx_rows_kernel<kScalar, true> : fx_rows_kernel<kScalar, false>;
  launch_next(kernel, grid, 256, 0, st, src, plane_elems, rows, ld, k_valid, chunks, oct, out, exps, bad);
  return cudaGetLastError();
}

}  // namespace fx
}  // namespace gdft
