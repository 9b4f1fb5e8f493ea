// FP64 trailing update A22 -= U^T W on the integer tensor cores
// (UpdateTrailingBlocks, src/block_ldlt_decomposition.cc:706-744 in
// wentianshu/BlockedBunchKaufmanLDLT).
//
// The FP64 tensor cores give 28 of a nominal 37 TFLOP/s on this update; the
// INT8 ones have more than a hundred times that rate.  Every operand row is
// scaled by a power of two and written as a 55-bit integer in seven signed
// 8-bit digits (the splitting of Ozaki, Ogita, Oishi and Rump, "Error-free
// transformations of matrix multiplication", Numer. Algorithms 59, 2012).
// Digit products of level l = t + u (weights 256^-l) sum exactly in a 32-bit
// accumulator (7 x 257 x 2^14 < 2^25); the 34 products with l <= 7 are kept.
// The eight levels' sums join in two groups of four, each an integer that a
// double holds exactly and that is subtracted from C in one rounding.
// Without level 7 the update's error was three times that of FP64 sums on
// factors of uniform random matrices (n = 2000, block 256: rms 5.7e-15
// against 1.8e-15), with it half (9.5e-16), so fewer products would not do.
// Factorization residuals: 9.2e-14 (FP64 tensor cores 1.14e-13) at n = 16000,
// 7.4e-15 (8.9e-15) on a spectral matrix of order 4000.
//
// A row's digits are fixed-point: an entry far below the row's largest keeps
// fewer bits than a double would, and a product of such entries is inaccurate
// by itself, whatever it adds up to by norm.  With u and w the scaled
// magnitudes, of K entries each, sum(u w) of an entry of C is off by at most
// 2^-56 (sum(u) + sum(w)) for the operands' rounding and 5.1 K 2^-64 for the
// products left out.  So a pass over the leading 7 bits of the magnitudes
// (bound_kernel, one product for 34) bounds sum(u w) from below, and a tile
// of C holding an entry whose error could exceed 16 x 2^-53 sum(u w)
// is left to the FP64 tensor cores, whose own bound is K 2^-53 sum(u w) (a
// panel with more than half of its tiles left so goes there whole).  Against
// |L| |D| |L^T|, in units of 2^-53, n = 2304, block 256, two index sets at scales s
// and 1 coupled by entries of size 1: digits alone 2.6, 45 and 4485 at s = 10^3,
// 10^4 and 10^6; with the bound 1.3, 2.4 and 2.5, as the FP64 tensor cores alone.
// The random, KKT and spectral matrices timed here need 5 to 15 of the 16, a
// few tiles of a KKT matrix's first panel more.
//
// Scaling, all by powers of two: factor row k of W is divided by w_k, its
// largest trailing entry, and column k of U multiplied by it, so a panel
// whose pivots differ in scale keeps every product's leading bits; then each
// row of U w and each column of W / w by its own largest entry.  A panel
// with an entry that is not finite or a scale beyond 2^+-400 is left to the
// FP64 tensor-core kernel, which is launched behind this one and returns
// unless the flag is set.
//
// Measured (B200): update at n = 40000, block 256: 758 -> 317 ms per
// factorization (13 of them the bound); n = 16000, block 256: 48.9 -> 22.4 ms;
// n = 10000, block 128: 13.9 -> 10.9 ms.
#include <algorithm>
#include <cfloat>
#include <climits>
#include <mutex>

#include "bbk_internal.cuh"
#include "umma.cuh"

namespace bbk {
namespace {

constexpr int kDigits = 7;
constexpr int kTile = 128;       // C tile rows and columns, rows of a digit block
constexpr int kChunk = 32;       // k (bytes) of a digit block and of one MMA
constexpr int kBlock = kTile * kChunk;  // 4 KB: one digit of 128 rows x 32 k
constexpr int kLowDigits = 4;    // digits the pass over the levels 0..3 reads
constexpr int kStageBytes = 2 * kDigits * kBlock;
constexpr int kStages = 3;
constexpr int kEpiWarps = 16;
constexpr int kCols = 4 * kTile / kEpiWarps;  // columns of an epilogue warp
constexpr int kThreads = (kEpiWarps + 2) * 32;
constexpr int kMaxTiles = 4096;  // of one CTA
constexpr int kAll = 1, kSome = 2;  // what a panel's flag leaves to the FP64 kernel
constexpr size_t kSmem = static_cast<size_t>(kStages) * kStageBytes + kEpiWarps * kCols * sizeof(double) + 256 +
                         kMaxTiles;
static_assert(kSmem <= 227 * 1024, "stages fit the shared memory of one CTA");

constexpr int kMaxExp = 400;  // larger scales go to the FP64 kernel
constexpr int kMaxK = 1024;   // keeps 5 x k x 2^14 x 2^24 below 2^51: the joined sums are exact doubles

struct SliceArgs {
  const DeviceState* st;
  int panel;
  int n;
  const double* u;  // U[x, q] = u[x * ldu + q]
  int ldu;
  const double* w;  // W[q, x] = w[q * ldw + x]
  long long ldw;
  double* c;
  long long ldc;
  int nkc;          // digit blocks per row block (the buffers' pitch)
  unsigned char* da;  // digits of U: block (row block, k chunk, digit)
  unsigned char* db;  // digits of W
  double* sa;       // 2^(scale exponent) per row of U, from the 128-aligned origin
  double* sb;       // the same per column of W, times 2^-70
  unsigned long long* wmax;  // 2 x (nkc * kChunk): bits of w_k, by panel parity
  int* flag;        // by panel parity: kAll the panel, kSome its marked tiles are left to the FP64 kernel
  unsigned char* ma;  // leading 7 bits of U's scaled magnitudes: block (row block, k chunk)
  unsigned char* mb;  // W's
  int* ta;          // per row of U and column of W: its part of the least 2^14 sum(u w)
  int* tb;          // that the digits are accurate enough for (kNone: an empty row)
  unsigned char* marks;  // per tile (J (J + 1) / 2 + I): left to the FP64 kernel
  int* count;       // marked tiles, CTAs done (zero between launches)
  unsigned long long timeout_ns;
};

struct Range {
  int k0, e, inner, t0;  // panel [k0, e), its width, the tiles' origin
};

__device__ __forceinline__ bool panel_range_of(const SliceArgs& S, Range& r) {
  if (ld_relaxed_s32(&S.st->abort)) return false;
  r.k0 = ldcg(&S.st->kstart[S.panel & 1]);
  r.e = ldcg(&S.st->kstart[(S.panel + 1) & 1]);
  r.inner = r.e - r.k0;
  r.t0 = r.e / kTile * kTile;
  return r.inner > 0 && r.e < S.n;
}

// w_k: the largest magnitude of each W row over the trailing columns, as
// bits (they order like the magnitudes; NaN is above infinity).  Reads W
// once, coalesced.
__global__ void __launch_bounds__(256) row_max_kernel(SliceArgs S) {
  Range r;
  if (!panel_range_of(S, r)) return;
  const int k = blockIdx.y;
  if (k >= r.inner) return;
  const double* row = S.w + static_cast<long long>(k) * S.ldw;
  unsigned long long m = 0;
  const int step = gridDim.x * 256;
  for (int x = r.e + blockIdx.x * 256 + threadIdx.x; x < S.n; x += 4 * step) {
    double v[4];  // four loads in flight
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = x + u * step < S.n ? row[x + u * step] : 0.0;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const unsigned long long w =
          static_cast<unsigned long long>(__double_as_longlong(v[u])) & 0x7fffffffffffffffull;
      m = w > m ? w : m;
    }
  }
  for (int off = 16; off > 0; off >>= 1) {
    const unsigned long long o = __shfl_down_sync(0xffffffffu, m, off);
    m = o > m ? o : m;
  }
  __shared__ unsigned long long red[8];
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < 8; ++i) m = red[i] > m ? red[i] : m;
    if (m) atomicMax(S.wmax + static_cast<size_t>(S.panel & 1) * S.nkc * kChunk + k, m);
  }
}

// 2^x, x clamped to what a normal double holds (a clamped scale belongs to a
// panel that is left to the FP64 kernel, or to an entry that rounds to 0)
__device__ __forceinline__ double pow2(int x) {
  const int b = min(max(x + 1023, 0), 2046);
  return __longlong_as_double(static_cast<long long>(b) << 52);
}

// The exponent x of a row whose largest magnitude is m: |v| 2^-x <= 0.996,
// so that the leading digit of v 2^(55 - x) fits a signed byte.
__device__ __forceinline__ int row_exponent(double m) {
  int x = 0;
  const double f = frexp(m, &x);
  return m > 0.0 ? x + (f > 0.996) : 0;
}

constexpr int kNone = -(1 << 29);

// A row's part of that least sum: 2^14 times ((1 / 8) sum(u) + 5.1 K / 4096) /
// 16, from sum(u), its largest entry's scale taken out.
__device__ __forceinline__ int row_threshold(double sum, int k) {
  return __double2int_ru(1024.0 * (0.125 * sum + 5.1 / 4096.0 * k));
}

// Digits of both operands.  One CTA takes 32 rows (columns of W): lane l row
// l, warp w the k groups w, w + 8, ... of 16.  The rows are read twice (the
// scale, then the digits; the second time from L1 or L2) and each thread
// stores 16 bytes per digit, eight lanes to a 128-byte core matrix.
__global__ void __launch_bounds__(256) slice_kernel(SliceArgs S) {
  extern __shared__ int kexp[];  // exponent of w_k
  __shared__ double red[8][32], rsum[8][32];
  __shared__ int bad;
  Range r;
  if (!panel_range_of(S, r)) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int kcap = S.nkc * kChunk;
  const int nchunks = (r.inner + kChunk - 1) / kChunk;
  if (blockIdx.x == 0) {  // the next panel's maxima and flag start from zero
    for (int k = threadIdx.x; k < kcap; k += 256) S.wmax[static_cast<size_t>((S.panel + 1) & 1) * kcap + k] = 0ull;
    if (threadIdx.x == 0) S.flag[(S.panel + 1) & 1] = 0;
  }
  if (threadIdx.x == 0) bad = 0;
  __syncthreads();
  for (int k = threadIdx.x; k < nchunks * kChunk; k += 256) {
    int x = 0;
    if (k < r.inner) {
      const double m = __longlong_as_double(
          static_cast<long long>(S.wmax[static_cast<size_t>(S.panel & 1) * kcap + k]));
      if (m > 0.0 && m <= DBL_MAX) frexp(m, &x);
      if (!(m <= DBL_MAX) || x > kMaxExp || x < -kMaxExp) bad = 1;
    }
    kexp[k] = x;
  }
  __syncthreads();
  const int rows = (S.n - r.t0 + kTile - 1) / kTile * kTile;
  const int groups = rows / 32;
  const int ntiles = (rows / kTile) * (rows / kTile + 1) / 2;
  for (int i = blockIdx.x * 256 + threadIdx.x; i < ntiles; i += gridDim.x * 256) S.marks[i] = 0;
  for (int job = blockIdx.x; job < 2 * groups; job += gridDim.x) {
    const bool is_u = job < groups;
    const int rr = (is_u ? job : job - groups) * 32 + lane;  // row from the tiles' origin
    const int x = r.t0 + rr;
    const bool live = x >= r.e && x < S.n;
    auto load = [&](int g, double (&v)[16]) {
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const int k = g * 16 + i;
        v[i] = live && k < r.inner
                   ? (is_u ? S.u[static_cast<long long>(x) * S.ldu + k] : S.w[static_cast<long long>(k) * S.ldw + x])
                   : 0.0;
      }
    };
    double m = 0.0, sum = 0.0;
    bool fin = true;
    for (int g = warp; g < 2 * nchunks; g += 8) {
      double v[16];
      load(g, v);
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const int kx = kexp[g * 16 + i];
        const double s = fabs(v[i]) * pow2(is_u ? kx : -kx);
        fin = fin && s <= DBL_MAX;
        m = fmax(m, s);
        sum += s;
      }
    }
    red[warp][lane] = m;
    rsum[warp][lane] = sum;
    if (!fin) bad = 1;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 8; ++i) m = fmax(m, red[i][lane]);
    const int ex = row_exponent(m);
    if (ex > kMaxExp || ex < -kMaxExp) bad = 1;
    if (warp == 0) {
      (is_u ? S.sa : S.sb)[rr] = pow2(is_u ? ex : ex - 70);
      sum = 0.0;
#pragma unroll
      for (int i = 0; i < 8; ++i) sum += rsum[i][lane];
      (is_u ? S.ta : S.tb)[rr] = m > 0.0 ? row_threshold(sum * pow2(-ex), r.inner) : kNone;
    }
    unsigned char* dst = (is_u ? S.da : S.db) + static_cast<size_t>(rr / kTile) * S.nkc * (kDigits * kBlock) +
                         (rr % kTile / 8) * 256 + (rr % 8) * 16;
    unsigned char* mdst = (is_u ? S.ma : S.mb) + static_cast<size_t>(rr / kTile) * S.nkc * kBlock +
                          (rr % kTile / 8) * 256 + (rr % 8) * 16;
    for (int g = warp; g < 2 * nchunks; g += 8) {
      double v[16];
      load(g, v);
      uint32_t d[kDigits][4], mag[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        uint32_t lo[4], hi[4], top[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int kx = kexp[g * 16 + 4 * q + i];
          // y = x + 128 in every lower byte: the bytes of y, less 128 each,
          // are the signed digits of x
          const long long x = __double2ll_rn(v[4 * q + i] * pow2(55 - ex + (is_u ? kx : -kx)));
          const long long y = x + 0x0000808080808080ll;
          top[i] = static_cast<uint32_t>(static_cast<unsigned long long>(x < 0 ? -x : x) >> 32);
          lo[i] = static_cast<uint32_t>(y) ^ 0x80808080u;
          hi[i] = static_cast<uint32_t>(static_cast<unsigned long long>(y) >> 32) ^ 0x00008080u;
        }
        auto gather = [](const uint32_t (&v4)[4], int byte) {
          const uint32_t sel = static_cast<uint32_t>(byte | ((byte + 4) << 4));
          return __byte_perm(__byte_perm(v4[0], v4[1], sel), __byte_perm(v4[2], v4[3], sel), 0x5410);
        };
        mag[q] = gather(top, 2);
        d[0][q] = gather(hi, 2);
        d[1][q] = gather(hi, 1);
        d[2][q] = gather(hi, 0);
        d[3][q] = gather(lo, 3);
        d[4][q] = gather(lo, 2);
        d[5][q] = gather(lo, 1);
        d[6][q] = gather(lo, 0);
      }
      unsigned char* blk = dst + static_cast<size_t>(g / 2) * (kDigits * kBlock) + (g & 1) * 128;
#pragma unroll
      for (int t = 0; t < kDigits; ++t)
        *reinterpret_cast<uint4*>(blk + t * kBlock) = make_uint4(d[t][0], d[t][1], d[t][2], d[t][3]);
      *reinterpret_cast<uint4*>(mdst + static_cast<size_t>(g / 2) * kBlock + (g & 1) * 128) =
          make_uint4(mag[0], mag[1], mag[2], mag[3]);
    }
    __syncthreads();  // red is written again
  }
  __syncthreads();
  if (threadIdx.x == 0 && bad) atomicExch(S.flag + (S.panel & 1), kAll);
}

// Instruction descriptor of kind::i8: 32-bit integer accumulators, signed A
// and B, both K-major, M = 128, N = cols.
__host__ __device__ constexpr uint32_t umma_i8_desc(int cols) {
  return (2u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(cols >> 3) << 17) |
         (static_cast<uint32_t>(kTile >> 4) << 24);
}
constexpr uint32_t kIdesc = umma_i8_desc(kTile);

// One MMA.  Products that share their A digit keep it in the tensor core's
// operand buffer (kUse: 0 fills it, 1 reads it, 2 reads it for the last
// time, 3 does without): with A and B read from shared memory each time, an MMA of this size
// takes all of its bandwidth and leaves none for the copies.
template <int kUse>
__device__ __forceinline__ void umma_i8(uint32_t d, uint64_t da, uint64_t db, bool accumulate,
                                        uint32_t idesc = kIdesc) {
#define BBK_UMMA_I8(use)                                                                 \
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"                         \
               "tcgen05.mma.cta_group::1.kind::i8" use " [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d), \
               "l"(da), "l"(db), "r"(idesc), "r"(accumulate ? 1u : 0u))
  if (kUse == 0) BBK_UMMA_I8(".collector::a::fill");
  if (kUse == 1) BBK_UMMA_I8(".collector::a::use");
  if (kUse == 2) BBK_UMMA_I8(".collector::a::lastuse");
  if (kUse == 3) BBK_UMMA_I8("");
#undef BBK_UMMA_I8
}

// The products of one k chunk whose level t + u is in [kFirst, kFirst + 4):
// A digits at a + t blocks, B digits at b + u blocks (descriptors), level l
// into accumulator l - kFirst; the accumulators start from zero with kFresh.
template <int kFirst, int kDigitsUsed, bool kFresh>
__device__ __forceinline__ void chunk_products(uint32_t tmem, uint64_t a, uint64_t b) {
#pragma unroll
  for (int t = 0; t < kDigitsUsed; ++t) {
    constexpr int kLast = kFirst + 3;
    const int u0 = t < kFirst ? kFirst - t : 0;
    const int u1 = kLast - t < kDigitsUsed - 1 ? kLast - t : kDigitsUsed - 1;
#pragma unroll
    for (int u = u0; u <= u1; ++u) {
      const uint32_t d = tmem + static_cast<uint32_t>((t + u - kFirst) * kTile);
      const uint64_t da = a + t * (kBlock >> 4), db = b + u * (kBlock >> 4);
      const int first = t + u < kDigitsUsed ? 0 : t + u - (kDigitsUsed - 1);  // the level's first t
      const bool acc = !kFresh || t > first;
      if (u0 == u1)
        umma_i8<3>(d, da, db, acc);
      else if (u == u0)
        umma_i8<0>(d, da, db, acc);
      else if (u < u1)
        umma_i8<1>(d, da, db, acc);
      else
        umma_i8<2>(d, da, db, acc);
    }
  }
}

// Marks the tiles whose sums of magnitudes are too small for the digits (see
// the top of this file).  Persistent CTAs over steps of a row block times a
// strip of `cb` column blocks, each CTA a run of consecutive steps down the
// strips: the strip's columns stay in shared memory, so only the row blocks
// stream from L2 (with both operands streamed per tile the pass took 2.4 us per
// tile and CTA, a seventh of the update).  Warps 0-15 compare the sums (warp
// w: rows 32 (w % 4).., columns 32 (w / 4).. of each block), then one warp for
// the bulk copies and one that issues the MMAs.
constexpr int kGroup = 4;  // chunks of a stage of the ring of row blocks
constexpr int kRingBytes = kGroup * kBlock;
constexpr int kRingMax = 12;
constexpr int kAcc = 2;    // accumulators of 2 kTile columns
constexpr size_t kBoundData = 208 * 1024;  // the strips' columns, then the ring
constexpr size_t kBoundSmem = kBoundData + kEpiWarps * 2 * 32 * sizeof(int) + 512;
static_assert(kBoundSmem <= 227 * 1024 && (2 * kRingMax + 4 + 2 * kAcc) * 8 + 4 <= 512, "shared memory of one CTA");

struct BoundShape {
  int cb;    // column blocks of a strip
  int nbuf;  // strips in shared memory
  int ring;  // stages of row blocks
};
__host__ __device__ inline BoundShape bound_shape(int nkc) {
  BoundShape b{2, 2, 0};
  if (b.nbuf * b.cb * nkc * kBlock > 144 * 1024) b.nbuf = 1;
  if (b.nbuf * b.cb * nkc * kBlock > 144 * 1024) b.cb = 1;
  const int left = (static_cast<int>(kBoundData) - b.nbuf * b.cb * nkc * kBlock) / kRingBytes;
  b.ring = left < kRingMax ? left : kRingMax;
  return b;
}
static_assert(kBoundData >= kMaxK / kChunk * kBlock + 2 * kRingBytes, "the widest panel leaves a ring");

__global__ void __launch_bounds__(kThreads, 1) bound_kernel(SliceArgs S) {
  extern __shared__ __align__(1024) unsigned char sm[];
  int* cols = reinterpret_cast<int*>(sm + kBoundData);  // 2 x 32 columns' parts per epilogue warp
  uint64_t* full = reinterpret_cast<uint64_t*>(cols + kEpiWarps * 64);
  uint64_t* empty = full + kRingMax;
  uint64_t* bfull = empty + kRingMax;
  uint64_t* bempty = bfull + 2;
  uint64_t* accfull = bempty + 2;
  uint64_t* accempty = accfull + kAcc;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(accempty + kAcc);
  Range r;
  if (!panel_range_of(S, r)) return;
  int* flag = S.flag + (S.panel & 1);
  // (another CTA may raise it to kSome meanwhile; kAll was set before this kernel)
  if (ldcg(flag) == kAll) return;
  const BoundShape shape = bound_shape(S.nkc);
  const int cb = shape.cb;
  const int tm = (S.n - r.t0 + kTile - 1) / kTile;
  // strip j: row blocks 0 .. min(cb (j + 1), tm) - 1, after cb j (j + 1) / 2
  // steps of the strips before it
  const int strips = (tm + cb - 1) / cb;
  const int total = cb * strips * (strips - 1) / 2 + tm;
  const int first = static_cast<int>(static_cast<long long>(total) * blockIdx.x / gridDim.x);
  const int last = static_cast<int>(static_cast<long long>(total) * (blockIdx.x + 1) / gridDim.x);
  if (first >= last) return;
  int j0 = static_cast<int>((sqrtf(8.0f * first / cb + 1.0f) - 1.0f) * 0.5f);
  while (j0 > 0 && cb * j0 * (j0 + 1) / 2 > first) --j0;
  while (j0 + 1 < strips && cb * (j0 + 1) * (j0 + 2) / 2 <= first) ++j0;
  const int i0 = first - cb * j0 * (j0 + 1) / 2;
  const int nchunks = (r.inner + kChunk - 1) / kChunk;
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;

  if (warp == kEpiWarps + 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(kAcc * 2 * kTile)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    if (lane == 0) {
      for (int b = 0; b < 2 * kRingMax + 4; ++b)  // full, empty, bfull, bempty
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&full[b])) : "memory");
      for (int b = 0; b < kAcc; ++b) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&accfull[b])) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&accempty[b])), "r"(kEpiWarps)
                     : "memory");
      }
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  auto wait = [&](uint64_t* bar, int phase) {  // of a whole warp
    const bool got = mbar_wait(smem_u32(bar), static_cast<uint32_t>(phase & 1), S.st, S.timeout_ns);
    if (!__all_sync(0xffffffffu, got)) return false;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    return true;
  };
  auto finish = [&](uint64_t* bar, int phase, unsigned long long t0) {
    mbar_finish(smem_u32(bar), static_cast<uint32_t>(phase & 1), t0);
  };
  const size_t row_block = static_cast<size_t>(S.nkc) * kBlock;
  const int strip_bytes = cb * S.nkc * kBlock;
  const uint32_t ring0 = smem_u32(sm) + static_cast<uint32_t>(shape.nbuf * strip_bytes);
  // the steps of this CTA, in order: f(step, strip's count here, row block,
  // strip, first step of the strip, last step of it)
  auto steps = [&](auto&& f) {
    int i = i0, j = j0, strip = 0;
    bool fresh = true;
    for (int t = first; t < last; ++t) {
      const bool ends = i + 1 == min(cb * (j + 1), tm) || t + 1 == last;
      if (!f(t - first, strip, i, j, fresh, ends)) return false;
      fresh = ends;
      if (ends) {
        i = 0;
        ++j;
        ++strip;
      } else {
        ++i;
      }
    }
    return true;
  };
  bool ok = true;

  if (warp == kEpiWarps) {
    if (lane == 0) {
      int item = 0, loaded = 0;
      ok = steps([&](int, int strip, int i, int j, bool fresh, bool) {
        if (fresh) {
          const int b = strip % shape.nbuf, use = strip / shape.nbuf;
          if (use >= 1 && !mbar_wait(smem_u32(&bempty[b]), static_cast<uint32_t>((use - 1) & 1), S.st, S.timeout_ns))
            return false;
          const int blocks = min(cb, tm - cb * j);
          const uint32_t bar = smem_u32(&bfull[b]);
          const uint32_t base = smem_u32(sm) + static_cast<uint32_t>(b * strip_bytes);
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                       "r"(blocks * nchunks * kBlock)
                       : "memory");
          for (int ch = 0; ch < nchunks; ++ch)
            for (int h = 0; h < blocks; ++h)
              bulk_load(base + static_cast<uint32_t>((ch * cb + h) * kBlock),
                        S.mb + (cb * j + h) * row_block + static_cast<size_t>(ch) * kBlock, kBlock, bar);
          ++loaded;
        }
        for (int ch = 0; ch < nchunks; ch += kGroup, ++item) {
          const int st = item % shape.ring;
          if (item >= shape.ring && !mbar_wait(smem_u32(&empty[st]), static_cast<uint32_t>((item / shape.ring - 1) & 1),
                                               S.st, S.timeout_ns))
            return false;
          const uint32_t bar = smem_u32(&full[st]);
          const uint32_t bytes = static_cast<uint32_t>(min(kGroup, nchunks - ch) * kBlock);
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
          bulk_load(ring0 + static_cast<uint32_t>(st * kRingBytes), S.ma + i * row_block + static_cast<size_t>(ch) * kBlock,
                    bytes, bar);
        }
        return true;
      });
      // the copies in flight land before the CTA gives up its memory
      const unsigned long long t0 = globaltimer_ns();
      for (int k = max(0, item - shape.ring); k < item; ++k) finish(&full[k % shape.ring], k / shape.ring, t0);
      for (int k = max(0, loaded - shape.nbuf); k < loaded; ++k) finish(&bfull[k % shape.nbuf], k / shape.nbuf, t0);
    }
  } else if (warp == kEpiWarps + 1) {
    const bool one = elect_one();
    int item = 0;
    ok = steps([&](int step, int strip, int, int j, bool fresh, bool ends) {
      const int b = strip % shape.nbuf, acc = step % kAcc;
      if (fresh && !wait(&bfull[b], strip / shape.nbuf)) return false;
      if (step >= kAcc && !wait(&accempty[acc], step / kAcc - 1)) return false;
      const uint32_t idesc = umma_i8_desc(min(cb, tm - cb * j) * kTile);
      const uint64_t bd = umma_desc(smem_u32(sm) + static_cast<uint32_t>(b * strip_bytes), 256);
      for (int ch = 0; ch < nchunks; ch += kGroup, ++item) {
        const int st = item % shape.ring;
        if (!wait(&full[st], item / shape.ring)) return false;
        const uint64_t ad = umma_desc(ring0 + static_cast<uint32_t>(st * kRingBytes), 256);
        if (one) {
          for (int c = 0; c < min(kGroup, nchunks - ch); ++c)
            umma_i8<3>(tmem + static_cast<uint32_t>(acc * 2 * kTile), ad + c * (kBlock >> 4),
                       bd + (ch + c) * cb * (kBlock >> 4), ch + c > 0, idesc);
          umma_commit(smem_u32(&empty[st]));
        }
      }
      if (one) {
        umma_commit(smem_u32(&accfull[acc]));
        if (ends) umma_commit(smem_u32(&bempty[b]));
      }
      return true;
    });
    // the MMAs issued finish before the accumulators are released
    if (item > 0) finish(&empty[(item - 1) % shape.ring], (item - 1) / shape.ring, globaltimer_ns());
  } else {
    const int row = (warp & 3) * 32 + lane, col0 = (warp >> 2) * 32;  // this thread's row, its columns
    int* tb = cols + warp * 64;
    int ta = S.ta[i0 * kTile + row];
    ok = steps([&](int step, int, int i, int j, bool fresh, bool ends) {
      const int acc = step % kAcc, blocks = min(cb, tm - cb * j);
      if (fresh) {
        __syncwarp();  // every lane is done with the last strip's columns
        for (int h = 0; h < blocks; ++h) tb[h * 32 + lane] = S.tb[(cb * j + h) * kTile + col0 + lane];
        __syncwarp();
      }
      const int t = ta;
      if (step + 1 < last - first) ta = S.ta[(ends ? 0 : i + 1) * kTile + row];  // on its way during the wait
      if (!wait(&accfull[acc], step / kAcc)) return false;
      unsigned low = 0;  // bit h: an entry of block h
      for (int h = 0; h < blocks; ++h) {
        int p[32];
        tmem_ld32x32(tmem + static_cast<uint32_t>(acc * 2 * kTile + h * kTile + col0) +
                         (static_cast<uint32_t>((warp & 3) * 32) << 16), p);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        const int J = cb * j + h;
        if (i > J) continue;
        const int from = i == J ? row - col0 : 0;  // the upper triangle's columns of this row
        int least = INT_MAX;
#pragma unroll
        for (int c = 0; c < 32; ++c) {
          const int v = p[c] - tb[h * 32 + c];
          least = min(least, c >= from ? v : INT_MAX);
        }
        if (least < t) low |= 1u << h;
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&accempty[acc]));
      low = __reduce_or_sync(0xffffffffu, low);
      if (low && lane == 0) {
        for (int h = 0; h < blocks; ++h) {
          const int J = cb * j + h;
          const int tile = J * (J + 1) / 2 + i;
          const unsigned bit = 1u << 8 * (tile & 3);
          if ((low >> h & 1) && !(atomicOr(reinterpret_cast<unsigned*>(S.marks) + (tile >> 2), bit) & bit))
            atomicAdd(S.count, 1);
        }
        atomicCAS(flag, 0, kSome);
      }
      return true;
    });
  }
  if (!ok) {
    atomicCAS(const_cast<int*>(&S.st->status), 0, BBK_ERR_TIMEOUT);
    atomicExch(const_cast<int*>(&S.st->abort), 1);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (warp == kEpiWarps + 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kAcc * 2 * kTile)
                 : "memory");
  // the last CTA: beyond half of the tiles, the FP64 kernel takes all (a tile in
  // digits takes 0.4 of its time there)
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(S.count + 1, 1) == min(total, static_cast<int>(gridDim.x)) - 1) {
      if (2 * atomicExch(S.count, 0) > tm * (tm + 1) / 2) atomicExch(flag, kAll);
      atomicExch(S.count + 1, 0);
    }
  }
}

// An integer below 2^51 in magnitude as a double, exactly.
__device__ __forceinline__ double int_to_double(long long v) {
  return __longlong_as_double(v + 0x4338000000000000ll) - 6755399441055744.0;
}

// The tiles: persistent CTAs over the 128 x 128 tiles of the trailing upper
// triangle.  Tensor memory holds four 128-column accumulators and the eight
// levels need eight, so a tile takes two passes over k: the levels 4..7 (24
// products, all digits), then 0..3 (10 products of the four leading digits).
// The epilogue warps load their part of C during the first pass, subtract
// each pass's sums when it ends and store after the second.
// Warps 0-15: epilogue (warp w: rows 32 (w % 4).., columns 32 (w / 4)..),
// then one warp for the bulk copies and one that issues the MMAs.
// A tile with k = 256 takes about 27 000 cycles: the MMAs' 272 x 64 at the
// tensor core's rate, 3 000 to read and join the sums of each pass (while
// the tensor core waits: all of tensor memory is in use), and the fill of
// the first stages.  Eight epilogue warps joined in 4 000; C loaded between
// the passes, one row per thread, cost 10 000 more.
__global__ void __launch_bounds__(kThreads, 1) i8_update_kernel(SliceArgs S) {
  extern __shared__ __align__(1024) unsigned char sm[];
  double* scales = reinterpret_cast<double*>(sm + kStages * kStageBytes);  // kCols column scales per epilogue warp
  uint64_t* full = reinterpret_cast<uint64_t*>(scales + kEpiWarps * kCols);
  uint64_t* empty = full + kStages;
  uint64_t* accfull = empty + kStages;
  uint64_t* accempty = accfull + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(accempty + 1);
  unsigned char* skip = sm + kSmem - kMaxTiles;  // per tile of this CTA: left to the FP64 kernel
  Range r;
  if (!panel_range_of(S, r)) return;
  const int left = ldcg(S.flag + (S.panel & 1));  // what the FP64 kernel takes
  if (left == kAll) return;
  const int tm = (S.n - r.t0 + kTile - 1) / kTile;
  const int ntiles = tm * (tm + 1) / 2;
  if (static_cast<int>(blockIdx.x) >= ntiles) return;
  const int my_tiles = (ntiles - static_cast<int>(blockIdx.x) + static_cast<int>(gridDim.x) - 1) /
                       static_cast<int>(gridDim.x);
  const int nchunks = (r.inner + kChunk - 1) / kChunk;
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;

  if (warp == kEpiWarps + 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    if (lane == 0) {
      for (int st = 0; st < kStages; ++st) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&full[st])) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&empty[st])) : "memory");
      }
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(accfull)) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(accempty)), "r"(kEpiWarps) : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
  }
  for (int m = threadIdx.x; m < my_tiles; m += kThreads) {
    int I, J;
    strip_tile(static_cast<int>(blockIdx.x) + m * static_cast<int>(gridDim.x), tm, I, J);
    skip[m] = left == kSome ? __ldcg(S.marks + J * (J + 1) / 2 + I) : 0;
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  auto tile_of = [&](int m, int& I, int& J) {  // tile m of this CTA
    strip_tile(static_cast<int>(blockIdx.x) + m * static_cast<int>(gridDim.x), tm, I, J);
  };
  const size_t row_block = static_cast<size_t>(S.nkc) * (kDigits * kBlock);
  bool ok = true;

  if (warp == kEpiWarps) {
    if (lane == 0) {
      int item = 0;
      for (int m = 0; m < my_tiles && ok; ++m) {
        int I, J;
        tile_of(m, I, J);
        const unsigned char* a = S.da + I * row_block;
        const unsigned char* b = S.db + J * row_block;
        for (int q = 0; q < 2 * nchunks; ++q, ++item) {
          const int st = item % kStages;
          if (item >= kStages &&
              !mbar_wait(smem_u32(&empty[st]), static_cast<uint32_t>((item / kStages - 1) & 1), S.st, S.timeout_ns)) {
            ok = false;
            break;
          }
          const uint32_t bar = smem_u32(&full[st]);
          const uint32_t base = smem_u32(sm + st * kStageBytes);
          const bool low = q >= nchunks;
          const int ch = low ? q - nchunks : q;
          const uint32_t bytes = static_cast<uint32_t>((low ? kLowDigits : kDigits) * kBlock);
          const size_t off = static_cast<size_t>(ch) * (kDigits * kBlock);
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(2 * bytes) : "memory");
          bulk_load(base, a + off, bytes, bar);
          bulk_load(base + bytes, b + off, bytes, bar);
        }
      }
      // the copies in flight land before the CTA gives up its memory
      const unsigned long long t0 = globaltimer_ns();
      for (int k = max(0, item - kStages); k < item; ++k)
        mbar_finish(smem_u32(&full[k % kStages]), static_cast<uint32_t>((k / kStages) & 1), t0);
    }
  } else if (warp == kEpiWarps + 1) {
    // the whole warp walks the stages, so that descriptors stay in uniform
    // registers (one lane alone took 96 cycles per MMA to issue them, of 64
    // that the tensor core needs); one lane issues
    const bool one = elect_one();
    int item = 0, committed = -1;
    for (int pass = 0; pass < 2 * my_tiles && ok; ++pass) {
      if (pass >= 1)
        ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(accempty), static_cast<uint32_t>((pass - 1) & 1), S.st,
                                               S.timeout_ns));
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const bool low = pass & 1;
      for (int q = 0; q < nchunks; ++q, ++item) {
        const int st = item % kStages;
        ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&full[st]), static_cast<uint32_t>((item / kStages) & 1),
                                               S.st, S.timeout_ns));
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t a = umma_desc(smem_u32(sm) + st * kStageBytes, 256);
        if (one) {
          if (low) {
            const uint64_t b = a + kLowDigits * (kBlock >> 4);
            if (q == 0)
              chunk_products<0, kLowDigits, true>(tmem, a, b);
            else
              chunk_products<0, kLowDigits, false>(tmem, a, b);
          } else {
            const uint64_t b = a + kDigits * (kBlock >> 4);
            if (q == 0)
              chunk_products<4, kDigits, true>(tmem, a, b);
            else
              chunk_products<4, kDigits, false>(tmem, a, b);
          }
          umma_commit(smem_u32(&empty[st]));
        }
        committed = item;
      }
      if (!ok) break;
      if (one) umma_commit(smem_u32(accfull));
    }
    if (committed >= 0)  // the MMAs issued finish before the accumulators are released
      mbar_finish(smem_u32(&empty[committed % kStages]), static_cast<uint32_t>((committed / kStages) & 1),
                  globaltimer_ns());
  } else {
    const int half = (warp >> 2) * kCols;  // first column of this warp's part
    double* sb = scales + warp * kCols;
    const uint32_t tacc = tmem + static_cast<uint32_t>(half) + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    auto wait_full = [&](int pass) {
      const bool got = mbar_wait(smem_u32(accfull), static_cast<uint32_t>(pass & 1), S.st, S.timeout_ns);
      if (!__all_sync(0xffffffffu, got)) return false;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      return true;
    };
    auto release = [&]() {
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(accempty));
    };
    for (int m = 0; m < my_tiles; ++m) {
      int I, J;
      tile_of(m, I, J);
      const int i0 = r.t0 + I * kTile, j0 = r.t0 + J * kTile + half;
      const int iw = i0 + (warp & 3) * 32;  // this warp's 32 rows, kCols columns from j0
      const int ir = iw + (lane >> 2), jc = j0 + 2 * (lane & 3);
      const double* sap = S.sa + (ir - r.t0);
      const double sa[4] = {sap[0], sap[8], sap[16], sap[24]};
      __syncwarp();  // every lane is done with the last tile's scales
      if (lane < kCols / 2)
        *reinterpret_cast<double2*>(sb + 2 * lane) = *reinterpret_cast<const double2*>(S.sb + (j0 - r.t0) + 2 * lane);
      __syncwarp();
      double* cp = S.c + static_cast<long long>(ir) * S.ldc + jc;
      const long long step = 8 * S.ldc;
      const bool inside = i0 >= r.e && i0 + kTile <= S.n && i0 + kTile <= j0 && j0 + kCols <= S.n;
      auto mine = [&](int q, int c) {  // row ir + 8 q, column jc + c of the trailing upper triangle
        const int i = ir + 8 * q, j = jc + c;
        return i >= r.e && i < S.n && j >= r.e && j < S.n && i <= j;
      };
      // This thread's part of C, loaded while the MMAs of the first pass run:
      // v[h][g][.] holds rows 16 h .. 16 h + 15, columns 8 g .. 8 g + 7 as
      // tmem_ld16x8 has them (row ir + 8 q is q = 2 h + (x >> 1 & 1); four
      // lanes cover 64 bytes of it).
      double v[2][kCols / 8][4];
#pragma unroll
      for (int g = 0; g < kCols / 8; ++g)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          double* vv = &v[q >> 1][g][(q & 1) * 2];
          const double* p = cp + q * step + 8 * g;
          if (inside) {
            const double2 c = *reinterpret_cast<const double2*>(p);
            vv[0] = c.x;
            vv[1] = c.y;
          } else {
            vv[0] = mine(q, 8 * g) ? p[0] : 0.0;
            vv[1] = mine(q, 8 * g + 1) ? p[1] : 0.0;
          }
        }
      // v -= the four levels' sums, joined as an integer below 2^51 (exactly
      // a double, exactly scaled): each entry of C is rounded twice
      auto drain = [&](double unit) {
        double su[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) su[q] = sa[q] * unit;
#pragma unroll
        for (int k = 0; k < kCols / 4; ++k) {
          const int h = k / (kCols / 8), g = k % (kCols / 8);
          int d[4][4];
#pragma unroll
          for (int l = 0; l < 4; ++l)
            tmem_ld16x8(tacc + (static_cast<uint32_t>(16 * h) << 16) + l * kTile + 8 * g, d[l]);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          const double2 s2 = *reinterpret_cast<const double2*>(sb + 8 * g + 2 * (lane & 3));
#pragma unroll
          for (int x = 0; x < 4; ++x) {
            const double t = int_to_double(static_cast<long long>(d[0][x]) * 16777216 +
                                           static_cast<long long>(d[1][x]) * 65536 +
                                           static_cast<long long>(d[2][x]) * 256 + d[3][x]);
            v[h][g][x] = __fma_rn(-t, su[2 * h + (x >> 1)] * (x & 1 ? s2.y : s2.x), v[h][g][x]);
          }
        }
      };
      if (!(ok = wait_full(0))) break;
      drain(1.0);
      release();
      if (!(ok = wait_full(1))) break;
      drain(4294967296.0);
      release();
      if (skip[m]) continue;
#pragma unroll
      for (int g = 0; g < kCols / 8; ++g)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const double* vv = &v[q >> 1][g][(q & 1) * 2];
          double* p = cp + q * step + 8 * g;
          if (inside) {
            *reinterpret_cast<double2*>(p) = make_double2(vv[0], vv[1]);
          } else {
            if (mine(q, 8 * g)) p[0] = vv[0];
            if (mine(q, 8 * g + 1)) p[1] = vv[1];
          }
        }
    }
  }
  if (!ok) {
    atomicCAS(const_cast<int*>(&S.st->status), 0, BBK_ERR_TIMEOUT);
    atomicExch(const_cast<int*>(&S.st->abort), 1);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (warp == kEpiWarps + 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
}

}  // namespace

// Launches the digit update of `panel` where it applies (see the rule below);
// *gate and *marks then say what is left to the FP64 kernel that the caller
// launches behind it (the flag: 0 nothing, 1 the panel, 2 the marked tiles).
int launch_update_i8(const FactorPlan& plan, int panel, long long order, const int** gate,
                     const unsigned char** marks, cudaStream_t s) {
  *gate = nullptr;
  *marks = nullptr;
  // Sorting out digits, scales and the bound costs about 40 us per panel whatever the
  // width, and a tile's epilogue the same for any k, so the line lies at a
  // product of order and width (n = 8000, ms per factorization with the
  // digit update, without the bound, down to order 1024 / 2048 / 4096 / 6144 / never:
  // block 256: 3.74 / 3.71 / 3.95 / 4.93 / 6.67; block 128: 6.12 / 6.02 / 6.06 /
  // 6.61 / 7.72; block 64: 10.7 / 10.5 / 10.1 / 9.87 / 9.76), and at a width, since
  // the FP64 kernel of a narrow panel waits for C as well (ms per factorization with
  // digits / without: n = 24000, block 48: 407 / 377, 64: 340 / 346, 80: 302 / 330, 96:
  // 276 / 320; n = 12000: 93.7 / 92.4, 86.6 / 86.2, 81.5 / 83.3, 77.7 / 81.6).
  if (order * plan.b < 512 * 1024 || order < 1024 || plan.b < 64) return BBK_OK;
  const long long npad = plan.ldw;
  const size_t mags = static_cast<size_t>(npad) * plan.kpad;
  const size_t digits = kDigits * mags;
  const size_t tiles = static_cast<size_t>(npad / kTile + 1) * (npad / kTile + 2) / 2;
  // the digits live in what the update phase leaves idle of the workspace:
  // U's in the BF16 operands' buffer, with the scales and marks behind them, W's in
  // the panel kernel's slot-ordered U and W (one after the other)
  char* hs = static_cast<char*>(plan.hsplit);
  char* us = reinterpret_cast<char*>(plan.uslot);
  const size_t us_room = static_cast<size_t>(reinterpret_cast<char*>(plan.wslot) - us) +
                         static_cast<size_t>(plan.b + 2) * npad * sizeof(double);
  const size_t hs_need = digits + mags + 2 * npad * sizeof(double) + (2 * plan.kpad + 2) * sizeof(unsigned long long) +
                         2 * npad * sizeof(int) + tiles;
  const int sms = device_sm_count();
  const long long tm = order / kTile + 2;
  const int grid = static_cast<int>(std::min<long long>(tm * (tm + 1) / 2, sms));
  // (what depends on the panel is above: once a factorization's panels come
  // here, which starts with the first, they all do until `order` is too small)
  if (tiles > static_cast<size_t>(kMaxTiles) * sms || plan.kpad > kMaxK || digits + mags > us_room ||
      hs_need > 12 * plan.hstride || reinterpret_cast<uintptr_t>(hs) % 16 ||
      reinterpret_cast<uintptr_t>(us) % 16)
    return BBK_OK;
  SliceArgs S{};
  S.st = plan.state;
  S.panel = panel;
  S.n = plan.n;
  S.u = plan.ucm;
  S.ldu = plan.ldu;
  S.w = plan.w;
  S.ldw = plan.ldw;
  S.c = plan.a;
  S.ldc = plan.lda;
  S.nkc = plan.kpad / kChunk;
  S.da = reinterpret_cast<unsigned char*>(hs);
  S.db = reinterpret_cast<unsigned char*>(us);
  S.ma = S.da + digits;
  S.mb = S.db + digits;
  S.sa = reinterpret_cast<double*>(hs + digits + mags);
  S.sb = S.sa + npad;
  S.wmax = reinterpret_cast<unsigned long long*>(S.sb + npad);
  S.flag = reinterpret_cast<int*>(S.wmax + 2 * plan.kpad);
  S.count = S.flag + 2;
  S.ta = S.flag + 4;
  S.tb = S.ta + npad;
  S.marks = reinterpret_cast<unsigned char*>(S.tb + npad);
  S.timeout_ns = wait_timeout_ns();
  if (panel == 0)
    BBK_CUDA_TRY(cudaMemsetAsync(S.wmax, 0, (2 * plan.kpad + 2) * sizeof(unsigned long long), s));
  static std::once_flag attr_once[64];
  int dev = 0;
  BBK_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return set_error(BBK_ERR_NO_DEVICE, "device %d out of range", dev);
  cudaError_t attr_err = cudaSuccess;
  std::call_once(attr_once[dev], [&] {
    attr_err = cudaFuncSetAttribute(i8_update_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    static_cast<int>(kSmem));
    if (attr_err == cudaSuccess)
      attr_err = cudaFuncSetAttribute(bound_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      static_cast<int>(kBoundSmem));
  });
  BBK_CUDA_TRY(attr_err);
  const int segs = static_cast<int>(std::max(1LL, std::min(16LL, order / 2048)));
  row_max_kernel<<<dim3(segs, plan.b + 1), 256, 0, s>>>(S);
  BBK_CUDA_TRY(cudaGetLastError());
  const int slices = static_cast<int>(std::min<long long>(4 * sms, 2 * ((order + 256) / 32)));
  slice_kernel<<<slices, 256, plan.kpad * sizeof(int), s>>>(S);
  BBK_CUDA_TRY(cudaGetLastError());
  bound_kernel<<<grid, kThreads, kBoundSmem, s>>>(S);
  BBK_CUDA_TRY(cudaGetLastError());
  i8_update_kernel<<<grid, kThreads, kSmem, s>>>(S);
  BBK_CUDA_TRY(cudaGetLastError());
  count_launch(4);
  *gate = S.flag + (panel & 1);
  *marks = S.marks;
  return BBK_OK;
}

}  // namespace bbk
