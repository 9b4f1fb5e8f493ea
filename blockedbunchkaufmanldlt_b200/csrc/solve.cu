// Solve A X = B with compact Bunch-Kaufman factors, and the dense
// reconstruction P^T L D L^T P.
//
// The reference has no solve; L and D are read exactly as its stress test
// reads them (tests/block_ldlt_large_stress_test.cc:160-194 in
// wentianshu/BlockedBunchKaufmanLDLT): L(i,k) = F(k,i) for k < i, except
// L(k+1,k) = 0 when a 2x2 pivot starts at k; D(k,k) = F(k,k) and
// D(k,k+1) = F(k,k+1) for that 2x2.  With (P A P^T)(i,j) = A(perm[i], perm[j]):
//   y = B[perm]; L z = y; D w = z; L^T v = w; X[perm] = v.
// Each triangular sweep is a persistent cooperative launch over 64-row
// blocks in sweep order: CTA c owns blocks c, c+G, ...; a solved block is
// published with a release flag.  The owner of a block gathers the
// contributions of all earlier blocks into it, the old ones while the blocks
// just before it are still being solved elsewhere, then solves its triangle
// with inverses it formed meanwhile, or by substitution where they have grown.
// The critical path per block is one flag, one fold and three 32 x 32 products.
// Right-hand sides go in groups of eight, up to sixteen groups side by side on
// CTAs of their own.
// Measured: n = 10000, 1 right-hand side: 1.72 -> 1.32 ms (4.2 us per block);
// n = 5000, 64: 11.4 -> 1.51 ms.  A block that is substituted through takes 2.7
// us more.  Orders of one block gain nothing: a sweep of n = 64 takes 11 us, 8
// before.
#include <algorithm>
#include <mutex>

#include "bbk_internal.cuh"

namespace bbk {
namespace {

constexpr int kSB = 64;           // solve block
constexpr int kSolveThreads = 256;
constexpr int kMaxRhsChunk = 8;   // right-hand sides of a group
// Groups per launch.  A block step's latency does not depend on how many
// groups run beside it, and the folds' work is shared by all CTAs either way
// (ms per solve with 1 / 2 / 4 / 8 / 16 groups at most: n = 5000, 64
// right-hand sides: 6.87 / 3.61 / 2.12 / 1.49 / 1.49; n = 16000, 256: 100 / 63 /
// 49 / 44 / 43; a sweep that reads the factor once for all of them: 11.4 and
// 162).
constexpr int kMaxGroups = 16;
// Beyond this many right-hand sides the backward sweep adds the sums of every
// kWindow blocks over the lanes and sets them aside.  A lane's one running sum over
// all columns has an error that grows with n: mean backward error of 64 right-hand
// sides, n = 2000, 5000, 10000: 7.1e-16, 1.4e-15, 2.4e-15, with the sums set aside
// 7.0e-16, 1.0e-15, 1.3e-15 (the sweep that read the factor once for all of them, and
// subtracted block by block: 6.8e-16, 1.0e-15, 1.5e-15).  It takes 4 % longer (n =
// 5000, 64: 1.45 -> 1.51 ms; with the lanes' sums kept apart in shared memory
// 1.58).  Up to kPlainRhs the sums never were split, and are not.
constexpr int kPlainRhs = 32;
constexpr int kWindow = 16;
constexpr int kAhead = 4;         // factor blocks prefetched into L2 ahead of the fold

__global__ void gather_kernel(int n, int nrhs, const double* b, long long ldb, const int* perm,
                              double* y) {
  const long long total = static_cast<long long>(n) * nrhs;
  for (long long t = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; t < total;
       t += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int c = static_cast<int>(t / n), i = static_cast<int>(t % n);
    y[t] = b[c * ldb + perm[i]];
  }
}

__global__ void scatter_kernel(int n, int nrhs, double* b, long long ldb, const int* perm,
                               const double* y) {
  const long long total = static_cast<long long>(n) * nrhs;
  for (long long t = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; t < total;
       t += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int c = static_cast<int>(t / n), i = static_cast<int>(t % n);
    b[c * ldb + perm[i]] = y[t];
  }
}

// D w = z for all right-hand sides.
__global__ void dsolve_kernel(int n, int nrhs, const double* f, long long ldf, const int* pt,
                              double* y) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    if (pt[k] == -2) continue;  // handled with its partner
    if (pt[k] == 2 && k + 1 < n) {
      const double d11 = f[k * ldf + k], d21 = f[k * ldf + k + 1], d22 = f[(k + 1) * ldf + k + 1];
      const double det = d11 * d22 - d21 * d21;
      const double i11 = d22 / det, i22 = d11 / det, i21 = -d21 / det;
      for (int c = 0; c < nrhs; ++c) {
        double* yc = y + static_cast<long long>(c) * n;
        const double x = yc[k], z = yc[k + 1];
        yc[k] = i11 * x + i21 * z;
        yc[k + 1] = i21 * x + i22 * z;
      }
    } else {
      const double d = f[k * ldf + k];
      for (int c = 0; c < nrhs; ++c) {
        double* yc = y + static_cast<long long>(c) * n;
        yc[k] = d == 0.0 ? 0.0 : yc[k] / d;
      }
    }
  }
}

struct SweepArgs {
  int n;
  int nrhs;
  const double* f;
  long long ldf;
  const int* pt;
  double* y;       // n x nrhs (ld n), solved in place
  int* flags;      // per block: == mark once the block is solved in this sweep
  int* status;     // nonzero: a wait ran out; every CTA returns
  int mark;
  unsigned long long timeout_ns;
  int group_ctas;  // CTAs that share a group of kMaxRhsChunk right-hand sides
};

__device__ __forceinline__ int ld_acquire_s32(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void cp_async_8z(double* smem_dst, const double* gsrc, bool valid) {
  const unsigned saddr = static_cast<unsigned>(__cvta_generic_to_shared(smem_dst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(saddr), "l"(gsrc), "r"(valid ? 8 : 0)
               : "memory");
}

constexpr int kTriPitch = kSB + 1;
constexpr int kInvTmp = 2 * 16 * 17;  // scratch of invert_unit_triangle, doubles
static_assert(kInvTmp <= 4 * kMaxRhsChunk * kSB, "it fits the partial sums' space");
constexpr size_t kSweepSmem = (2 * kSB * kTriPitch + 4 * kMaxRhsChunk * kSB + kMaxRhsChunk * kSB) * sizeof(double);

// One sweep for up to kMaxGroups groups of kMaxRhsChunk right-hand sides, each
// with CTAs and flags of its own.  CTA c of a group owns blocks c, c+G, ... in
// sweep order and handles one at a time: it inverts the triangle's two 32 x 32
// diagonal blocks, folds in the contribution of every earlier block (in sweep
// order) as soon as that block is solved, then solves the block's own triangle
// by products with them and raises its flag.  Contributions of blocks solved
// long ago stream in while the blocks just before this one are still being
// solved elsewhere, so the critical path per block is one flag, one load of
// the newest solved block, its fold, the reduction and the triangle.
//   forward: thread (row, quarter) accumulates L(i, kg) y(kg) over its
//     quarter of each earlier block (warp loads of F rows are contiguous in
//     i); the four quarters are added at the end.
//   backward: warp w owns rows i = 8w..8w+7 and lane l the columns kg = l,
//     l + 32 of each later block (F rows are contiguous in kg); the lanes
//     are added by a butterfly at the end.
// Each warp learns which blocks are solved on its own (one relaxed scan of
// up to 32 flags, one acquire load of the newest set one, or a bounded wait
// on the next), so no CTA barrier is taken per block.
// Substitution through every triangle, one right-hand side per warp, took 2.7
// of 5.5 us per block; the inverses are ready before the block's turn.
__device__ __forceinline__ int ld_relaxed_flag(const int* p) {
  int v;
  asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Makes block k (and every block before it in sweep order) visible to this
// warp; returns the newest block in sweep order known to be solved (>= k in
// sweep order), or `fail` when the wait ran out or another CTA gave up.
template <bool kForward>
__device__ int warp_wait_solved(const SweepArgs& A, int k, int k_end, int fail) {
  const int lane = threadIdx.x & 31;
  const int dir = kForward ? 1 : -1;
  const int idx = k + dir * lane;
  const bool valid = kForward ? idx <= k_end : idx >= k_end;
  const bool set = valid && ld_relaxed_flag(A.flags + idx) == A.mark;
  const unsigned run = __ballot_sync(0xffffffffu, set);
  const int m = run == 0xffffffffu ? 32 : __ffs(~run) - 1;  // solved blocks from k on, in order
  int top = fail;
  if (lane == 0) {
    if (m > 0) {
      top = k + dir * (m - 1);
      (void)ld_acquire_s32(A.flags + top);
    } else {
      // the bound is checked after every unsuccessful poll (a poll is an L2
      // round trip), the other CTAs' status every 32 polls
      const unsigned long long t0 = globaltimer_ns();
      for (unsigned it = 1;; ++it) {
        if (ld_acquire_s32(A.flags + k) == A.mark) {
          top = k;
          break;
        }
        if (globaltimer_ns() - t0 > A.timeout_ns) {
          atomicCAS(A.status, 0, BBK_ERR_TIMEOUT);
          break;
        }
        if ((it & 31u) == 0 && ld_relaxed_s32(A.status) != 0) break;
      }
    }
  }
  top = __shfl_sync(0xffffffffu, top, 0);
  __syncwarp();
  return top;
}

// inv <- the inverses of the two 32 x 32 diagonal blocks of the unit lower
// triangle in tri (64 x 64; both by columns: entry (i, k) at [k * kTriPitch
// + i], entries not below the diagonal zero in tri).  Their 16 x 16 diagonal
// blocks by substitution, one column per thread, then the blocks below by
// X21 = -X22 (L21 X11).  Only terms of the triangles enter (an infinity
// times a zero beside them would not be a zero).  tmp: kInvTmp doubles.
// (The inverse of the whole triangle left residuals 6 to 15 % larger than
// substitution does, n = 1000 and 2000; these leave the same.)
// Bunch-Kaufman does not bound L, and a product with an inverse is as accurate
// as substitution only while the inverse does not grow.  So the inverse is not
// used (*unusable is set) where an entry of it exceeds kGrowth times the largest
// of 1 and its row's (backward: column's) entries of the triangle.  32 x 32
// blocks with every entry below the diagonal c, largest backward error by
// substitution / by the inverse, growth: c = -0.1: 1.3e-16 / 1.8e-16, 1.7; -0.12:
// 1.1e-16 / 3.1e-16, 3.6; -0.15: 1.2e-16 / 7.5e-16, 9.9; -0.3: 9e-17 / 2.8e-14, 786;
// -0.5: 8e-17 / 1.4e-12.  Blocks of Bunch-Kaufman factors of random, KKT and
// spectral matrices: up to 4.3, 8 blocks of 1000 above 4.
constexpr double kGrowth = 4.0;

template <bool kForward>
__device__ void invert_unit_triangle(const double* tri, double* inv, double* tmp, int* unusable) {
  constexpr int P = kTriPitch;
  const int t = threadIdx.x;
  for (int idx = t; idx < kSB * P; idx += kSolveThreads) inv[idx] = 0.0;
  __syncthreads();
  if (t < kSB) {
    const int base = t & ~15, j = t & 15;
    double x[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      double acc = 0.0;
#pragma unroll
      for (int k = 0; k < i; ++k) {
        const double l = k >= j ? tri[(base + k) * P + base + i] : 0.0;
        acc = __fma_rn(l, x[k], acc);
      }
      x[i] = i == j ? 1.0 : i < j ? 0.0 : -acc;
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) inv[(base + j) * P + base + i] = x[i];
  }
  __syncthreads();
  {
    const int i = t & 15, c = t >> 4;
    for (int b = 0; b < kSB; b += 32) {
      double acc = 0.0;
#pragma unroll
      for (int k = 0; k < 16; ++k) {
        const double l = k >= c ? tri[(b + k) * P + b + 16 + i] : 0.0;
        acc = __fma_rn(l, inv[(b + c) * P + b + k], acc);
      }
      tmp[(b / 32) * 16 * 17 + c * 17 + i] = acc;
    }
    __syncthreads();
    for (int b = 0; b < kSB; b += 32) {
      double acc = 0.0;
#pragma unroll
      for (int k = 0; k < 16; ++k) {
        const double v = k <= i ? tmp[(b / 32) * 16 * 17 + c * 17 + k] : 0.0;
        acc = __fma_rn(inv[(b + 16 + k) * P + b + 16 + i], v, acc);
      }
      inv[(b + c) * P + b + 16 + i] = -acc;
    }
  }
  __syncthreads();
  // four threads per row (column) of its diagonal block
  const int row = t >> 2, base = (row & ~31) + (t & 3) * 8;
  auto at = [&](const double* m, int k) { return fabs(kForward ? m[(base + k) * P + row] : m[row * P + base + k]); };
  double limit = 1.0;
#pragma unroll
  for (int k = 0; k < 8; ++k) limit = fmax(limit, at(tri, k));
  limit = fmax(limit, __shfl_xor_sync(0xffffffffu, limit, 1));
  limit = kGrowth * fmax(limit, __shfl_xor_sync(0xffffffffu, limit, 2));
  bool grown = false;
#pragma unroll
  for (int k = 0; k < 8; ++k) grown = grown || !(at(inv, k) <= limit);
  if (grown) *unusable = 1;
}

// The block's triangle, by halves h (backward: the transpose, the second half
// first): x_h = inv(T_hh) (r_h - T_hg x_g) for the right-hand sides in ys.
// Each product is 32 x 32: warp w takes the terms 4 w.. of row `lane`, the
// eight partial sums are added by the thread of (right-hand side, row), which
// returns its entries lane and lane + 32 of the solution.
template <bool kForward>
__device__ __forceinline__ void solve_triangle(const double* tri, const double* inv, double* red, double* ys, int nc,
                                               double& x0, double& x1) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int cc0 = warp;
  auto product = [&](const double* m, int rows, int terms) -> double {
    double acc[kMaxRhsChunk];
#pragma unroll
    for (int cc = 0; cc < kMaxRhsChunk; ++cc) acc[cc] = 0.0;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int k = 4 * warp + u;
      const double e = kForward ? m[(terms + k) * kTriPitch + rows + lane] : m[(rows + lane) * kTriPitch + terms + k];
#pragma unroll
      for (int cc = 0; cc < kMaxRhsChunk; ++cc)
        if (cc < nc) acc[cc] = __fma_rn(e, ys[cc * kSB + terms + k], acc[cc]);
    }
#pragma unroll
    for (int cc = 0; cc < kMaxRhsChunk; ++cc)
      if (cc < nc) red[(warp * kMaxRhsChunk + cc) * 32 + lane] = acc[cc];
    __syncthreads();
    double sum = 0.0;
    if (cc0 < nc) {
      double v[8];
#pragma unroll
      for (int w = 0; w < 8; ++w) v[w] = red[(w * kMaxRhsChunk + cc0) * 32 + lane];
      sum = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
    }
    return sum;
  };
  constexpr int g = kForward ? 0 : 32, h = 32 - g;
  double* yo = ys + cc0 * kSB;
  const double xg = product(inv, g, g);
  __syncthreads();  // every term of r_g is read, and every partial sum
  if (cc0 < nc) yo[g + lane] = xg;
  __syncthreads();
  const double th = product(tri, h, g);
  __syncthreads();
  if (cc0 < nc) yo[h + lane] -= th;
  __syncthreads();
  const double xh = product(inv, h, h);
  x0 = kForward ? xg : xh;
  x1 = kForward ? xh : xg;
}

// The same by substitution, a right-hand side per warp: its entries lane and
// lane + 32 in x0, x1, the solution to y.  Terms outside the triangle and the
// coupling entries of 2x2 pivots (types pt) do not enter.  (Where the inverse is
// not used, and where a result is not finite.)
template <bool kForward>
__device__ __forceinline__ void substitute(const double* tri, int bsz, const int* pt, double x0, double x1, double* y) {
  const int i0 = threadIdx.x & 31, i1 = i0 + 32;
  const bool in0 = i0 < bsz, in1 = i1 < bsz;
  const unsigned lo = __ballot_sync(0xffffffffu, in0 && pt[i0] == 2);
  const unsigned hi = __ballot_sync(0xffffffffu, in1 && pt[i1] == 2);
  const unsigned long long opens = static_cast<unsigned long long>(hi) << 32 | lo;  // bit k: a 2x2 starts at row k
  if (!in0) x0 = 0.0;
  if (!in1) x1 = 0.0;
  if (kForward) {
    // row i takes the columns k < i, less the one that its 2x2 pivot couples
    const int end0 = !in0 || i0 == 0 ? 0 : i0 - static_cast<int>(opens >> (i0 - 1) & 1);
    const int end1 = !in1 ? 0 : i1 - static_cast<int>(opens >> (i1 - 1) & 1);
#pragma unroll 4
    for (int k = 0; k < kSB; ++k) {
      const double e0 = tri[k * kTriPitch + i0], e1 = tri[k * kTriPitch + i1];
      const double xk = __shfl_sync(0xffffffffu, k < 32 ? x0 : x1, k & 31);
      if (k < end0) x0 = __fma_rn(-e0, xk, x0);
      if (k < end1) x1 = __fma_rn(-e1, xk, x1);
    }
  } else {
    const int end0 = !in0 ? kSB : i0 + static_cast<int>(opens >> i0 & 1);
    const int end1 = !in1 ? kSB : i1 + static_cast<int>(opens >> i1 & 1);
#pragma unroll 4
    for (int k = kSB - 1; k >= 0; --k) {
      const double e0 = tri[i0 * kTriPitch + k], e1 = tri[i1 * kTriPitch + k];
      const double xk = __shfl_sync(0xffffffffu, k < 32 ? x0 : x1, k & 31);
      if (k > end0) x0 = __fma_rn(-e0, xk, x0);
      if (k > end1) x1 = __fma_rn(-e1, xk, x1);
    }
  }
  if (i0 < bsz) y[i0] = x0;
  if (i1 < bsz) y[i1] = x1;
}

template <bool kForward, bool kAside>
__global__ void __launch_bounds__(kSolveThreads, 1) psweep_kernel(SweepArgs A) {
  extern __shared__ double psm[];
  double* tri = psm;                            // [kSB][kTriPitch]: the block's triangle, by columns
  double* inv = tri + kSB * kTriPitch;          // its inverse
  double* red = inv + kSB * kTriPitch;          // [4][kMaxRhsChunk][kSB] partial sums
  double* ys = red + 4 * kMaxRhsChunk * kSB;    // [kMaxRhsChunk][kSB]: the block being solved
  __shared__ int s_fail, s_grown;
  const int n = A.n;
  const long long ldf = A.ldf;
  const int nblk = (n + kSB - 1) / kSB;
  // this CTA's group of right-hand sides and its place in it
  const int G = A.group_ctas, c = blockIdx.x % G, group = blockIdx.x / G;
  const int nc = min(kMaxRhsChunk, A.nrhs - group * kMaxRhsChunk);
  A.y += static_cast<long long>(group) * kMaxRhsChunk * n;
  A.flags += static_cast<long long>(group) * nblk;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int dir = kForward ? 1 : -1;
  const int my_first = kForward ? c : (nblk - 1) - ((nblk - 1 - c) % G);
  if (kForward ? my_first >= nblk : my_first < 0) return;
  const int my_last = kForward ? c + ((nblk - 1 - c) / G) * G : c;
  const int kNone = kForward ? -1 : nblk;  // "no block" in sweep order
  const int kFail = kForward ? -2 : nblk + 1;
  auto stage_tri = [&](int b) {
    const int b0 = b * kSB, bsz = min(n, b0 + kSB) - b0;
    for (int idx = t; idx < kSB * kSB; idx += kSolveThreads) {
      const int r = idx / kSB, cc = idx % kSB;
      // L(cc, r) = F(b0 + r, b0 + cc), r < cc, except the entry of a 2x2
      const bool ok = r < cc && cc < bsz && !(cc == r + 1 && A.pt[b0 + r] == 2);
      cp_async_8z(&tri[r * kTriPitch + cc], ok ? A.f + static_cast<long long>(b0 + r) * ldf + b0 + cc : A.f, ok);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  if (t == 0) s_fail = 0;
  __syncthreads();
  int known = kNone;  // per warp: newest block (sweep order) known to be solved
  stage_tri(my_first);
  for (int b = my_first; kForward ? b <= my_last : b >= my_last; b += dir * G) {
    const int b0 = b * kSB, bsz = min(n, b0 + kSB) - b0;
    // the triangle's inverse, while earlier blocks are still being solved
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    // (but for the first block's, which is waited for)
    const bool opens = b == (kForward ? 0 : nblk - 1);
    if (t == 0) s_grown = opens;
    if (!opens) invert_unit_triangle<kForward>(tri, inv, red, &s_grown);
    // this block's right-hand sides, for the threads that finish them
    double yin[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int idx = t + h * kSolveThreads, cc = idx / kSB, r = idx % kSB;
      yin[h] = cc < nc && r < bsz ? A.y[static_cast<long long>(cc) * n + b0 + r] : 0.0;
    }
    // the 32 KB of the factor that fold k reads, into L2 (one 128-byte line
    // per thread: 64 rows of 4 lines; a row's lines may straddle a fifth)
    auto prefetch_f = [&](int k) {
      const int a = t >> 2, seg = (t & 3) * 16;
      const int x = kForward ? k * kSB + a : b0 + a;    // factor row
      const int y0 = kForward ? b0 + seg : k * kSB + seg;  // first column
      if (x < n && y0 < n) {
        const double* p = A.f + static_cast<long long>(x) * ldf + y0;
        asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
        asm volatile("prefetch.global.L2 [%0];" ::"l"(p + min(15, n - 1 - y0)));
      }
    };
    const int k_first = kForward ? 0 : nblk - 1;
    const int k_end = b - dir;  // the last block folded into b (sweep order)
    const bool any = kForward ? b > 0 : b < nblk - 1;
    bool fail = false;
    if (kForward) {
      const int row = t & (kSB - 1), quarter = t >> 6;
      const int i = b0 + row;
      double acc[kMaxRhsChunk];
#pragma unroll
      for (int cc = 0; cc < kMaxRhsChunk; ++cc) acc[cc] = 0.0;
      auto load_f = [&](int k, double (&l)[kSB / 4]) {
        const int k0 = k * kSB, bs = min(n, k0 + kSB) - k0;
        const bool edge = k == b - 1 && A.pt[k0 + bs - 1] == 2;  // 2x2 across the boundary
#pragma unroll
        for (int u = 0; u < kSB / 4; ++u) {
          const int kk = quarter * (kSB / 4) + u, kg = k0 + kk;
          const bool ok = i < n && kk < bs && !(edge && i == kg + 1);
          l[u] = ok ? A.f[static_cast<long long>(kg) * ldf + i] : 0.0;
        }
      };
      // lane l: entries l, l + 32, ... of (cc, u) = (e / 16, e % 16) of
      // this quarter's solved values of block k
      auto load_y = [&](int k, double (&yv)[kMaxRhsChunk / 2]) {
        const int kq = k * kSB + quarter * (kSB / 4);
#pragma unroll
        for (int e2 = 0; e2 < kMaxRhsChunk / 2; ++e2) {
          const int e = lane + 32 * e2, cc = e >> 4, u = e & 15;
          yv[e2] = cc < nc && kq + u < n ? __ldcg(A.y + static_cast<long long>(cc) * n + kq + u) : 0.0;
        }
      };
      double fc[kSB / 4], fn[kSB / 4];
      for (int k = k_first; any && k < k_first + kAhead && k <= k_end; ++k) prefetch_f(k);
      if (any) load_f(k_first, fc);
      for (int k = k_first; any && k <= k_end; ++k) {
        if (k + kAhead <= k_end) prefetch_f(k + kAhead);
        if (k < k_end) load_f(k + 1, fn);
        if (k > known) {
          known = warp_wait_solved<true>(A, k, k_end, kFail);
          if (known == kFail) {
            fail = true;
            known = k_end;
          }
        }
        // this quarter's 16 x nc solved values, all loaded at once and each
        // broadcast to the warp by a shuffle
        double yl[kMaxRhsChunk / 2];
        load_y(k, yl);
#pragma unroll
        for (int u = 0; u < kSB / 4; ++u)
#pragma unroll
          for (int cc = 0; cc < kMaxRhsChunk; ++cc)
            if (cc < nc) {
              const double yv = __shfl_sync(0xffffffffu, yl[(cc * 16 + u) >> 5], (cc * 16 + u) & 31);
              acc[cc] = __fma_rn(fc[u], yv, acc[cc]);
            }
#pragma unroll
        for (int u = 0; u < kSB / 4; ++u) fc[u] = fn[u];
      }
#pragma unroll
      for (int cc = 0; cc < kMaxRhsChunk; ++cc)
        if (cc < nc) red[(quarter * kMaxRhsChunk + cc) * kSB + row] = acc[cc];
    } else {
      // rows 8 warp .. 8 warp + 7 of the block, columns lane and lane + 32 of block k
      double acc[8][kMaxRhsChunk];
#pragma unroll
      for (int j = 0; j < 8; ++j)
#pragma unroll
        for (int cc = 0; cc < kMaxRhsChunk; ++cc) acc[j][cc] = 0.0;
      // add the 64 sums of (j, cc) over the lanes by recursive halving: at
      // offset o each lane keeps one half of its values and adds the
      // partner's copy of that half; after five levels lane l holds the
      // totals of entries 2l and 2l + 1 (62 shuffles, depth 5)
      static_assert(8 * kMaxRhsChunk == 64, "the halving below assumes 64 sums per lane");
      auto add_lanes = [&](double& s0, double& s1) {
        double v[64];
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
          for (int cc = 0; cc < kMaxRhsChunk; ++cc) v[j * kMaxRhsChunk + cc] = acc[j][cc];
#pragma unroll
        for (int o = 16, m = 64; o > 0; o >>= 1, m >>= 1) {
          const bool up = (lane & o) != 0;
#pragma unroll
          for (int e = 0; e < m / 2; ++e) {
            const double send = up ? v[e] : v[e + m / 2];
            const double keep = up ? v[e + m / 2] : v[e];
            v[e] = keep + __shfl_xor_sync(0xffffffffu, send, o);
          }
        }
        s0 = v[0];
        s1 = v[1];
      };
      double aside0 = 0.0, aside1 = 0.0;  // the totals of the windows before
      auto load_f = [&](int k, double (&l)[16]) {
        const int k0 = k * kSB;
        const bool edge = k == b + 1 && b0 + kSB - 1 < n && A.pt[b0 + kSB - 1] == 2;
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int ii = b0 + warp * 8 + j, kg = k0 + lane + 32 * h;
            const bool ok = ii < n && kg < n && !(edge && kg == ii + 1);
            l[j * 2 + h] = ok ? A.f[static_cast<long long>(ii) * ldf + kg] : 0.0;
          }
      };
      double fc[16], fn[16];
      for (int k = k_first; any && k > k_first - kAhead && k >= k_end; --k) prefetch_f(k);
      if (any) load_f(k_first, fc);
      for (int k = k_first; any && k >= k_end; --k) {
        if (k - kAhead >= k_end) prefetch_f(k - kAhead);
        if (k > k_end) load_f(k - 1, fn);
        if (k < known) {
          known = warp_wait_solved<false>(A, k, k_end, kFail);
          if (known == kFail) {
            fail = true;
            known = k_end;
          }
        }
        double yv[2][kMaxRhsChunk];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int kg = k * kSB + lane + 32 * h;
#pragma unroll
          for (int cc = 0; cc < kMaxRhsChunk; ++cc)
            yv[h][cc] = cc < nc && kg < n ? __ldcg(A.y + static_cast<long long>(cc) * n + kg) : 0.0;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int cc = 0; cc < kMaxRhsChunk; ++cc)
              if (cc < nc) acc[j][cc] = __fma_rn(fc[j * 2 + h], yv[h][cc], acc[j][cc]);
#pragma unroll
        for (int u = 0; u < 16; ++u) fc[u] = fn[u];
        if (kAside && (k_first - k) % kWindow == kWindow - 1 && k > k_end) {
          double s0, s1;
          add_lanes(s0, s1);
          aside0 += s0;
          aside1 += s1;
#pragma unroll
          for (int j = 0; j < 8; ++j)
#pragma unroll
            for (int cc = 0; cc < kMaxRhsChunk; ++cc) acc[j][cc] = 0.0;
        }
      }
      double v[2];
      add_lanes(v[0], v[1]);
      if (kAside) {
        v[0] += aside0;
        v[1] += aside1;
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int e = 2 * lane + h, j = e / kMaxRhsChunk, cc = e % kMaxRhsChunk;
        if (cc < nc) red[cc * kSB + warp * 8 + j] = v[h];
      }
    }
    if (fail) s_fail = 1;
    __syncthreads();
    if (s_fail) return;  // uniform: the status word already says why
    // ---- this block's right-hand sides less the folded sums
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int idx = t + h * kSolveThreads, cc = idx / kSB, r = idx % kSB;
      if (cc < nc) {
        double sum;
        if (kForward)
          sum = (red[(0 * kMaxRhsChunk + cc) * kSB + r] + red[(1 * kMaxRhsChunk + cc) * kSB + r]) +
                (red[(2 * kMaxRhsChunk + cc) * kSB + r] + red[(3 * kMaxRhsChunk + cc) * kSB + r]);
        else
          sum = red[cc * kSB + r];
        ys[cc * kSB + r] = any ? yin[h] - sum : yin[h];
      }
    }
    __syncthreads();
    // ---- the block's triangle.  The zeros beside a diagonal block's triangle
    // are harmless while everything is finite, and what is not shows in the
    // result; then once more by substitution, as where the inverse has grown.
    // (The products run either way, the flag waits in shared memory and the
    // substitution is inline: with a branch around the products, a register for
    // the flag or a call, n = 10000 took 1.37 to 1.47 ms.)
    const int cc0 = t >> 5;  // this thread's right-hand side
    double* yc = A.y + static_cast<long long>(cc0) * n + b0;
    const double r0 = cc0 < nc ? ys[cc0 * kSB + lane] : 0.0, r1 = cc0 < nc ? ys[cc0 * kSB + 32 + lane] : 0.0;
    double x0, x1;
    solve_triangle<kForward>(tri, inv, red, ys, nc, x0, x1);
    if (cc0 < nc) {
      if (lane < bsz) yc[lane] = x0;
      if (lane + 32 < bsz) yc[lane + 32] = x1;
    }
    if (__syncthreads_or(s_grown || !(isfinite(x0) && isfinite(x1)))) {
      if (cc0 < nc) substitute<kForward>(tri, bsz, A.pt + b0, r0, r1, yc);
    }
    __syncthreads();
    if (t == 0) {
      fence_acq_rel_gpu();
      asm volatile("st.relaxed.gpu.global.b32 [%0], %1;" ::"l"(A.flags + b), "r"(A.mark) : "memory");
    }
    const int nb = b + dir * G;
    if (kForward ? nb <= my_last : nb >= my_last) stage_tri(nb);  // the buffers are free again
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
}

__global__ void reset_flags_kernel(int* flags, int count) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) flags[i] = 0;
}

// L(row, col) of the compact factors: unit diagonal, F(col, row) below it
// except the coupling entry of a 2x2 pivot (ExtractRegularFactorsFromCompact,
// src/block_ldlt_decomposition.cc:746-763).
__device__ __forceinline__ double l_entry(const double* f, long long ldf, const int* pt, int row, int col) {
  if (row == col) return 1.0;
  if (row < col) return 0.0;
  if (pt[col] == 2 && row == col + 1) return 0.0;
  return f[static_cast<long long>(col) * ldf + row];
}

// M = L D and U = L^T (both ld x ld, zero outside the order n): the two
// operands of the reconstruction product.
__global__ void ld_lt_kernel(int n, const double* f, long long ldf, const int* pt, long long ld, double* m,
                             double* u) {
  const long long total = ld * ld;
  for (long long t = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; t < total;
       t += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int i = static_cast<int>(t / ld), k = static_cast<int>(t % ld);
    double mv = 0.0, uv = 0.0;
    if (i < n && k < n) {
      if (pt[k] == 2 && k + 1 < n) {
        mv = l_entry(f, ldf, pt, i, k) * f[k * ldf + k] + l_entry(f, ldf, pt, i, k + 1) * f[k * ldf + k + 1];
      } else if (pt[k] == -2 && k > 0) {
        mv = l_entry(f, ldf, pt, i, k - 1) * f[(k - 1) * ldf + k] + l_entry(f, ldf, pt, i, k) * f[k * ldf + k];
      } else {
        mv = l_entry(f, ldf, pt, i, k) * f[k * ldf + k];
      }
      uv = l_entry(f, ldf, pt, k, i);  // U(i, k) = L(k, i)
    }
    m[t] = mv;
    u[t] = uv;
  }
}

// out(perm[i], perm[j]) = (L D L^T)(i, j) = -C(min(i,j), max(i,j)).
__global__ void rec_scatter_kernel(int n, const double* c, long long ld, const int* perm, double* out,
                                   long long ldo) {
  const long long total = static_cast<long long>(n) * n;
  for (long long t = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; t < total;
       t += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int i = static_cast<int>(t / n), j = static_cast<int>(t % n);
    const int lo = min(i, j), hi = max(i, j);
    out[static_cast<long long>(perm[i]) * ldo + perm[j]] = -c[static_cast<long long>(lo) * ld + hi];
  }
}

// Dense L (unit lower) and D (block diagonal) from the compact factors.
__global__ void extract_ld_kernel(int n, const double* f, long long ldf, const int* pt, double* l, long long ldl,
                                  double* d, long long ldd) {
  const long long total = static_cast<long long>(n) * n;
  for (long long t = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; t < total;
       t += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int i = static_cast<int>(t / n), k = static_cast<int>(t % n);
    if (l) l[static_cast<long long>(i) * ldl + k] = l_entry(f, ldf, pt, i, k);
    if (d) {
      double v = 0.0;
      if (i == k) {
        v = f[static_cast<long long>(i) * ldf + i];
      } else if (k == i + 1 && pt[i] == 2) {
        v = f[static_cast<long long>(i) * ldf + k];
      } else if (i == k + 1 && pt[k] == 2) {
        v = f[static_cast<long long>(k) * ldf + i];
      }
      d[static_cast<long long>(i) * ldd + k] = v;
    }
  }
}

constexpr int kMaxAttrDevices = 64;
std::once_flag g_sweep_attr[kMaxAttrDevices];

int grid_for(long long work, int threads) {
  const long long g = (work + threads - 1) / threads;
  return static_cast<int>(std::max(1LL, std::min(g, 4096LL)));
}

}  // namespace

size_t solve_work_doubles(int n, int nrhs) { return 2 * static_cast<size_t>(n) * nrhs; }

int* solve_status_word(double* work, int n, int nrhs) {
  return reinterpret_cast<int*>(work + static_cast<long long>(n) * nrhs);
}

int solve_status(double* work, int n, int nrhs, cudaStream_t s) {
  int h = BBK_OK;
  BBK_CUDA_TRY(cudaMemcpyAsync(&h, solve_status_word(work, n, nrhs), sizeof(int), cudaMemcpyDeviceToHost, s));
  BBK_CUDA_TRY(cudaStreamSynchronize(s));
  if (h != BBK_OK) return set_error(h, "solve aborted on the device: %s", bbk_status_string(h));
  return BBK_OK;
}

// work: 2 n nrhs doubles: the right-hand sides being solved in place, then
// the status word and the block flags (one set per group of right-hand sides).
int solve_enqueue(int n, const double* f, long long ldf, const int* perm, const int* pivot_types,
                  int nrhs, double* b, long long ldb, double* work, cudaStream_t s) {
  double* y = work;
  const long long total = static_cast<long long>(n) * nrhs;
  const int nblk = (n + kSB - 1) / kSB;
  int* status = solve_status_word(work, n, nrhs);
  int* flags = status + 1;
  const int ngroups = (nrhs + kMaxRhsChunk - 1) / kMaxRhsChunk;
  const int nflags = 1 + ngroups * nblk;
  reset_flags_kernel<<<std::max(1, std::min(64, (nflags + 255) / 256)), 256, 0, s>>>(status, nflags);
  BBK_CUDA_TRY(cudaGetLastError());
  count_launch();
  gather_kernel<<<grid_for(total, 256), 256, 0, s>>>(n, nrhs, b, ldb, perm, y);
  BBK_CUDA_TRY(cudaGetLastError());
  count_launch();
  SweepArgs A{n, nrhs, f, ldf, pivot_types, y, flags, status, 1, wait_timeout_ns(), 1};
  // both sweeps need more than the default 48 KB of dynamic shared memory;
  // the attributes are set per device, each under its own once-flag
  // (callers may be on several host threads)
  int dev = 0;
  BBK_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxAttrDevices) return set_error(BBK_ERR_NO_DEVICE, "device %d out of range", dev);
  cudaError_t attr_err = cudaSuccess;
  std::call_once(g_sweep_attr[dev], [&] {
    const void* fns[3] = {reinterpret_cast<const void*>(psweep_kernel<true, false>),
                          reinterpret_cast<const void*>(psweep_kernel<false, false>),
                          reinterpret_cast<const void*>(psweep_kernel<false, true>)};
    for (int i = 0; i < 3 && attr_err == cudaSuccess; ++i)
      attr_err = cudaFuncSetAttribute(fns[i], cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      static_cast<int>(kSweepSmem));
  });
  BBK_CUDA_TRY(attr_err);
  const int sms = device_sm_count();
  // every sweep launch waits for its own flag value
  int mark = 0;
  auto sweeps = [&](bool forward) -> int {
    const bool aside = !forward && nrhs > kPlainRhs;
    const void* fn = forward ? reinterpret_cast<const void*>(psweep_kernel<true, false>)
                     : aside ? reinterpret_cast<const void*>(psweep_kernel<false, true>)
                             : reinterpret_cast<const void*>(psweep_kernel<false, false>);
    constexpr int chunk = kMaxGroups * kMaxRhsChunk;
    for (int c0 = 0; c0 < nrhs; c0 += chunk) {
      SweepArgs a = A;
      a.y = y + static_cast<long long>(c0) * n;
      a.nrhs = std::min(chunk, nrhs - c0);
      a.mark = ++mark;
      const int groups = (a.nrhs + kMaxRhsChunk - 1) / kMaxRhsChunk;
      a.group_ctas = std::max(1, std::min(nblk, sms / groups));
      void* kargs[] = {&a};
      BBK_CUDA_TRY(cudaLaunchCooperativeKernel(fn, dim3(groups * a.group_ctas), dim3(kSolveThreads), kargs,
                                               kSweepSmem, s));
      count_launch();
    }
    return BBK_OK;
  };
  int rc = sweeps(true);
  if (rc) return rc;
  dsolve_kernel<<<grid_for(n, 256), 256, 0, s>>>(n, nrhs, f, ldf, pivot_types, y);
  BBK_CUDA_TRY(cudaGetLastError());
  count_launch();
  rc = sweeps(false);
  if (rc) return rc;
  scatter_kernel<<<grid_for(total, 256), 256, 0, s>>>(n, nrhs, b, ldb, perm, y);
  BBK_CUDA_TRY(cudaGetLastError());
  count_launch();
  return BBK_OK;
}

size_t reconstruct_work_doubles(int n) {
  const size_t ld = align_up(static_cast<size_t>(n), 128);
  return 3 * ld * ld;
}

// P^T L D L^T P: M = L D and U = L^T formed on the device, the upper tiles
// of M U on the FP64 tensor cores (the trailing-update tile kernels with
// C = 0), then mirrored and permuted.  work: reconstruct_work_doubles(n).
int reconstruct_enqueue(int n, const double* f, long long ldf, const int* perm,
                        const int* pivot_types, double* out, long long ldo, double* work,
                        cudaStream_t s) {
  const long long ld = static_cast<long long>(align_up(static_cast<size_t>(n), 128));
  double* m = work;
  double* u = m + ld * ld;
  double* c = u + ld * ld;
  BBK_CUDA_TRY(cudaMemsetAsync(c, 0, static_cast<size_t>(ld * ld) * sizeof(double), s));
  ld_lt_kernel<<<grid_for(ld * ld, 256), 256, 0, s>>>(n, f, ldf, pivot_types, ld, m, u);
  BBK_CUDA_TRY(cudaGetLastError());
  count_launch();
  int rc = launch_upper_product(n, m, u, ld, c, s);
  if (rc) return rc;
  rec_scatter_kernel<<<grid_for(static_cast<long long>(n) * n, 256), 256, 0, s>>>(n, c, ld, perm, out, ldo);
  BBK_CUDA_TRY(cudaGetLastError());
  count_launch();
  return BBK_OK;
}

int extract_ld_enqueue(int n, const double* f, long long ldf, const int* pivot_types, double* l, long long ldl,
                       double* d, long long ldd, cudaStream_t s) {
  extract_ld_kernel<<<grid_for(static_cast<long long>(n) * n, 256), 256, 0, s>>>(n, f, ldf, pivot_types, l, ldl,
                                                                                 d, ldd);
  BBK_CUDA_TRY(cudaGetLastError());
  count_launch();
  return BBK_OK;
}

}  // namespace bbk
