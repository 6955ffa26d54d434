// reduce.cuh — deterministic fp64 sums over term arrays, in two selectable orders.
//
// Every reduction of the engine first materialises its per-element terms (double), then a
// SumPlan reduces them. Two orders:
//   exact: the reference CPU's own order. kSeq = one sequential chain (the reference's plain
//          host loops, e.g. kkt_general, cpu_backend.cpp:226-284); kChunk64 = 64 contiguous
//          chunks summed sequentially, then the 64 partials in order (la::parallel_sum,
//          parallel.h:169-188, used by Backend::dot / diff_norm2). Each chain's result is the
//          sequential chain's bit for bit, computed in parallel (k_xstat / k_xwalk below): the
//          order is exactly i = lo, lo+1, … as far as rounding can tell.
//   fast:  a fixed two-level tree (kTreeBlocks blocks per sum, block tree, then one block
//          combines the partials) — deterministic run to run, but a different rounding.
// Maxima never go through a SumPlan: they are taken with integer atomics on non-negative
// doubles, which is order-independent and exact.
#pragma once

#include <climits>
#include <vector>

#include "common.cuh"

namespace b200 {

enum class SumOrder { kSeq, kChunk64 };

struct TreeSeg {
  const double* t;
  long long lo, hi;
  double init;
  double* out;
};

constexpr int kTreeBlocks = 96;
constexpr int kChunks = 64;  // la::kReduceChunks

__device__ __forceinline__ double block_sum_fixed(double v, double* sh) {
  for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(kFull, v, off);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) sh[wid] = v;
  __syncthreads();
  if (wid == 0) {
    v = lane < static_cast<int>(blockDim.x >> 5) ? sh[lane] : 0.0;
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(kFull, v, off);
  }
  return v;  // valid in thread 0
}

// ------------------------------------------------------------------ exact chains, in parallel
// A chain s = init; s = fl(s + t[i]) for i = lo, lo+1, … is inherently sequential, and walking
// 2.5 million terms with one warp costs milliseconds. It is evaluated here in parallel, with the
// sequential chain's result bit for bit, from one property of round-to-nearest-even: while every
// partial sum stays inside one binade [2^e, 2^(e+1)) (ulp u = 2^(e−52)), each partial sum is an
// integer multiple S·u, and fl(S·u + t) = (S + k)·u with k = rint(t/u) — or, when t/u = f + ½ is a
// tie, k = f or f + 1, whichever makes S + k even. So inside such a run the chain is an integer
// walk whose only dependence on the past is the parity of S: a run of terms is summarised by its
// effect for each of the two parities (XRun), and effects compose associatively. So:
//   k_xstat   per tile of kXTile terms (one warp): an approximate fp64 sum, in any order; only used
//             to guess each tile's binade. A kernel that produces the terms may leave it itself. Long chains:
//             k_xspan adds them up by spans of kXSpan tiles.
//   k_xwalk   one warp per tile, kXWarps tiles per block: the guessed binade's u from the approximate
//             start (the approximate sums of the chain's earlier tiles), then the tile's XRun (change of
//             S, bounds of its running value, parity after, per parity before): each lane adds its terms
//             in fp64 to an approximate start of either parity, and the differences of the sums' bits are
//             the changes of S. A tile whose running sum changes binade once is summarised in three parts:
//             the run before the term that changes it, that term, the run after it in the new grid. The
//             block that finishes last of a group of kXGroup tiles composes the tiles' summaries into the
//             group's, of the same form (the first group's start is known, so it is walked instead, as
//             below, to its exact sum). The block that finishes last of a chain's walks the chain with the
//             EXACT s, with one warp: a run of groups is committed as s ← (S0 + K[S0 mod 2])·u as far as s = S0·u lies in their binade and
//             every running S provably stays within [2^52 + 1, 2^53 − 1] (then each exact partial sum
//             lies inside the binade, at least u/2 from its ends, and rounds to that grid); a group that
//             changes binade is committed by its three parts; any other one is walked by its tiles in the
//             same way; and the terms of a tile that cannot be committed are added one by one (x_add), so
//             that zeros, subnormals, infinities and NaN get exactly the sequential chain's arithmetic.
//             A chain of at most kXShort terms is added one by one from the start.
// The approximations only choose between two exact paths; the result never depends on them.
//
// What bounds it: latency. A dependent fp64 addition takes 8.3 cycles, 10.4 with its operand from
// shared memory, so a tile added one by one takes 1.4 us; the first one's terms are added while the others
// are summarised, and the few tiles that cross a binade more than once cost that in the walk. Its other
// steps are one check over 32 summaries held by the warp's lanes, and at a crossing one lane's x_commit, on
// integers and without a branch, run by every lane before the warp knows which one it is: a warp alone takes
// 5 or 6 cycles for an instruction, so a step is as long as its longest chain of them. Tiles of 256 terms,
// one warp's, keep the tiles that must be added one by one cheap. The first group, where most binades are
// crossed, is walked by its own last block, beside the other groups' composition. Of 14 us for the 525,600
// terms of the staircase T = 8760 the tiles take 5, the first group 2.5, the count of groups 1, the walk 4.5.
// Measured, 15,000 / 525,600 / 1.5M uniform terms, one launch by itself from cold caches: 16.8 / 18.5 / 33.8 us
// (15,000 in three launches over tiles of 2,048 terms, walked in windows with a scan and a restart per crossing:
// 68 us).
constexpr int kXPer = 8;              // terms per lane
constexpr int kXTile = 32 * kXPer;    // terms per tile (one warp)
constexpr int kXGroup = 32;           // tiles per group (one warp lane each)
constexpr int kXWarps = 8;            // warps per block of k_xwalk, tiles per block
constexpr long long kXShort = 1024;   // chains up to this long are added one by one by a warp
// Every block adds up the approximate sums of all tiles before its own: the reads grow with the square of the
// chain. In chains of more than kXSpanMin tiles (3M terms) the tiles come in spans of kXSpan whose sums k_xspan
// makes first, so that a block reads at most one span's tiles and the spans before it. One call, without / with
// spans: 8M terms 165 / 157 us, 16M 326 / 257, 64M 1.91 / 0.87 ms, 256M 22.8 / 3.4; 4.5M 108 / 111 us.
constexpr int kXSpan = 1024, kXSpanMin = 12288;

struct XChain {
  const double* t;
  long long lo, hi;  // terms t[lo, hi)
  double init;
  double* out;
  int tile0, ntiles;    // this chain's tiles in the tile arrays (ntiles = 0: added one by one)
  int group0, ngroups;  // its groups of kXGroup tiles
  int block0;           // its first block of kXWarps tiles
  int span0;            // its first span (−1: none)
  int job;              // its kChunk64 job (−1: *out is the chain's own result)
};
// A kChunk64 job: the chains of its chunks leave their sums in part[0, chunks); the chain that
// finishes last adds them in order (la::parallel_sum).
struct XJob {
  const double* part;
  int chunks;
  double init;
  double* out;
};
// The effect of a run of terms on S (the partial sum in units of u), for S even (index 0) and
// odd (1) at the run's start: K the change of S; mn / mx bounds of the running change over positions
// 1…len in units of 2^24, rounded outward (INT_MAX / INT_MIN for an empty run); out the parity after; bad: it
// cannot be told; ties: the two parities' changes differ somewhere (else a run is plain integer sums).
struct alignas(16) XRun {
  long long K[2];
  int mn[2], mx[2];
  int out[2];
  int bad, ties;
};
// A tile's summary: its terms before the split counted in the grid of binade e (that of the tile's
// approximate start), the term where the approximate running sum leaves that binade (split = false: none
// does) added as a plain fp64 addition, the terms after it counted in the grid of the binade e1 that the
// running sum moved to. A group's summary has the same form (its split is the tile that changes binade).
struct alignas(16) XTileAgg {
  double at;  // the term at the split
  int e, e1;
  XRun pre, suf;
  bool split;
};
// What a walk reads of every summary: a run in one grid without ties is complete here (kXPlain); one with
// ties or a change of binade is looked up in full (kXFull); kXNone: no summary; kXStart: the chain's
// first terms, added one by one from its start (the bits of that sum are K). first, len: the tile's terms,
// where a walk needs them from here.
enum : int { kXPlain = 0, kXFull = 1, kXNone = 2, kXStart = 3 };
struct alignas(16) XFast {
  long long K;
  int e;
  int mn, mx;
  int first;
  int kind, len;
};
struct XSummary {  // as it is made
  XFast fast;
  XTileAgg full;
};

constexpr long long kX52 = 1LL << 52, kX53 = 1LL << 53;
constexpr int kXShift = 24;  // the bounds' unit
// x in that unit, rounded down or up; far values (which no check lets pass) stay far.
__device__ __forceinline__ int x_down(long long x) {
  x >>= kXShift;
  return static_cast<int>(x < -(1LL << 29) - 64 ? -(1LL << 29) - 64 : (x > (1LL << 29) + 64 ? (1LL << 29) + 64 : x));
}
__device__ __forceinline__ int x_up(long long x) { return x_down(x + ((1LL << kXShift) - 1)); }

__device__ __forceinline__ XRun x_identity() {
  XRun r;
  r.K[0] = r.K[1] = 0;
  r.mn[0] = r.mn[1] = INT_MAX;
  r.mx[0] = r.mx[1] = INT_MIN;
  r.out[0] = 0, r.out[1] = 1;
  r.bad = r.ties = 0;
  return r;
}
// e = floor(log2 |v|) for a normal v whose ulp 2^(e−52) and 2^(52−e) are both normal doubles;
// otherwise returns false.
__device__ __forceinline__ bool x_binade(double v, int& e) {
  const long long bits = __double_as_longlong(v);
  const int ef = static_cast<int>((bits >> 52) & 0x7ff);
  if (ef == 0 || ef == 0x7ff) return false;  // zero, subnormal, inf, NaN
  e = ef - 1023;
  return e >= -970 && e <= 1023;
}
// The sign and exponent of v: two numbers of which one lies in a binade lie in the same one, with the
// same sign, where these agree.
__device__ __forceinline__ int x_top(double v) { return __double2hiint(v) >> 20; }
// A normal s as an integer multiple S of its binade's ulp, |S| in [2^52, 2^53), and back (by its bits).
__device__ __forceinline__ long long x_int(double s) {
  const long long b = __double_as_longlong(s), m = (b & (kX52 - 1)) | kX52;
  return b < 0 ? -m : m;
}
__device__ __forceinline__ double x_double(long long S, int e) {
  const long long a = S < 0 ? -S : S;
  return __longlong_as_double((a & (kX52 - 1)) | (static_cast<long long>(e + 1023) << 52) | (S < 0 ? LLONG_MIN : 0LL));
}
// The composition of the warp's runs in lane order (in every lane). A run's effect on the parity is to
// keep it, to turn it, or to leave it at 0 or 1 whatever it was, so three ballots tell the parity before each
// lane, and with it which K is that lane's; then it is one prefix sum for each parity at the start.
__device__ __forceinline__ XRun x_warp_ordered(const XRun& r) {
  const int lane = threadIdx.x & 31;
  const bool any = r.mn[0] != INT_MAX;
  XRun x;
  x.bad = __any_sync(kFull, r.bad) ? 1 : 0;
  x.ties = __any_sync(kFull, r.ties) ? 1 : 0;
  if (!x.ties) {
    const long long K = r.K[0];
    long long inc = K;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const long long o = __shfl_up_sync(kFull, inc, off);
      if (lane >= off) inc += o;
    }
    x.K[0] = x.K[1] = __shfl_sync(kFull, inc, 31);
    x.mn[0] = x.mn[1] = __reduce_min_sync(kFull, any ? x_down(inc - K) + r.mn[0] : INT_MAX);
    x.mx[0] = x.mx[1] = __reduce_max_sync(kFull, any ? x_up(inc - K) + r.mx[0] : INT_MIN);
    x.out[0] = static_cast<int>(x.K[0] & 1), x.out[1] = x.out[0] ^ 1;
    return x;
  }
  const unsigned fixed = __ballot_sync(kFull, r.out[0] == r.out[1]), ones = __ballot_sync(kFull, r.out[0] & r.out[1]);
  const unsigned turns = __ballot_sync(kFull, r.out[0] & ~r.out[1] & 1);
  const unsigned below = (1u << lane) - 1u, known = fixed & below;
  const int last = known ? 31 - __clz(known) : 0;
  const unsigned after = known ? below & ~((2u << last) - 1u) : below;
  const int turned = __popc(turns & after) & 1;
  long long K[2], inc[2];
  int q[2];
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    q[p] = (known ? static_cast<int>((ones >> last) & 1u) : p) ^ turned;  // the parity before this lane
    K[p] = inc[p] = q[p] ? r.K[1] : r.K[0];
  }
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const long long o0 = __shfl_up_sync(kFull, inc[0], off), o1 = __shfl_up_sync(kFull, inc[1], off);
    if (lane >= off) inc[0] += o0, inc[1] += o1;
  }
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    x.K[p] = __shfl_sync(kFull, inc[p], 31);
    x.mn[p] = __reduce_min_sync(kFull, any ? x_down(inc[p] - K[p]) + (q[p] ? r.mn[1] : r.mn[0]) : INT_MAX);
    x.mx[p] = __reduce_max_sync(kFull, any ? x_up(inc[p] - K[p]) + (q[p] ? r.mx[1] : r.mx[0]) : INT_MIN);
    x.out[p] = __shfl_sync(kFull, q[p] ? r.out[1] : r.out[0], 31);
  }
  return x;
}
// Whether every S + r, mn ≤ r ≤ mx in units of 2^24, lies inside [2^52 + 1, 2^53 − 1] with the sign of S0
// (S: S0 plus the change before the run, |S| < 2^53; the answer for any other S means nothing).
__device__ __forceinline__ bool x_inside(long long S0, long long S, int mn, int mx) {
  constexpr int a = static_cast<int>(kX52 >> kXShift) + 1, b = static_cast<int>(kX53 >> kXShift) - 1;
  const int s = static_cast<int>(S >> kXShift);
  return (s + mn >= (S0 < 0 ? -b : a)) & (s + 1 + mx <= (S0 < 0 ? -a : b));
}

// 16 bytes another block wrote into shared memory, behind the instructions that follow.
__device__ __forceinline__ void x_copy16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
// A struct of 16-byte words another block wrote, read past this SM's L1.
template <class S>
__device__ __forceinline__ S x_load(const S* p) {
  static_assert(sizeof(S) % 16 == 0, "whole 16-byte words");
  S v;
  const uint4* src = reinterpret_cast<const uint4*>(p);
  uint4* dst = reinterpret_cast<uint4*>(&v);
#pragma unroll
  for (unsigned k = 0; k < sizeof(S) / 16; ++k) dst[k] = __ldcg(src + k);
  return v;
}

__device__ __forceinline__ void x_tile_range(const XChain& c, int tile, long long& a, long long& b) {
  a = c.lo + static_cast<long long>(tile - c.tile0) * kXTile;
  b = a + kXTile < c.hi ? a + kXTile : c.hi;
}

// s + t[a] + t[a+1] + … + t[b−1], one rounding per addition in that order; every lane of the warp
// calls it with the same s and returns the same sum. The terms come in chunks of kXTile through the
// warp's shared buffer `sh` (16-byte aligned), the next chunk on its way while one is added. Places
// past the end hold −0.0, which leaves every s as it is (−0.0 included).
__device__ __forceinline__ double x_add(const double* t, long long a, long long b, double s, double* sh) {
  const int lane = threadIdx.x & 31;
  double nx[kXPer];
#pragma unroll
  for (int q = 0; q < kXPer; ++q) nx[q] = a + q * 32 + lane < b ? __ldcg(t + a + q * 32 + lane) : -0.0;
  for (long long pos = a; pos < b; pos += kXTile) {
    __syncwarp();  // the previous chunk has been read
#pragma unroll
    for (int q = 0; q < kXPer; ++q) sh[q * 32 + lane] = nx[q];
    __syncwarp();
#pragma unroll
    for (int q = 0; q < kXPer; ++q) {
      const long long i = pos + kXTile + q * 32 + lane;
      nx[q] = i < b ? __ldcg(t + i) : -0.0;
    }
    const int cnt = b - pos < kXTile ? static_cast<int>(b - pos) : kXTile;
    const double2* p = reinterpret_cast<const double2*>(sh);
    double2 v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = p[q];
    for (int i = 0; i < cnt; i += 8) {  // 8 terms ahead in registers (wrapping at the buffer's end)
      double2 w[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) w[q] = p[((i >> 1) + 4 + q) & (kXTile / 2 - 1)];
#pragma unroll
      for (int q = 0; q < 4; ++q) s += v[q].x, s += v[q].y;
#pragma unroll
      for (int q = 0; q < 4; ++q) v[q] = w[q];
    }
  }
  return s;
}

// Blocks as k_xwalk's: kXWarps tiles of one chain each.
static __global__ void __launch_bounds__(32 * kXWarps) k_xstat(const XChain* ch, const int* block_chain, double* stat,
                                                               const int* skip) {
  if (skip && *skip) return;
  const XChain& c = ch[block_chain[blockIdx.x]];
  const int lane = threadIdx.x & 31;
  const int tile = c.tile0 + (static_cast<int>(blockIdx.x) - c.block0) * kXWarps + static_cast<int>(threadIdx.x >> 5);
  if (tile >= c.tile0 + c.ntiles) return;
  long long a, b;
  x_tile_range(c, tile, a, b);
  double v[kXPer], s = 0.0;
#pragma unroll
  for (int q = 0; q < kXPer; ++q) v[q] = a + q * 32 + lane < b ? c.t[a + q * 32 + lane] : 0.0;
#pragma unroll
  for (int q = 0; q < kXPer; ++q) s += v[q];
  for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(kFull, s, off);
  if (lane == 0) stat[tile] = s;
}
// Approximate sums of spans of tiles; one block each. span_chain: the chain.
static __global__ void __launch_bounds__(256) k_xspan(const XChain* ch, const int* span_chain, const double* stat, double* span,
                                                      const int* skip) {
  __shared__ double sh[32];
  if (skip && *skip) return;
  const XChain& c = ch[span_chain[blockIdx.x]];
  const int k0 = (static_cast<int>(blockIdx.x) - c.span0) * kXSpan;
  double s = 0.0;
  for (int k = k0 + static_cast<int>(threadIdx.x); k < min(k0 + kXSpan, c.ntiles); k += 256) s += stat[c.tile0 + k];
  s = block_sum_fixed(s, sh);
  if (threadIdx.x == 0) span[blockIdx.x] = s;
}
// A producer's own tile sum: called by every thread of a block of kXTile threads whose thread i
// made term i of tile blockIdx.x; stat may be null (a chain that needs none).
__device__ __forceinline__ void x_leave_stat(double* stat, double term) {
  __shared__ double sh[kXTile / 32];
  if (!stat) return;
  for (int off = 16; off > 0; off >>= 1) term += __shfl_xor_sync(kFull, term, off);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = term;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = sh[0];
    for (int w = 1; w < kXTile / 32; ++w) s += sh[w];
    stat[blockIdx.x] = s;
  }
}

__device__ __forceinline__ XTileAgg x_no_full() {
  XTileAgg T;
  T.at = 0.0, T.e = T.e1 = 0;
  T.pre = T.suf = x_identity();
  T.split = false;
  return T;
}

// One lane's terms v[q0, q1) added to a start of either parity near `start`, whose binade (top bits `top`)
// they are meant to stay in: for each parity the change of S, read off the bits; bounds of the running
// change in units of 2^24; and whether every sum had those top bits. Every double of a binade is a multiple
// of its ulp, so these are the chain's own steps for any start of that parity as far as it stays inside.
// The two sums are never more than two ulps apart, so the first one's bounds, widened, serve both: where the
// other could leave the binade the bounds are too near its end for any commit. start > 0.
struct XLane {
  long long K[2];
  int mn, mx;
  double end;  // the sum from `start` itself
  bool clean;
};
template <class V>
__device__ __forceinline__ XLane x_lane(V&& v, int q0, int q1, double start, int top) {
  XLane r;
  const double o0 = __longlong_as_double(__double_as_longlong(start) ^ 1);
  double s = start, o = o0;
  const auto mid = [](double x) {  // bits 24 … 55: the exponent's lowest and the fraction's highest
    return static_cast<unsigned>(__funnelshift_r(__double2loint(x), __double2hiint(x), kXShift));
  };
  int lo = __double2hiint(start), hi = lo;
  unsigned mn = mid(start), mx = mn;
#pragma unroll
  for (int q = 0; q < kXPer; ++q)
    if (q >= q0 && q < q1) {
      s += v(q), o += v(q);
      lo = min(lo, __double2hiint(s)), hi = max(hi, __double2hiint(s));
      mn = min(mn, mid(s)), mx = max(mx, mid(s));
    }
  r.end = s;
  r.clean = (lo >> 20) == top && (hi >> 20) == top;
  const long long b = __double_as_longlong(start);
  const long long same = __double_as_longlong(s) - b, other = __double_as_longlong(o) - __double_as_longlong(o0);
  const bool odd = (b & 1) != 0;
  r.K[0] = odd ? other : same, r.K[1] = odd ? same : other;
  r.mn = static_cast<int>(mn - mid(start)) - 2;
  r.mx = static_cast<int>(mx - mid(start)) + 2;
  return r;
}
// The composition of the warp's lanes in lane order (`in`: a lane's part counts, `any`: it has terms), valid
// in lane 0; flip: the terms' and the sum's signs were turned.
__device__ __forceinline__ XRun x_compose_lanes(const XLane& r, bool in, bool any, bool flip) {
  XRun x = x_identity();
  if (in && any) {
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      x.K[p] = flip ? -r.K[p] : r.K[p];
      x.out[p] = static_cast<int>((p + r.K[p]) & 1);
      x.mn[p] = flip ? -r.mx : r.mn, x.mx[p] = flip ? -r.mn : r.mx;
    }
    x.ties = r.K[0] != r.K[1];
  }
  return x_warp_ordered(x);
}

// One lane's terms of a tile t[a, b): kXPer from a + lane·kXPer, zeros past the end.
struct XTerms {
  double v[kXPer];
  int cnt;
};
__device__ __forceinline__ XTerms x_terms(const double* __restrict__ t, long long a, long long b) {
  const long long i0 = a + static_cast<long long>(threadIdx.x & 31) * kXPer;
  XTerms r;
  r.cnt = b - i0 >= kXPer ? kXPer : (b > i0 ? static_cast<int>(b - i0) : 0);
#pragma unroll
  for (int q = 0; q < kXPer; ++q) r.v[q] = q < r.cnt ? t[i0 + q] : 0.0;
  return r;
}
// The summary of a tile (one warp, its terms in the lanes) for a chain whose approximate sum before it is s0;
// valid in lane 0.
__device__ __forceinline__ XTileAgg x_tile_full(XTerms t, double s0) {
  const int lane = threadIdx.x & 31, cnt = t.cnt;
  XTileAgg g = x_no_full();
  int e0;
  if (!x_binade(s0, e0)) {  // uniform over the warp
    g.pre.bad = 1;
    return g;
  }
  const bool flip = s0 < 0;
  double(&v)[kXPer] = t.v;
#pragma unroll
  for (int q = 0; q < kXPer; ++q)
    if (flip) v[q] = -v[q];
  double run = 0.0;
#pragma unroll
  for (int q = 0; q < kXPer; ++q) run += v[q];
  double inc = run;
  for (int off = 1; off < 32; off <<= 1) {
    const double o = __shfl_up_sync(kFull, inc, off);
    if (lane >= off) inc += o;
  }
  const double start = (flip ? -s0 : s0) + (inc - run);  // this lane's approximate start
  const auto term = [&](int q) { return v[q]; };
  const int top0 = x_top(flip ? -s0 : s0);
  const XLane r = x_lane(term, 0, cnt, start, x_top(start));
  // lanes before k stay in s0's binade; lane k, if there is one, leaves it
  const unsigned left = __ballot_sync(kFull, cnt > 0 && !(r.clean && x_top(start) == top0));
  const int k = left ? __ffs(left) - 1 : 32;
  g.e = e0;
  if (k == 32) {
    g.pre = x_compose_lanes(r, true, cnt > 0, flip);
    return g;
  }
  // the term of lane k that leaves it, and its terms before and after that one
  int split = kXPer, top1 = 0;
  double at = 0.0, after = 0.0;
  XLane pre = r, suf = r;
  bool ok = lane < k || cnt == 0;
  if (lane == k) {
    double s = start;
#pragma unroll
    for (int q = 0; q < kXPer; ++q)
      if (q < cnt && split == kXPer) {
        s += v[q];
        if (x_top(s) != top0) split = q, at = v[q], after = s;
      }
    int e1;
    ok = x_top(start) == top0 && split < kXPer && after > 0 && x_binade(after, e1);
    top1 = x_top(after);
    pre = x_lane(term, 0, split, start, top0);
    suf = x_lane(term, split + 1, cnt, after, top1);
    ok = ok && pre.clean && suf.clean;
  }
  const int top1k = __shfl_sync(kFull, top1, k);
  if (lane > k) ok = cnt == 0 || (r.clean && x_top(start) == top1k);
  if (!__all_sync(kFull, ok)) {
    g.pre.bad = 1;
    return g;
  }
  g.pre = x_compose_lanes(pre, lane <= k, lane < k ? cnt > 0 : split > 0, flip);
  g.suf = x_compose_lanes(suf, lane >= k, lane > k ? cnt > 0 : split + 1 < cnt, flip);
  g.e1 = (top1k & 0x7ff) - 1023;
  g.split = true;
  at = __shfl_sync(kFull, at, k);
  g.at = flip ? -at : at;
  return g;
}

// A full summary's short form.
__device__ __forceinline__ XSummary x_summary(const XTileAgg& T) {
  XSummary r;
  r.full = T;
  r.fast.K = T.pre.K[0], r.fast.e = T.e, r.fast.mn = T.pre.mn[0], r.fast.mx = T.pre.mx[0];
  r.fast.first = 0, r.fast.len = 0;
  r.fast.kind = T.pre.bad ? kXNone : (T.split || T.pre.ties ? kXFull : kXPlain);
  return r;
}
__device__ __forceinline__ XFast x_no_fast() {
  XFast f;
  f.K = 0, f.e = 0, f.mn = INT_MAX, f.mx = INT_MIN, f.first = 0, f.kind = kXNone, f.len = 0;
  return f;
}
// The sum after the chain's first terms, as a summary (its walk starts with it).
__device__ __forceinline__ XSummary x_start(double s) {
  XSummary r;
  r.full = x_no_full();
  r.fast = x_no_fast();
  r.fast.kind = kXStart, r.fast.K = __double_as_longlong(s);
  return r;
}
__device__ __forceinline__ void x_leave(const XSummary& S, XFast* fast, XTileAgg* full) {  // one lane
  *fast = S.fast;
  if (S.fast.kind == kXFull) *full = S.full;
}

// Commits a whole summary, its change of binade included, to the sum S·2^(e − 52); returns false (S and e
// mean nothing) where a running S could leave its binade. Without a branch: a chain of about fifty
// instructions, which every lane can run for its own summary.
__device__ __forceinline__ bool x_commit(long long& S, int& e, const XTileAgg& T) {
  const bool odd = (S & 1) != 0;
  bool ok = (T.e == e) & ((T.pre.mn[0] == INT_MAX) |
                          x_inside(S, S, odd ? T.pre.mn[1] : T.pre.mn[0], odd ? T.pre.mx[1] : T.pre.mx[0]));
  // the term that changes the binade, as the chain adds it (no split: the term is zero)
  const double s = x_double(S + (odd ? T.pre.K[1] : T.pre.K[0]), e) + T.at;
  const int e1 = T.split ? T.e1 : T.e;
  e = ((__double2hiint(s) >> 20) & 0x7ff) - 1023;
  ok = ok & (e == e1);
  const long long R = x_int(s);
  const bool odd1 = (R & 1) != 0;
  ok = ok & ((T.suf.mn[0] == INT_MAX) |
             x_inside(R, R, odd1 ? T.suf.mn[1] : T.suf.mn[0], odd1 ? T.suf.mx[1] : T.suf.mx[0]));
  S = R + (odd1 ? T.suf.K[1] : T.suf.K[0]);
  return ok;
}

// What one lane holds of a walk's round of up to 32 summaries; `full` means something where the kind is
// kXFull (it is read whatever the kind, so that it need not wait for it).
struct XRound {
  XFast fast;
  XTileAgg full;
};
__device__ __forceinline__ XRound x_round(const XFast* fast, const XTileAgg* full, bool here) {
  XRound r;
  r.fast = x_no_fast(), r.full = x_no_full();
  if (here) r.fast = x_load(fast), r.full = x_load(full);
  return r;
}

// One warp walks cnt consecutive summaries, lane l holding the l-th, with the exact s. other(k, s) returns
// the sum after the k-th where its summary cannot be committed. A step commits all plain summaries up to
// the first that is not one, not in s's binade, or whose running S would leave it, and then that one by
// itself. Without ties a run's K does not depend on what came before, so one prefix sum over the lanes
// serves all steps (across a change of grid the sum means nothing, but a step only uses differences within
// one); and every lane commits its own summary to the sum that the step has there, if it gets that far,
// before the warp knows which lane that is: a step is then one x_commit long.
template <class F>
__device__ __forceinline__ double x_walk_lanes(double s, const XRound& G, int cnt, F&& other) {
  const int lane = threadIdx.x & 31;
  const bool here = lane < cnt;
  const bool plain = here && G.fast.kind == kXPlain, empty = plain && G.fast.mn == INT_MAX;
  const bool full = here && G.fast.kind == kXFull, start = here && G.fast.kind == kXStart;
  long long inc = plain ? G.fast.K : 0;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const long long o = __shfl_up_sync(kFull, inc, off);
    if (lane >= off) inc += o;
  }
  const long long before = inc - (plain ? G.fast.K : 0);
  int j = 0, e;
  bool have = x_binade(s, e);
  long long S = x_int(s), base = 0;  // base: `before` at lane j
  while (j < cnt) {
    const long long Sl = S + (before - base);  // the sum before this lane's summary
    const bool ok = plain & have & (empty | ((G.fast.e == e) & x_inside(S, Sl, G.fast.mn, G.fast.mx)));
    long long S2 = Sl;
    int e2 = e;
    const bool can = x_commit(S2, e2, G.full) & full & have;
    const unsigned stop = __ballot_sync(kFull, lane >= j && !ok);
    const int f = stop ? __ffs(stop) - 1 : 32;
    if (f >= cnt) {
      S = __shfl_sync(kFull, Sl + (plain ? G.fast.K : 0), cnt - 1);
      break;
    }
    // lane f, on its own. way: 1 committed, 2 the chain's start, 0 neither
    const int way = __shfl_sync(kFull, can ? 1 : (start ? 2 : 0), f);
    S = __shfl_sync(kFull, can ? S2 : (start ? G.fast.K : Sl), f);
    const int ef = __shfl_sync(kFull, e2, f);
    base = __shfl_sync(kFull, inc, f);
    j = f + 1;
    if (way == 1) {
      e = ef;
    } else {
      s = way == 2 ? __longlong_as_double(S) : other(f, have ? x_double(S, e) : s);
      have = x_binade(s, e);
      S = x_int(s);
    }
  }
  return have ? x_double(S, e) : s;
}

// The cnt tiles of chain c from its tile t0 on, from their summaries (one warp), with the exact s before them.
__device__ __forceinline__ double x_walk_tiles(const XChain& c, int t0, int cnt, double s, const XFast* tf, const XTileAgg* ag,
                                               double* sh) {
  const int lane = threadIdx.x & 31, ti = c.tile0 + t0;
  const XRound T = x_round(tf + ti + lane, ag + ti + lane, lane < cnt);
  return x_walk_lanes(s, T, cnt, [&](int k, double st) {
    long long a, b;
    x_tile_range(c, ti + k, a, b);
    return x_add(c.t, a, b, st, sh);
  });
}
__device__ __forceinline__ int x_group_tiles(const XChain& c, int g) {
  return min(kXGroup, c.ntiles - g * kXGroup);
}
// The chain c from its groups' summaries (one warp); the first one is its exact sum there. The next round's
// summaries come into shared memory while one is walked.
__device__ __forceinline__ double x_walk(const XChain& c, const XFast* tf, const XTileAgg* ag, const XFast* gf,
                                         const XTileAgg* gg, XRound (*stage)[32], double* sh) {
  const int lane = threadIdx.x & 31;
  const auto fetch = [&](int g0) {
    if (g0 + lane < c.ngroups) {
      XRound* r = &stage[(g0 >> 5) & 1][lane];
      const char* f = reinterpret_cast<const char*>(gf + c.group0 + g0 + lane);
      const char* a = reinterpret_cast<const char*>(gg + c.group0 + g0 + lane);
#pragma unroll
      for (unsigned k = 0; k < sizeof(XFast); k += 16) x_copy16(reinterpret_cast<char*>(&r->fast) + k, f + k);
#pragma unroll
      for (unsigned k = 0; k < sizeof(XTileAgg); k += 16) x_copy16(reinterpret_cast<char*>(&r->full) + k, a + k);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  double s = c.init;
  fetch(0);
  for (int g0 = 0; g0 < c.ngroups; g0 += 32) {
    const int cnt = c.ngroups - g0 < 32 ? c.ngroups - g0 : 32;
    fetch(g0 + 32);
    asm volatile("cp.async.wait_group 1;" ::: "memory");  // this lane's own, of this round
    XRound G = stage[(g0 >> 5) & 1][lane];
    if (lane >= cnt) G.fast = x_no_fast(), G.full = x_no_full();
    s = x_walk_lanes(s, G, cnt, [&](int g, double sg) {
      return x_walk_tiles(c, (g0 + g) * kXGroup, x_group_tiles(c, g0 + g), sg, tf, ag, sh);
    });
  }
  return s;
}

// The summary of a group of tiles (a warp; lane l takes the l-th of cnt), valid in lane 0: all tiles in one
// grid and none that changes binade, or one that does, with the tiles before it in its first grid and
// those after it in its second. Else it has none.
__device__ __forceinline__ XSummary x_group(const XFast* tf, const XTileAgg* ag, int cnt) {
  const int lane = threadIdx.x & 31;
  const bool here = lane < cnt;
  const XRound R = x_round(tf + lane, ag + lane, here);
  XTileAgg T = R.fast.kind == kXFull ? R.full : x_no_full();
  if (here && R.fast.kind == kXPlain) {
    T.e = R.fast.e;
    T.pre.K[0] = T.pre.K[1] = R.fast.K, T.pre.mn[0] = T.pre.mn[1] = R.fast.mn, T.pre.mx[0] = T.pre.mx[1] = R.fast.mx;
    T.pre.out[0] = static_cast<int>(R.fast.K & 1), T.pre.out[1] = T.pre.out[0] ^ 1;
  }
  const unsigned splits = __ballot_sync(kFull, here && T.split);
  const int k = splits ? __ffs(splits) - 1 : 31;  // the last lane in the first grid
  XTileAgg G = x_no_full();
  const int e0 = __shfl_sync(kFull, T.e, 0), e1 = splits ? __shfl_sync(kFull, T.e1, k) : e0;
  const bool ok = !here || ((R.fast.kind == kXPlain || R.fast.kind == kXFull) && T.e == (lane <= k ? e0 : e1));
  if (!__all_sync(kFull, ok) || __popc(splits) > 1) {
    G.pre.bad = 1;
    return x_summary(G);
  }
  G.e = e0;
  G.pre = x_warp_ordered(here && lane <= k ? T.pre : x_identity());
  if (splits) {
    G.e1 = e1, G.split = true;
    G.at = __shfl_sync(kFull, T.at, k);
    G.suf = x_warp_ordered(lane == k ? T.suf : (here && lane > k ? T.pre : x_identity()));
  }
  return x_summary(G);
}

// Blocks [0, nblocks): kXWarps tiles of one chain each (block_chain: the chain). The blocks after them:
// one chain of at most kXShort terms per warp (short_chain). done: counters of a group's finished blocks,
// a chain's finished groups and a job's finished chains; the last one goes on, and sets its counter back to
// zero for the next launch.
static __global__ void __launch_bounds__(32 * kXWarps) k_xwalk(const XChain* __restrict__ ch, const XJob* __restrict__ jobs,
                                                               const int* __restrict__ block_chain, int nblocks,
                                                               const int* __restrict__ short_chain, int nshort,
                                                               const double* stat, const double* span, XFast* tf,
                                                               XTileAgg* ag, XFast* gf,
                                                               XTileAgg* gg, unsigned* group_done, unsigned* chain_done,
                                                               unsigned* job_done, const int* skip) {
  __shared__ alignas(16) double sh_add[kXWarps][kXTile];
  __shared__ double sh_sum[kXWarps];
  // the walk's two rounds: in the buffers of the block's other warps, which are done by then
  static_assert(2 * 32 * sizeof(XRound) <= (kXWarps - 1) * kXTile * sizeof(double), "two rounds fit");
  XRound(*stage)[32] = reinterpret_cast<XRound(*)[32]>(&sh_add[1][0]);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const bool tiled = static_cast<int>(blockIdx.x) < nblocks;
  const int ks = (static_cast<int>(blockIdx.x) - nblocks) * kXWarps + w;
  const int ci = tiled ? block_chain[blockIdx.x] : ks < nshort ? short_chain[ks] : -1;
  XChain c;
  if (ci >= 0) c = ch[ci];
  pdl_wait();
  if (skip && *skip) return;
  double s;
  // counts one more at *counter; true in every lane of the warp that made it `of`
  auto last_of = [&](unsigned* counter, int of) {
    unsigned last = 0;
    if (lane == 0) {
      __threadfence();
      last = atomicAdd(counter, 1u) + 1u == static_cast<unsigned>(of) ? 1u : 0u;
      if (last) *counter = 0u;
    }
    last = __shfl_sync(kFull, last, 0);
    if (last) __threadfence();
    return last != 0;
  };
  if (tiled) {
    const int k0 = (static_cast<int>(blockIdx.x) - c.block0) * kXWarps, k = k0 + w;
    long long a, b;
    x_tile_range(c, c.tile0 + k, a, b);
    const XTerms mine_t = x_terms(c.t, a, b);  // none past the chain's last tile
    const double mine = lane < w && k0 + lane < c.ntiles ? stat[c.tile0 + k0 + lane] : 0.0;
    double pre = 0.0;  // the approximate sum before this block's tiles
    int from = 0;
    if (c.span0 >= 0) {
      from = k0 / kXSpan * kXSpan;
      for (int q = threadIdx.x; q < k0 / kXSpan; q += 32 * kXWarps) pre += span[c.span0 + q];
    }
    for (int q = from + static_cast<int>(threadIdx.x); q < k0; q += 32 * kXWarps) pre += stat[c.tile0 + q];
    for (int off = 16; off > 0; off >>= 1) pre += __shfl_xor_sync(kFull, pre, off);
    if (lane == 0) sh_sum[w] = pre;
    __syncthreads();
    double s0 = mine;
    for (int off = 16; off > 0; off >>= 1) s0 += __shfl_xor_sync(kFull, s0, off);
    s0 += c.init;
    for (int q = 0; q < kXWarps; ++q) s0 += sh_sum[q];
    if (k < c.ntiles) {
      // the first tile's start is known: its terms are added here, while the other tiles are summarised
      const XSummary T = k == 0 ? x_start(x_add(c.t, a, b, c.init, sh_add[0])) : x_summary(x_tile_full(mine_t, s0));
      if (lane == 0) x_leave(T, tf + c.tile0 + k, ag + c.tile0 + k);
    }
    __syncthreads();  // last_of's fence then covers what the other warps left
    if (w != 0) return;
    const int g = k0 / kXGroup, t0 = g * kXGroup, cnt = x_group_tiles(c, g);
    if (!last_of(group_done + c.group0 + g, (cnt + kXWarps - 1) / kXWarps)) return;
    // the first group's start is known too, so it is walked here, while the others are summarised
    if (g == 0) s = x_walk_tiles(c, 0, cnt, c.init, tf, ag, sh_add[0]);
    if (c.ngroups > 1) {
      const XSummary G = g == 0 ? x_start(s) : x_group(tf + c.tile0 + t0, ag + c.tile0 + t0, cnt);
      if (lane == 0) x_leave(G, gf + c.group0 + g, gg + c.group0 + g);
      if (!last_of(chain_done + ci, c.ngroups)) return;
      s = x_walk(c, tf, ag, gf, gg, stage, sh_add[0]);
    }
  } else {
    if (ci < 0) return;
    s = x_add(c.t, c.lo, c.hi, c.init, sh_add[w]);
  }
  if (lane == 0) *c.out = s;
  if (c.job < 0 || !last_of(job_done + c.job, jobs[c.job].chunks)) return;
  const XJob& J = jobs[c.job];
  s = x_add(J.part, 0, J.chunks, J.init, sh_add[w]);
  if (lane == 0) *J.out = s;
}

// The fixed tree: kTreeBlocks blocks per sum, the block that finishes last adds the partials (done: a
// counter per sum, back to zero for the next launch).
static __global__ void __launch_bounds__(kBlock) k_tree(const TreeSeg* segs, double* partials, unsigned* done,
                                                        const int* skip) {
  __shared__ double sh[32];
  __shared__ bool last;
  if (skip && *skip) return;
  const int s = blockIdx.x / kTreeBlocks, b = blockIdx.x % kTreeBlocks;
  const TreeSeg g = segs[s];
  const long long len = g.hi - g.lo;
  const long long a = g.lo + len * b / kTreeBlocks, e = g.lo + len * (b + 1) / kTreeBlocks;
  double acc = 0.0;
  for (long long i = a + threadIdx.x; i < e; i += blockDim.x) acc += g.t[i];
  acc = block_sum_fixed(acc, sh);
  double* part = partials + static_cast<long long>(s) * kTreeBlocks;
  if (threadIdx.x == 0) {
    part[b] = acc;
    __threadfence();
    last = atomicAdd(done + s, 1u) + 1u == static_cast<unsigned>(kTreeBlocks);
    if (last) done[s] = 0u;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  acc = 0.0;
  for (int i = threadIdx.x; i < kTreeBlocks; i += blockDim.x) acc += __ldcg(part + i);
  acc = block_sum_fixed(acc, sh);
  if (threadIdx.x == 0) *g.out = g.init + acc;
}

// A fixed set of sums over fixed term arrays. Built once (descriptors live on the device),
// launched any number of times, also inside stream capture.
class SumPlan {
 public:
  void add(const double* terms, long long lo, long long hi, double init, SumOrder order, double* out) {
    jobs_.push_back({terms, lo, hi, init, order, out});
  }
  // skip: optional device int; when non-zero at run time every kernel of the plan returns.
  // st: the stream the plan is launched on; the segment descriptors are copied to the device on
  // it, so they are in place before the plan's first launch on that stream.
  void build(bool exact, const int* skip, cudaStream_t st) {
    exact_ = exact;
    skip_ = skip;
    if (exact) {
      std::vector<XChain> chains;
      std::vector<XJob> jobs;
      ntiles_ = ngroups_ = 0;
      std::vector<int> block_chain, short_chain, span_chain;
      long long nchunk_jobs = 0;
      for (const Job& j : jobs_)
        if (j.order == SumOrder::kChunk64) ++nchunk_jobs;
      partials_.alloc(static_cast<std::size_t>(nchunk_jobs > 0 ? nchunk_jobs * kChunks : 1));
      auto chain = [&](const double* t, long long lo, long long hi, double init, double* out, int job) {
        XChain c{t, lo, hi, init, out, ntiles_, 0, ngroups_, 0,
                 static_cast<int>(block_chain.size()), -1, job};
        const int id = static_cast<int>(chains.size());
        if (hi - lo > kXShort) {
          c.ntiles = static_cast<int>((hi - lo + kXTile - 1) / kXTile);
          c.ngroups = (c.ntiles + kXGroup - 1) / kXGroup;
          ntiles_ += c.ntiles;
          ngroups_ += c.ngroups;
          block_chain.insert(block_chain.end(), static_cast<std::size_t>((c.ntiles + kXWarps - 1) / kXWarps), id);
          if (c.ntiles > kXSpanMin) {
            c.span0 = static_cast<int>(span_chain.size());
            span_chain.insert(span_chain.end(), static_cast<std::size_t>((c.ntiles + kXSpan - 1) / kXSpan), id);
          }
        } else {
          short_chain.push_back(id);
        }
        chains.push_back(c);
      };
      for (const Job& j : jobs_) {
        const long long n = j.hi - j.lo;
        if (j.order == SumOrder::kSeq) {
          chain(j.t, j.lo, j.hi, j.init, j.out, -1);
        } else {  // parallel_sum: the chunks' sums added in order
          const long long chunks = n < kChunks ? (n < 1 ? 1 : n) : kChunks;
          double* part = partials_.get() + static_cast<long long>(jobs.size()) * kChunks;
          for (long long c = 0; c < chunks; ++c)
            chain(j.t, j.lo + n * c / chunks, j.lo + n * (c + 1) / chunks, 0.0, part + c, static_cast<int>(jobs.size()));
          jobs.push_back({part, static_cast<int>(chunks), j.init, j.out});
        }
      }
      nblocks_ = static_cast<int>(block_chain.size());
      nshort_ = static_cast<int>(short_chain.size());
      nspans_ = static_cast<int>(span_chain.size());
      upload(chains, chains_, st);
      upload(jobs, xjobs_, st);
      upload(block_chain, block_chain_, st);
      upload(short_chain, short_chain_, st);
      if (nspans_ > 0) upload(span_chain, span_chain_, st), span_.alloc(span_chain.size());
      stat_.alloc(static_cast<std::size_t>(ntiles_ > 0 ? ntiles_ : 1));
      tile_fast_.alloc(static_cast<std::size_t>(ntiles_ > 0 ? ntiles_ : 1) * sizeof(XFast));
      group_fast_.alloc(static_cast<std::size_t>(ngroups_ > 0 ? ngroups_ : 1) * sizeof(XFast));
      tile_agg_.alloc(static_cast<std::size_t>(ntiles_ > 0 ? ntiles_ : 1) * sizeof(XTileAgg));
      group_agg_.alloc(static_cast<std::size_t>(ngroups_ > 0 ? ngroups_ : 1) * sizeof(XTileAgg));
      const std::size_t counters = static_cast<std::size_t>(ngroups_) + chains.size() + jobs.size();
      done_.alloc(counters + 1);
      B200_CHECK(cudaMemsetAsync(done_.get(), 0, (counters + 1) * sizeof(unsigned), st));
      nchains_ = static_cast<int>(chains.size());
    } else {
      std::vector<TreeSeg> tree;
      for (const Job& j : jobs_) tree.push_back({j.t, j.lo, j.hi, j.init, j.out});
      upload(tree, tseg_, st);
      nt_ = static_cast<int>(tree.size());
      partials_.alloc(static_cast<std::size_t>(nt_ > 0 ? nt_ : 1) * kTreeBlocks);
      done_.alloc(tree.size() + 1);
      B200_CHECK(cudaMemsetAsync(done_.get(), 0, (tree.size() + 1) * sizeof(unsigned), st));
    }
  }
  // The tile sums a producer may leave itself (x_leave_stat) before launch(st, true): of the plan's
  // only chain, starting at its first term. Null when the chain needs none.
  double* stat() { return exact_ && ntiles_ > 0 ? stat_.get() : nullptr; }
  // skippable: whether the plan's skip flag counts in this launch.
  void launch(cudaStream_t st, bool have_stat = false, bool skippable = true) const {
    const int* skip = skippable ? skip_ : nullptr;
    if (exact_) {
      const XChain* ch = reinterpret_cast<const XChain*>(chains_.get());
      if (ntiles_ > 0 && !have_stat) {
        k_xstat<<<nblocks_, 32 * kXWarps, 0, st>>>(ch, reinterpret_cast<const int*>(block_chain_.get()), stat_.get(), skip);
        B200_LAUNCH_CHECK();
      }
      if (nspans_ > 0) {
        k_xspan<<<nspans_, 256, 0, st>>>(ch, reinterpret_cast<const int*>(span_chain_.get()), stat_.get(), span_.get(), skip);
        B200_LAUNCH_CHECK();
      }
      const int blocks = nblocks_ + (nshort_ + kXWarps - 1) / kXWarps;
      if (blocks > 0) {
        // its descriptors load while the kernel that makes the terms ends (programmatic dependent launch)
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(static_cast<unsigned>(blocks));
        cfg.blockDim = dim3(32 * kXWarps);
        cfg.stream = st;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        unsigned* done = done_.get();
        B200_CHECK(cudaLaunchKernelEx(&cfg, k_xwalk, ch, reinterpret_cast<const XJob*>(xjobs_.get()),
                                      reinterpret_cast<const int*>(block_chain_.get()), nblocks_,
                                      reinterpret_cast<const int*>(short_chain_.get()), nshort_,
                                      static_cast<const double*>(stat_.get()), static_cast<const double*>(span_.get()),
                                      reinterpret_cast<XFast*>(tile_fast_.get()),
                                      reinterpret_cast<XTileAgg*>(tile_agg_.get()),
                                      reinterpret_cast<XFast*>(group_fast_.get()),
                                      reinterpret_cast<XTileAgg*>(group_agg_.get()), done, done + ngroups_,
                                      done + ngroups_ + nchains_, skip));
      }
    } else if (nt_ > 0) {
      k_tree<<<nt_ * kTreeBlocks, kBlock, 0, st>>>(reinterpret_cast<const TreeSeg*>(tseg_.get()), partials_.get(),
                                                   done_.get(), skip);
      B200_LAUNCH_CHECK();
    }
  }
  int kernel_count() const {
    return exact_ ? (ntiles_ > 0) + (nspans_ > 0) + (nblocks_ + nshort_ > 0) : (nt_ > 0 ? 1 : 0);
  }
  bool empty() const { return jobs_.empty(); }

 private:
  struct Job {
    const double* t;
    long long lo, hi;
    double init;
    SumOrder order;
    double* out;
  };
  // Stream-ordered copy from pageable memory: cudaMemcpyAsync stages the source before it
  // returns, and the device copy lands before any later work on `st`. (A plain cudaMemcpy on the
  // legacy stream may return before the copy lands and is not ordered with a non-blocking `st`.)
  template <class S>
  static void upload(const std::vector<S>& v, DevBuf<unsigned char>& dst, cudaStream_t st) {
    dst.alloc(v.size() * sizeof(S) + 1);
    if (!v.empty())
      B200_CHECK(cudaMemcpyAsync(dst.get(), v.data(), v.size() * sizeof(S), cudaMemcpyHostToDevice, st));
  }
  std::vector<Job> jobs_;
  bool exact_ = false;
  const int* skip_ = nullptr;
  DevBuf<unsigned char> chains_, xjobs_, tseg_, block_chain_, short_chain_, span_chain_;
  mutable DevBuf<unsigned char> tile_fast_, group_fast_, tile_agg_, group_agg_;
  mutable DevBuf<double> partials_, stat_, span_;
  mutable DevBuf<unsigned> done_;
  int nchains_ = 0, nshort_ = 0, nt_ = 0, ntiles_ = 0, nblocks_ = 0, ngroups_ = 0, nspans_ = 0;
};

}  // namespace b200
