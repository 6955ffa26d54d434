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
//             to guess each tile's binade. A kernel that produces the terms may leave it itself.
//   k_xwalk   one warp per tile, kXWarps tiles per block: the guessed binade's u from the approximate
//             start (the approximate sums of the chain's earlier tiles), then the tile's XRun (exact
//             int64: change of S, its lowest and highest running value, parity after, per parity
//             before); a term with |t/u| ≥ 2^51 (or non-finite) marks the tile. A tile whose running sum
//             changes binade once is summarised in three parts: the run before the term that changes it,
//             that term, the run after it in the new grid. The block that finishes last of a group of
//             kXGroup tiles composes the tiles' summaries into the group's, of the same form. The block
//             that finishes last of a chain's walks the chain with the EXACT s, with one warp: a run of
//             groups is committed as s ← (S0 + K[S0 mod 2])·u as far as s = S0·u lies in their binade and
//             every running S provably stays within [2^52 + 1, 2^53 − 1] (then each exact partial sum
//             lies inside the binade, at least u/2 from its ends, and rounds to that grid); a group that
//             changes binade is committed by its three parts; any other one is walked by its tiles in the
//             same way; and the terms of a tile that cannot be committed are added one by one (x_add), so
//             that zeros, subnormals, infinities and NaN get exactly the sequential chain's arithmetic.
//             A chain of at most kXShort terms is added one by one from the start.
// The approximations only choose between two exact paths; the result never depends on them.
//
// What bounds it: latency. A dependent fp64 addition takes 8.3 cycles, 10.4 with its operand from
// shared memory, so a tile added one by one takes 1.4 us, and the walk of a chain pays that for its
// first tile (the sum starts at zero) and for the few tiles that cross a binade more than once; the
// other steps are one check over 32 summaries held by the warp's lanes, and a hand-over per crossing.
// Tiles of 256 terms, one warp's, keep the tiles that must be added one by one cheap. Measured, 15,000
// terms: 18.5 us a launch (24 with summaries read from shared memory and scanned anew at every crossing,
// 16 warps of a block on 32 tiles); three launches over tiles of 2,048 terms, the first tile walked in
// windows of 256 with a scan and a restart per binade crossing, took 68 us.
constexpr int kXPer = 8;              // terms per lane
constexpr int kXTile = 32 * kXPer;    // terms per tile (one warp)
constexpr int kXGroup = 32;           // tiles per group (one warp lane each)
constexpr int kXWarps = 8;            // warps per block of k_xwalk, tiles per block
constexpr long long kXShort = 1024;   // chains up to this long are added one by one by a warp

struct XChain {
  const double* t;
  long long lo, hi;  // terms t[lo, hi)
  double init;
  double* out;
  int tile0, ntiles;    // this chain's tiles in the tile arrays (ntiles = 0: added one by one)
  int group0, ngroups;  // its groups of kXGroup tiles
  int block0;           // its first block of kXWarps tiles
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
// odd (1) at the run's start: K the change of S, mn / mx the lowest / highest running change
// over positions 1…len (LLONG_MAX / LLONG_MIN for an empty run), out the parity after; bad: a
// term the integer form cannot take (|t/u| ≥ 2^51 or non-finite); ties: a term is a tie, so that the
// two parities may differ (without one they agree, and a run is plain integer sums).
struct alignas(16) XRun {
  long long K[2], mn[2], mx[2];
  int out[2];
  int bad, ties;
};
// A tile's summary: its terms before `split` counted in the grid u (the binade of the tile's
// approximate start), the term at `split` (where the approximate running sum leaves that binade;
// split = −1: it never does) added as a plain fp64 addition, the terms after it counted in the
// grid u1 of the binade the running sum moved to. u = 0: no usable guess (bad is set). A group's summary
// has the same form (its split is the tile that changes binade).
struct alignas(16) XTileAgg {
  double u, u1;
  double at;  // the term at `split`
  XRun pre, suf;
  int split;
};
constexpr long long kX52 = 1LL << 52, kX53 = 1LL << 53;

__device__ __forceinline__ XRun x_identity() {
  XRun r;
  r.K[0] = r.K[1] = 0;
  r.mn[0] = r.mn[1] = LLONG_MAX;
  r.mx[0] = r.mx[1] = LLONG_MIN;
  r.out[0] = 0, r.out[1] = 1;
  r.bad = r.ties = 0;
  return r;
}
// a then b (selects instead of indexing with a.out[p], so everything stays in registers)
__device__ __forceinline__ XRun x_compose(const XRun& a, const XRun& b) {
  XRun r;
  r.bad = a.bad | b.bad;
  r.ties = a.ties | b.ties;
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    const bool q = a.out[p] != 0;
    const long long bK = q ? b.K[1] : b.K[0], bmn = q ? b.mn[1] : b.mn[0], bmx = q ? b.mx[1] : b.mx[0];
    r.K[p] = a.K[p] + bK;
    r.mn[p] = bmn == LLONG_MAX ? a.mn[p] : min(a.mn[p], a.K[p] + bmn);
    r.mx[p] = bmx == LLONG_MIN ? a.mx[p] : max(a.mx[p], a.K[p] + bmx);
    r.out[p] = q ? b.out[1] : b.out[0];
  }
  return r;
}
__device__ __forceinline__ int x_pack(const XRun& v) { return v.out[0] | (v.out[1] << 1) | (v.bad << 2) | (v.ties << 3); }
__device__ __forceinline__ void x_unpack(XRun& r, int packed) {
  r.out[0] = packed & 1, r.out[1] = (packed >> 1) & 1, r.bad = (packed >> 2) & 1, r.ties = (packed >> 3) & 1;
}
__device__ __forceinline__ XRun x_shfl_down(const XRun& v, int off) {
  XRun r;
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    r.K[p] = __shfl_down_sync(kFull, v.K[p], off);
    r.mn[p] = __shfl_down_sync(kFull, v.mn[p], off);
    r.mx[p] = __shfl_down_sync(kFull, v.mx[p], off);
  }
  x_unpack(r, __shfl_down_sync(kFull, x_pack(v), off));
  return r;
}
__device__ __forceinline__ XRun x_shfl_up(const XRun& v, int off) {
  XRun r;
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    r.K[p] = __shfl_up_sync(kFull, v.K[p], off);
    r.mn[p] = __shfl_up_sync(kFull, v.mn[p], off);
    r.mx[p] = __shfl_up_sync(kFull, v.mx[p], off);
  }
  x_unpack(r, __shfl_up_sync(kFull, x_pack(v), off));
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
__device__ __forceinline__ double x_pow2(int p) {  // 2^p, p in [−1022, 1023]
  return __longlong_as_double(static_cast<long long>(p + 1023) << 52);
}
// A term in units of u (inv_u = 1/u, powers of two: t·inv_u is exact unless it under/overflows):
// false for |t/u| ≥ 2^51 or a non-finite t; else kf = rint(t/u), or floor(t/u) for a tie. Adding and
// taking away 1.5·2^52 rounds to an integer, and leaves it in the low bits of the sum.
__device__ __forceinline__ bool x_term(double t, double inv_u, long long& kf, bool& tie) {
  constexpr double kMagic = 6755399441055744.0;  // 1.5·2^52
  const double q = t * inv_u;
  if (!(fabs(q) < 2251799813685248.0)) return false;  // 2^51; also NaN / inf
  const double m = q + kMagic;
  kf = __double_as_longlong(m) - __double_as_longlong(kMagic);
  const double d = q - (m - kMagic);
  tie = fabs(d) == 0.5;
  if (d == -0.5) --kf;
  return true;
}
// The step of S with parity `par` for a term (kf, tie): returns k; par becomes S + k's parity.
__device__ __forceinline__ long long x_step(long long kf, bool tie, int& par) {
  long long k = kf;
  if (tie) {
    k += (par + kf) & 1;  // to the even neighbour
    par = 0;
  } else {
    par = static_cast<int>((par + k) & 1);
  }
  return k;
}
// The XRun of a warp's terms (lane l holds terms 8l … 8l+7; those whose bit q is set in `mask`, the
// others left out), valid in lane 0. Without a tie both parities make the same steps, and the run is
// integer sums: about a sixth of the general form's instructions.
__device__ __forceinline__ XRun x_warp_run(const double* v, unsigned mask, double inv_u) {
  const int lane = threadIdx.x & 31;
  XRun r = x_identity();
  long long kf[kXPer];
  bool tie[kXPer];
#pragma unroll
  for (int q = 0; q < kXPer; ++q) {
    kf[q] = 0, tie[q] = false;
    if ((mask >> q) & 1u) {
      if (!x_term(v[q], inv_u, kf[q], tie[q])) r.bad = 1, kf[q] = 0, tie[q] = false;
      r.ties |= tie[q] ? 1 : 0;
    }
  }
  if (__any_sync(kFull, r.ties)) {
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      int par = p;
      long long K = 0;
#pragma unroll
      for (int q = 0; q < kXPer; ++q)
        if ((mask >> q) & 1u) {
          K += x_step(kf[q], tie[q], par);
          r.mn[p] = min(r.mn[p], K);
          r.mx[p] = max(r.mx[p], K);
        }
      r.K[p] = K;
      r.out[p] = par;
    }
    for (int off = 1; off < 32; off <<= 1) {  // ordered reduction (lane order)
      const XRun o = x_shfl_down(r, off);
      if ((lane & (2 * off - 1)) == 0 && lane + off < 32) r = x_compose(r, o);
    }
    return r;
  }
  long long K = 0, mn = LLONG_MAX, mx = LLONG_MIN;
#pragma unroll
  for (int q = 0; q < kXPer; ++q)
    if ((mask >> q) & 1u) {
      K += kf[q];
      mn = min(mn, K);
      mx = max(mx, K);
    }
  long long inc = K;
  for (int off = 1; off < 32; off <<= 1) {
    const long long o = __shfl_up_sync(kFull, inc, off);
    if (lane >= off) inc += o;
  }
  if (mask) mn += inc - K, mx += inc - K;
  for (int off = 16; off > 0; off >>= 1) {
    mn = min(mn, __shfl_xor_sync(kFull, mn, off));
    mx = max(mx, __shfl_xor_sync(kFull, mx, off));
  }
  r.K[0] = r.K[1] = __shfl_sync(kFull, inc, 31);
  r.mn[0] = r.mn[1] = mn;
  r.mx[0] = r.mx[1] = mx;
  r.out[0] = static_cast<int>(r.K[0] & 1), r.out[1] = r.out[0] ^ 1;
  r.bad = __any_sync(kFull, r.bad) ? 1 : 0;
  return r;
}
// |S| inside [2^52 + 1, 2^53 − 1] with the sign of S0.
__device__ __forceinline__ bool x_inside(long long S0, long long S) {
  return S0 > 0 ? (S >= kX52 + 1 && S <= kX53 - 1) : (S <= -(kX52 + 1) && S >= -(kX53 - 1));
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

static __global__ void __launch_bounds__(256) k_xstat(const XChain* ch, const int* tile_chain, int ntiles,
                                                      double* stat, const int* skip) {
  if (skip && *skip) return;
  const int tile = static_cast<int>((blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (tile >= ntiles) return;
  const XChain& c = ch[tile_chain[tile]];
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

// The composition of the warp's runs in lane order, valid in lane 0.
__device__ __forceinline__ XRun x_warp_ordered(XRun r) {
  const int lane = threadIdx.x & 31;
  if (!__any_sync(kFull, r.ties)) {
    long long inc = r.K[0], mn = r.mn[0], mx = r.mx[0];
    for (int off = 1; off < 32; off <<= 1) {
      const long long o = __shfl_up_sync(kFull, inc, off);
      if (lane >= off) inc += o;
    }
    if (mn != LLONG_MAX) mn += inc - r.K[0], mx += inc - r.K[0];
    for (int off = 16; off > 0; off >>= 1) {
      mn = min(mn, __shfl_xor_sync(kFull, mn, off));
      mx = max(mx, __shfl_xor_sync(kFull, mx, off));
    }
    r.K[0] = r.K[1] = __shfl_sync(kFull, inc, 31);
    r.mn[0] = r.mn[1] = mn;
    r.mx[0] = r.mx[1] = mx;
    r.out[0] = static_cast<int>(r.K[0] & 1), r.out[1] = r.out[0] ^ 1;
    r.bad = __any_sync(kFull, r.bad) ? 1 : 0;
    return r;
  }
  for (int off = 1; off < 32; off <<= 1) {
    const XRun o = x_shfl_down(r, off);
    if ((lane & (2 * off - 1)) == 0 && lane + off < 32) r = x_compose(r, o);
  }
  return r;
}

// The summary of the terms t[a, b) (one tile, one warp; lane l holds terms 8l … 8l+7) for a chain
// whose approximate sum before them is s0; valid in lane 0.
__device__ __forceinline__ XTileAgg x_tile_agg(const double* __restrict__ t, long long a, long long b, double s0) {
  const int lane = threadIdx.x & 31;
  XTileAgg g;
  g.u = g.u1 = g.at = 0.0;
  g.split = -1;
  g.pre = g.suf = x_identity();
  int e0;
  if (!x_binade(s0, e0)) {  // uniform over the warp
    g.pre.bad = 1;
    return g;
  }
  const long long i0 = a + static_cast<long long>(lane) * kXPer;
  double v[kXPer];
  double run = 0.0;
#pragma unroll
  for (int q = 0; q < kXPer; ++q) v[q] = i0 + q < b ? t[i0 + q] : 0.0;
#pragma unroll
  for (int q = 0; q < kXPer; ++q) run += v[q];
  double inc = run;
  for (int off = 1; off < 32; off <<= 1) {
    const double o = __shfl_up_sync(kFull, inc, off);
    if (lane >= off) inc += o;
  }
  const double start = s0 + (inc - run);
  // the first position whose approximate running sum leaves e0's binade
  const int base = lane * kXPer;
  const int top0 = x_top(s0);
  int first = INT_MAX;
  double acc = start, at = 0.0, term = 0.0;
#pragma unroll
  for (int q = 0; q < kXPer; ++q)
    if (i0 + q < b) {
      acc += v[q];
      if (first == INT_MAX && x_top(acc) != top0) first = base + q, at = acc, term = v[q];
    }
  const int split = __reduce_min_sync(kFull, first);
  // the binade after the split: all later approximate running sums must share it
  int e1 = e0;
  bool ok1 = true;
  if (split != INT_MAX) {
    const double after = __shfl_sync(kFull, at, split / kXPer);
    ok1 = x_binade(after, e1);
    const int top1 = x_top(after);
    bool same = true;
    acc = start;
#pragma unroll
    for (int q = 0; q < kXPer; ++q)
      if (i0 + q < b) {
        acc += v[q];
        if (base + q > split && x_top(acc) != top1) same = false;
      }
    ok1 = __all_sync(kFull, same) && ok1;
  }
  unsigned mpre = 0, msuf = 0;
#pragma unroll
  for (int q = 0; q < kXPer; ++q)
    if (i0 + q < b) {
      if (base + q < split) mpre |= 1u << q;
      else if (split != INT_MAX && base + q > split) msuf |= 1u << q;
    }
  g.u = x_pow2(e0 - 52);
  g.pre = x_warp_run(v, mpre, x_pow2(52 - e0));
  if (split != INT_MAX) {
    g.split = split;
    g.at = __shfl_sync(kFull, term, split / kXPer);
    if (ok1) {
      g.u1 = x_pow2(e1 - 52);
      g.suf = x_warp_run(v, msuf, x_pow2(52 - e1));
    } else {
      g.suf.bad = 1;
    }
  }
  return g;
}

// Commits the run r (counted in the grid u) onto the exact s when s lies in u's binade and every
// running S stays inside it; returns false (s unchanged) otherwise.
__device__ __forceinline__ bool x_commit(double& s, double u, const XRun& r) {
  int e;
  if (r.bad || u == 0.0 || !x_binade(s, e) || x_pow2(e - 52) != u) return false;
  const long long S0 = static_cast<long long>(s * x_pow2(52 - e));
  const bool odd = (S0 & 1) != 0;
  if (r.mn[0] == LLONG_MAX) return true;  // an empty run
  const long long mn = odd ? r.mn[1] : r.mn[0], mx = odd ? r.mx[1] : r.mx[0];
  if (!x_inside(S0, S0 + mn) || !x_inside(S0, S0 + mx)) return false;
  s = static_cast<double>(S0 + (odd ? r.K[1] : r.K[0])) * u;
  return true;
}

// Commits a whole summary, its change of binade included; returns false (s unchanged) where it cannot.
__device__ __forceinline__ bool x_commit(double& s, const XTileAgg& T) {
  double s2 = s;
  if (!x_commit(s2, T.u, T.pre)) return false;
  if (T.split >= 0) {
    s2 += T.at;  // the term that changes the binade, as the chain adds it
    if (!x_commit(s2, T.u1, T.suf)) return false;
  }
  s = s2;
  return true;
}

// One warp walks cnt consecutive summaries, lane l holding T of the l-th, with the exact s. other(k, s)
// returns the sum after the k-th where its summary cannot be committed. Every step commits all summaries
// up to the first that changes binade, is not in s's binade, or whose running S would leave it. Without
// ties a run's K does not depend on what came before, so one prefix sum over the lanes serves all steps
// (across a change of grid the sum means nothing, but a step only uses differences within one).
template <class F>
__device__ __forceinline__ double x_walk_lanes(double s, const XTileAgg& T, int cnt, F&& other) {
  const int lane = threadIdx.x & 31;
  const bool here = lane < cnt;
  const bool plain = here && !T.pre.bad && T.split < 0 && T.u != 0.0;
  const unsigned ties = __ballot_sync(kFull, here && T.pre.ties);
  long long inc = here ? T.pre.K[0] : 0;
  for (int off = 1; off < 32; off <<= 1) {
    const long long o = __shfl_up_sync(kFull, inc, off);
    if (lane >= off) inc += o;
  }
  const long long before = inc - (here ? T.pre.K[0] : 0);
  int j = 0;
  while (j < cnt) {
    int e;
    const bool have = x_binade(s, e);
    const double u = have ? x_pow2(e - 52) : 0.0;
    const unsigned stop = __ballot_sync(kFull, lane >= j && !(plain && have && T.u == u));
    int f = stop ? __ffs(stop) - 1 : 32;  // the first that cannot be committed with those before it
    if (f > j) {
      const long long S0 = static_cast<long long>(s * x_pow2(52 - e));
      const bool in = lane >= j && lane < f;
      bool valid;
      long long K;  // the change of S up to and with this lane's run
      if ((ties & ((f < 32 ? (1u << f) : 0u) - (1u << j))) == 0) {
        const long long Kb = before - __shfl_sync(kFull, before, j);
        K = Kb + T.pre.K[0];
        valid = x_inside(S0, S0 + Kb + T.pre.mn[0]) && x_inside(S0, S0 + Kb + T.pre.mx[0]);
      } else {
        const int p0 = static_cast<int>(S0 & 1);
        XRun run = in ? T.pre : x_identity();
        for (int off = 1; off < 32; off <<= 1) {
          const XRun o = x_shfl_up(run, off);
          if (lane >= off) run = x_compose(o, run);
        }
        XRun ex = x_shfl_up(run, 1);
        if (lane == 0) ex = x_identity();
        const long long Kb = p0 ? ex.K[1] : ex.K[0];
        const bool pb = (p0 ? ex.out[1] : ex.out[0]) != 0;
        K = p0 ? run.K[1] : run.K[0];
        valid = x_inside(S0, S0 + Kb + (pb ? T.pre.mn[1] : T.pre.mn[0])) &&
                x_inside(S0, S0 + Kb + (pb ? T.pre.mx[1] : T.pre.mx[0]));
      }
      const unsigned bad = __ballot_sync(kFull, in && !valid);
      if (bad) f = __ffs(bad) - 1;
      if (f > j) s = static_cast<double>(S0 + __shfl_sync(kFull, K, f - 1)) * u;
    }
    if (f >= cnt) break;
    double s2 = s;
    const int done = lane == f && x_commit(s2, T) ? 1 : 0;
    s2 = __shfl_sync(kFull, s2, f);
    s = __shfl_sync(kFull, done, f) ? s2 : other(f, s);
    j = f + 1;
  }
  return s;
}
__device__ __forceinline__ XTileAgg x_no_summary() {
  XTileAgg T;
  T.u = T.u1 = T.at = 0.0;
  T.pre = T.suf = x_identity();
  T.split = -1;
  return T;
}

// The chain c from its tiles' and groups' summaries (one warp).
__device__ __forceinline__ double x_walk(const XChain& c, const XTileAgg* ag, const XTileAgg* gg, double* sh) {
  const int lane = threadIdx.x & 31;
  double s = c.init;
  for (int g0 = 0; g0 < c.ngroups; g0 += 32) {
    const int cntg = c.ngroups - g0 < 32 ? c.ngroups - g0 : 32;
    const XTileAgg G = lane < cntg ? x_load(gg + c.group0 + g0 + lane) : x_no_summary();
    s = x_walk_lanes(s, G, cntg, [&](int g, double sg) {
      const int t0 = (g0 + g) * kXGroup, cnt = c.ntiles - t0 < kXGroup ? c.ntiles - t0 : kXGroup;
      const XTileAgg T = lane < cnt ? x_load(ag + c.tile0 + t0 + lane) : x_no_summary();
      return x_walk_lanes(sg, T, cnt, [&](int k, double st) {
        long long a, b;
        x_tile_range(c, c.tile0 + t0 + k, a, b);
        return x_add(c.t, a, b, st, sh);
      });
    });
  }
  return s;
}

// The summary of a group of tiles, lane l holding T of the l-th (valid in lane 0): all tiles in one grid
// and none that changes binade, or one that does, with the tiles before it in its first grid and those
// after it in its second. Else u = 0.
__device__ __forceinline__ XTileAgg x_group(const XTileAgg& T, int cnt) {
  const int lane = threadIdx.x & 31;
  const bool here = lane < cnt;
  const unsigned splits = __ballot_sync(kFull, here && T.split >= 0);
  const int k = splits ? __ffs(splits) - 1 : 31;  // the last lane in the first grid
  XTileAgg G = x_no_summary();
  const double u0 = __shfl_sync(kFull, T.u, 0), u1 = splits ? __shfl_sync(kFull, T.u1, k) : u0;
  bool ok = !here || (!T.pre.bad && T.u != 0.0 && T.u == (lane <= k ? u0 : u1));
  if (lane == k && splits) ok = ok && !T.suf.bad && T.u1 != 0.0;
  if (!__all_sync(kFull, ok) || __popc(splits) > 1) {
    G.pre.bad = 1;
    return G;
  }
  G.u = u0;
  G.pre = x_warp_ordered(here && lane <= k ? T.pre : x_identity());
  if (splits) {
    G.u1 = u1, G.split = k;
    G.at = __shfl_sync(kFull, T.at, k);
    G.suf = x_warp_ordered(lane == k ? T.suf : (here && lane > k ? T.pre : x_identity()));
  }
  return G;
}

// Blocks [0, nblocks): kXWarps tiles of one chain each (block_chain: the chain). The blocks after them:
// one chain of at most kXShort terms per warp (short_chain). done: counters of a group's finished blocks,
// a chain's finished groups and a job's finished chains; the last one goes on, and sets its counter back to
// zero for the next launch.
static __global__ void __launch_bounds__(32 * kXWarps) k_xwalk(const XChain* __restrict__ ch, const XJob* __restrict__ jobs,
                                                               const int* __restrict__ block_chain, int nblocks,
                                                               const int* __restrict__ short_chain, int nshort,
                                                               const double* stat, XTileAgg* ag, XTileAgg* gg,
                                                               unsigned* group_done, unsigned* chain_done,
                                                               unsigned* job_done, const int* skip) {
  __shared__ alignas(16) double sh_add[kXWarps][kXTile];
  __shared__ double sh_sum[kXWarps];
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
    const double mine = lane < w && k0 + lane < c.ntiles ? stat[c.tile0 + k0 + lane] : 0.0;
    double pre = 0.0;  // the approximate sum before this block's tiles
    for (int q = threadIdx.x; q < k0; q += 32 * kXWarps) pre += stat[c.tile0 + q];
    for (int off = 16; off > 0; off >>= 1) pre += __shfl_xor_sync(kFull, pre, off);
    if (lane == 0) sh_sum[w] = pre;
    __syncthreads();
    double s0 = mine;
    for (int off = 16; off > 0; off >>= 1) s0 += __shfl_xor_sync(kFull, s0, off);
    s0 += c.init;
    for (int q = 0; q < kXWarps; ++q) s0 += sh_sum[q];
    if (k < c.ntiles) {
      long long a, b;
      x_tile_range(c, c.tile0 + k, a, b);
      const XTileAgg T = x_tile_agg(c.t, a, b, s0);
      if (lane == 0) ag[c.tile0 + k] = T;
    }
    __threadfence();
    __syncthreads();
    if (w != 0) return;
    const int g = k0 / kXGroup, t0 = g * kXGroup, cnt = c.ntiles - t0 < kXGroup ? c.ntiles - t0 : kXGroup;
    if (!last_of(group_done + c.group0 + g, (cnt + kXWarps - 1) / kXWarps)) return;
    const XTileAgg G = x_group(lane < cnt ? x_load(ag + c.tile0 + t0 + lane) : x_no_summary(), cnt);
    if (lane == 0) gg[c.group0 + g] = G;
    if (!last_of(chain_done + ci, c.ngroups)) return;
    s = x_walk(c, ag, gg, sh_add[0]);
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
      ngroups_ = 0;
      std::vector<int> tile_chain, block_chain, short_chain;
      long long nchunk_jobs = 0;
      for (const Job& j : jobs_)
        if (j.order == SumOrder::kChunk64) ++nchunk_jobs;
      partials_.alloc(static_cast<std::size_t>(nchunk_jobs > 0 ? nchunk_jobs * kChunks : 1));
      auto chain = [&](const double* t, long long lo, long long hi, double init, double* out, int job) {
        XChain c{t, lo, hi, init, out, static_cast<int>(tile_chain.size()), 0, ngroups_, 0,
                 static_cast<int>(block_chain.size()), job};
        const int id = static_cast<int>(chains.size());
        if (hi - lo > kXShort) {
          c.ntiles = static_cast<int>((hi - lo + kXTile - 1) / kXTile);
          c.ngroups = (c.ntiles + kXGroup - 1) / kXGroup;
          tile_chain.insert(tile_chain.end(), static_cast<std::size_t>(c.ntiles), id);
          ngroups_ += c.ngroups;
          block_chain.insert(block_chain.end(), static_cast<std::size_t>((c.ntiles + kXWarps - 1) / kXWarps), id);
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
      ntiles_ = static_cast<int>(tile_chain.size());
      nblocks_ = static_cast<int>(block_chain.size());
      nshort_ = static_cast<int>(short_chain.size());
      upload(chains, chains_, st);
      upload(jobs, xjobs_, st);
      upload(tile_chain, tile_chain_, st);
      upload(block_chain, block_chain_, st);
      upload(short_chain, short_chain_, st);
      stat_.alloc(static_cast<std::size_t>(ntiles_ > 0 ? ntiles_ : 1));
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
  void launch(cudaStream_t st, bool have_stat = false) const {
    if (exact_) {
      const XChain* ch = reinterpret_cast<const XChain*>(chains_.get());
      if (ntiles_ > 0 && !have_stat) {
        k_xstat<<<(ntiles_ + 7) / 8, 256, 0, st>>>(ch, reinterpret_cast<const int*>(tile_chain_.get()), ntiles_,
                                                   stat_.get(), skip_);
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
                                      static_cast<const double*>(stat_.get()), reinterpret_cast<XTileAgg*>(tile_agg_.get()),
                                      reinterpret_cast<XTileAgg*>(group_agg_.get()), done, done + ngroups_,
                                      done + ngroups_ + nchains_, skip_));
      }
    } else if (nt_ > 0) {
      k_tree<<<nt_ * kTreeBlocks, kBlock, 0, st>>>(reinterpret_cast<const TreeSeg*>(tseg_.get()), partials_.get(),
                                                   done_.get(), skip_);
      B200_LAUNCH_CHECK();
    }
  }
  int kernel_count() const {
    return exact_ ? (ntiles_ > 0) + (nblocks_ + nshort_ > 0) : (nt_ > 0 ? 1 : 0);
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
  DevBuf<unsigned char> chains_, xjobs_, tseg_, tile_chain_, block_chain_, short_chain_;
  mutable DevBuf<unsigned char> tile_agg_, group_agg_;
  mutable DevBuf<double> partials_, stat_;
  mutable DevBuf<unsigned> done_;
  int nchains_ = 0, nshort_ = 0, nt_ = 0, ntiles_ = 0, nblocks_ = 0, ngroups_ = 0;
};

}  // namespace b200
