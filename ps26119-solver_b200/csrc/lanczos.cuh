// lanczos.cuh — Lanczos steps on ÃᵀÃ (la::estimate_norm2, src/la/csr.cpp:86-132) as one cooperative kernel
// per batch of steps, for LPs that fit the SMs' shared memory: the matrix and the vectors stay there, the
// products' operands go through cells (resident.cuh), and α and β², sums over all columns in the
// reference's order, are evaluated as the chains of reduce.cuh are.
//
// A step: t = Ãv by the rows, w = Ãᵀt by the columns, α = Σ w·v, w −= αv + β_prev·v_prev, β² = Σ w²,
// v ← w/β. For a sum, every block's columns are a run of the chain (or several, of at most kXTile terms):
//   1  each block leaves its approximate sum in a cell and reads the earlier blocks' for the approximate
//      sum before its run, which tells the binade;
//   2  its warps summarise the runs (x_tile_agg) and the block counts itself in;
//   3  the block that is last walks all summaries in order with one warp (x_walk_lanes), and leaves the
//      exact sum in a cell that every block waits for.
// Everything is in the kernels' order and arithmetic, so α and β² are the same bits.
//
// A wait that runs out leaves the block with NaN and without its place among the runs: it goes on at place 0, and
// a walk may then meet summaries of other sums, or none. All of them (the arrays start at zero) name terms that
// exist, so every access stays inside its array and the kernel ends; the counter `err` makes the estimate an error.
//
// Why no cell is overwritten too early: v's and t's as in resident.cuh. A block writes its sums cell anew
// only after it has had the result of the sum before, which the last block to count in leaves, and a block
// counts in after it has read the earlier blocks' cells; the result's cell is written anew only once every
// block has counted in again, after it read the last one. The numbers of runs are read by blocks that the
// products tie to nothing (an LP whose columns fall into unconnected parts), at any time before they count
// in first: they have cells of their own, written once a launch, and the next launch follows this one.
//
// What bounds it: about ten trips through L2 a step (two half-steps, and four per sum) and the two walks, one
// x_commit for every binade that the sums pass. Measured, the whole estimate in ms, in six launches a step / so:
// 1k random rows 1.15 / 1.05, 10k 1.87 / 1.61, staircase T = 168 (389 steps) 12.6 / 10.1.
#pragma once

#include "reduce.cuh"
#include "resident.cuh"

namespace b200 {

struct LanczosArgs {
  int m, n, blocks;
  const int *t_rp, *t_ri, *a_rp, *a_col;
  const double *t_val, *a_val;
  Cell<double>*vcell, *tcell, *runs, *sums, *scalar;  // runs, sums: one per block
  double *v, *vprev, *terms, *hist;            // hist: (α, β²) by step
  XFast* fast;      // the runs' summaries, n / kXTile + blocks of them
  XTileAgg* full;
  unsigned* count;  // blocks that have counted in, over all sums
  unsigned tag;     // the first of 2 + 3·(to − from) tags
  // cells of an LP: n of v, m of t, two per block, the sums' result
  static long long cells(long long m, long long n, int blocks) { return n + m + 2LL * blocks + 1; }
  int from, to;
  int polls;  // reads of a cell before a wait for the sums gives up
  unsigned* err;
};
// What a block holds: three vectors and a term per column, nothing but the entries per row.
struct LanczosOp {
  static constexpr int kCol = 4, kRow = 0;
};

// Waits (one thread) until the cell has this tag.
__device__ __forceinline__ double cell_wait(const Cell<double>* c, unsigned tag, int limit, bool& dead) {
  CellRead<double> g{};
  for (int polls = 0; !dead; ++polls) {
    cell_load(g, c, true);
    if (g.is(tag)) return g.value();
    if (polls >= limit) dead = true;  // never expected
  }
  return __longlong_as_double(0x7ff8000000000000LL);
}

// Σ of all columns' terms in column order (see above); term[0, count) is this block's part, the chain's
// places [from, from + count). Every thread returns the sum; lane 0 of the walking warp leaves it in *out.
struct LanczosShared {
  double part[32], value;
  bool last;
  int tile0, tiles;  // this block's first run and the number of all blocks' runs
  alignas(16) double add[kXTile];
};
__device__ __forceinline__ double lanczos_sum(const LanczosArgs& p, LanczosShared& sh, const double* term, int from, int count,
                                              unsigned tag, double* out, bool& dead) {
  const int tid = static_cast<int>(threadIdx.x), lane = tid & 31, w = tid >> 5, warps = static_cast<int>(blockDim.x) >> 5;
  const int g = static_cast<int>(blockIdx.x);
  auto block_sum = [&](double s) {
    for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(kFull, s, off);
    __syncthreads();  // the last use of part is over
    if (lane == 0) sh.part[w] = s;
    __syncthreads();
    double t = 0.0;
    for (int k = 0; k < warps; ++k) t += sh.part[k];
    return t;
  };
  double s = 0.0;
  for (int e = tid; e < count; e += static_cast<int>(blockDim.x)) s += term[e], p.terms[from + e] = term[e];
  s = block_sum(s);
  if (tid == 0) cell_store(p.sums + g, s, tag);
  // the earlier blocks' sums: watch the nearest one, then read all of them
  if (g > 0 && w == 0) {
    if (lane == 0) cell_wait(p.sums + g - 1, tag, p.polls, dead);
    __syncwarp();
  }
  __syncthreads();
  s = 0.0;
  for (int k = tid; k < g; k += static_cast<int>(blockDim.x)) s += cell_wait(p.sums + k, tag, p.polls, dead);
  const double before = block_sum(s);
  const int tiles = (count + kXTile - 1) / kXTile;
  for (int q = w; q < tiles; q += warps) {
    const int a = q * kXTile, b = min(a + kXTile, count);
    double s0 = 0.0;
    for (int e = lane; e < a; e += 32) s0 += term[e];
    for (int off = 16; off > 0; off >>= 1) s0 += __shfl_xor_sync(kFull, s0, off);
    // the chain's first run starts at zero: its terms are added here, while the others are summarised
    XSummary T = sh.tile0 + q == 0 ? x_start(x_add(p.terms, from + a, from + b, 0.0, sh.add))
                                   : x_summary(x_tile_full(x_terms(term, a, b), before + s0));
    T.fast.first = from + a, T.fast.len = b - a;
    if (lane == 0) x_leave(T, p.fast + sh.tile0 + q, p.full + sh.tile0 + q);
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    sh.last = (atomicAdd(p.count, 1u) + 1u) % static_cast<unsigned>(p.blocks) == 0u;
  }
  __syncthreads();
  if (sh.last && w == 0) {
    __threadfence();
    const int all = sh.tiles;
    double r = 0.0;
    // the next round's summaries are on their way while one is walked
    auto round = [&](int k) { return x_round(p.fast + k + lane, p.full + k + lane, k + lane < all); };
    XRound R = round(0);
    for (int k0 = 0; k0 < all; k0 += 32) {
      const XRound N = round(k0 + 32);
      r = x_walk_lanes(r, R, min(32, all - k0), [&](int k, double st) {
        const int a = __shfl_sync(kFull, R.fast.first, k), len = __shfl_sync(kFull, R.fast.len, k);
        return x_add(p.terms, a, min(a + len, p.n), st, sh.add);
      });
      R = N;
    }
    if (lane == 0) {
      *out = r;
      cell_store(p.scalar, r, tag);
    }
  }
  if (tid == 0) sh.value = cell_wait(p.scalar, tag, p.polls, dead);
  __syncthreads();
  return sh.value;
}

template <int kThreads, int GB, bool kLong>
__global__ void __launch_bounds__(kThreads, 1) k_resident_lanczos(const __grid_constant__ LanczosArgs p) {
  using B = ResidentBytes<double, LanczosOp>;
  extern __shared__ __align__(16) unsigned char resident_smem[];
  __shared__ int cut[4];
  __shared__ LanczosShared sh;
  const int tid = static_cast<int>(threadIdx.x), lane = tid & 31, warp = tid >> 5, nt = static_cast<int>(blockDim.x),
            warps = nt >> 5, g = static_cast<int>(blockIdx.x);
  for (int q = warp; q < 4; q += warps) {  // columns [cut0, cut1), rows [cut2, cut3)
    const int r = q < 2 ? resident_cut(p.t_rp, p.n, B::kNz, B::kColumn, g + q, p.blocks)
                        : resident_cut(p.a_rp, p.m, B::kNz, B::kRowOf, g + q - 2, p.blocks);
    if (lane == 0) cut[q] = r;
  }
  __syncthreads();
  ResidentSide<double> C, R;
  resident_layout<kLong>(resident_smem, p.t_rp, cut[0], cut[1], LanczosOp::kCol, p.a_rp, cut[2], cut[3], LanczosOp::kRow, C, R);
  double *v = C.vec, *vprev = v + C.stride, *wv = vprev + C.stride, *term = wv + C.stride;
  bool dead = false;
  // every block's number of runs, for the places of its own
  if (tid == 0) cell_store(p.runs + g, static_cast<double>((C.count + kXTile - 1) / kXTile), p.tag);
  if (warp == 0) {
    double mine = 0.0, all = 0.0;
    for (int k = lane; k < p.blocks; k += 32) {
      const double t = cell_wait(p.runs + k, p.tag, p.polls, dead);
      all += t;
      if (k < g) mine += t;
    }
    for (int off = 16; off > 0; off >>= 1) {
      mine += __shfl_xor_sync(kFull, mine, off);
      all += __shfl_xor_sync(kFull, all, off);
    }
    dead = __any_sync(kFull, dead);
    if (dead) mine = all = 0.0;  // not NaN, which would become places outside the arrays
    if (lane == 0) sh.tile0 = static_cast<int>(mine), sh.tiles = static_cast<int>(all);
  }
  unsigned tag = p.tag + 1;
  for (int e = tid; e < C.count; e += nt) {  // v first, and out at once
    v[e] = p.v[C.from + e];
    cell_store(p.vcell + C.from + e, v[e], tag);
    vprev[e] = p.vprev[C.from + e];
  }
  resident_fill(C, p.t_rp, p.t_ri, p.t_val);
  resident_fill(R, p.a_rp, p.a_col, p.a_val);
  __syncthreads();
  double bsq = p.from > 0 ? p.hist[2 * p.from - 1] : 0.0;  // no β before the first step
  for (int k = p.from; k < p.to; ++k) {
    ResidentRow<GB, kLong, double> r;
    for (int e0 = 32 * warp; e0 < R.count; e0 += 32 * warps) {  // t = Ãv
      const int e = e0 + lane < R.count ? e0 + lane : -1;
      r.open(R, e);
      const double s = resident_sum(r, R, p.vcell, tag, e0 == 32 * warp, dead);
      if (e >= 0) cell_store(p.tcell + R.from + e, s, tag);
    }
    for (int e0 = 32 * warp; e0 < C.count; e0 += 32 * warps) {  // w = Ãᵀt
      const int e = e0 + lane < C.count ? e0 + lane : -1;
      r.open(C, e);
      const double s = resident_sum(r, C, p.tcell, tag, e0 == 32 * warp, dead);
      if (e >= 0) wv[e] = s, term[e] = s * v[e];
    }
    __syncthreads();
    const double al = lanczos_sum(p, sh, term, C.from, C.count, tag + 1, p.hist + 2 * k, dead), bp = sqrt(bsq);
    for (int e = tid; e < C.count; e += nt) {
      const double x = wv[e] - (al * v[e] + bp * vprev[e]);
      wv[e] = x;
      term[e] = x * x;
    }
    __syncthreads();
    bsq = lanczos_sum(p, sh, term, C.from, C.count, tag + 2, p.hist + 2 * k + 1, dead);
    const double bn = sqrt(bsq);
    tag += 3;
    for (int e = tid; e < C.count; e += nt) {
      vprev[e] = v[e];
      v[e] = wv[e] / bn;
      cell_store(p.vcell + C.from + e, v[e], tag);
    }
    __syncthreads();
  }
  for (int e = tid; e < C.count; e += nt) p.v[C.from + e] = v[e], p.vprev[C.from + e] = vprev[e];
  if (dead) count_stage_timeout(p.err);
}

// Past this many columns the walks over one run per 256 of them outweigh the launches saved (the kernels'
// form composes groups of 32). The estimate in one launch / by kernels, ms: staircase T = 360 (21,600 columns) 12.4 /
// 13.4, T = 680 (40,800) 13.9 / 14.1, 27k random rows (40,500) 1.94 / 1.91; past the line, in an earlier build, T = 720
// (43,200) 14.8 / 14.3, 30k rows (45,000) 2.34 / 2.24, 60k (90,000) 4.4 / 2.8.
constexpr long long kLanczosColumns = 40960;
// Columns a block: few blocks leave SMs to other solves, many make a longer walk and wider exchanges. The
// estimate with 112 / 224 / 448 / 896 columns a block, ms: 10k random rows 1.79 / 1.63 / 1.61 / 1.83, 27k 2.17 / 2.18 /
// 1.94 / 2.43, staircase T = 360 13.4 / 12.4 / 12.4 / 15.4, T = 680 16.3 / 16.2 / 13.9 / 17.8; 16 solves of 64 iterations side by
// side 38.5 / 34.7 / 33.4 / 29.4.
constexpr long long kLanczosShare = 448;
// The launch of such a kernel: as few blocks as hold the LP with about kLanczosShare columns each, because
// every block is a summary in the sums and a party to their three exchanges; blocks = 0: it does not fit.
struct LanczosShape {
  int blocks = 0, threads = 0;
  int longest = 0;
  unsigned smem = 0;
};
inline LanczosShape lanczos_shape(long long m, long long n, long long nnz, long long max_row, long long max_col, int sms) {
  using B = ResidentBytes<double, LanczosOp>;
  LanczosShape s;
  if (m < 1 || n < 1 || nnz < 1 || n > kLanczosColumns) return s;
  int blocks = static_cast<int>(std::max(1LL, std::min<long long>(sms, (n + kLanczosShare - 1) / kLanczosShare)));
  auto bytes = [&](int b) { return resident_bytes<double, LanczosOp>(m, n, nnz, max_row, max_col, b); };
  while (blocks < sms && bytes(blocks) > kResidentSmem / 2) ++blocks;
  const long long warps = std::max(n, m) / blocks / 32 + 2;
  const int threads = static_cast<int>(32 * std::min(32LL, std::max(2LL, warps)));
  const int longest = static_cast<int>(std::max(max_row, max_col));
  const long long smem = bytes(blocks) + resident_chunks(longest, threads);
  if (smem > static_cast<long long>(kResidentSmem - sizeof(LanczosShared)) || (m + n) / blocks > kResidentElements) return s;
  s.blocks = blocks;
  s.threads = threads;
  s.longest = longest;
  s.smem = static_cast<unsigned>(smem);
  return s;
}
// PS26119_LANCZOS_POLLS: another limit of those waits (read at every estimate; a test lets them run out).
inline int lanczos_polls() {
  const char* e = std::getenv("PS26119_LANCZOS_POLLS");
  return e && *e ? std::max(0, std::atoi(e)) : kResidentPolls;
}
// false: refused (launch_cooperative).
inline bool launch_lanczos(const LanczosArgs& p, const LanczosShape& s, cudaStream_t st) {
  const auto kernel = [&](auto is_long) {
    constexpr bool kLong = decltype(is_long)::value;
    return s.threads <= 256   ? reinterpret_cast<const void*>(&k_resident_lanczos<256, 16, kLong>)
           : s.threads <= 512 ? reinterpret_cast<const void*>(&k_resident_lanczos<512, 8, kLong>)
                              : reinterpret_cast<const void*>(&k_resident_lanczos<1024, 4, kLong>);
  };
  const void* f = resident_is_long(s.longest, s.threads) ? kernel(std::true_type{}) : kernel(std::false_type{});
  B200_CHECK(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kResidentSmem)));
  void* args[] = {const_cast<LanczosArgs*>(&p)};
  return launch_cooperative(f, s.blocks, s.threads, args, s.smem, st);
}

}  // namespace b200
