// resident.cuh — the iterations of an epoch as ONE kernel, for LPs that fit the SMs' shared memory.
//
// Every block (one per SM, launched cooperatively, so that all run at the same time) keeps a range of
// Ã's columns and a range of its rows in shared memory for the whole epoch: their nonzeros and the
// vectors the updates read (x, x0, c, l, u; y, y0, rl, ru). A step then moves nothing but x̄ and y.
// These go through CELLS in global memory (L2): a value beside the number of the step that made it (its
// tag). A thread that needs an element reads its cell until the
// step number is the one it waits for; there is no barrier, and no other traffic between the blocks.
//
// Why no cell is overwritten too early: column j gathers the y of the rows in it, row i the x̄ of the
// columns in it, and Ã and Ãᵀ have the same pattern. Row i's next y is written after row i has read the x̄
// of all its columns, each made after that column read row i's y; so every reader of a y has had it when
// the next one is written, and likewise for x̄.
//
// Waits: all blocks are resident (cooperative launch), and a step's columns wait for rows of the step
// before, its rows for columns of the same step, so some thread can always go on. Every wait is bounded
// all the same: a thread that runs out of polls counts into the solve's error counter, goes on with NaN
// and waits no more, so the kernel ends and the host reports the solve.
//
// Arithmetic: a row's products are added in CSR order by one thread and the updates are the expressions
// of EpiPrimal / EpiDual / EpiPdlp* (spmv.cuh): the iterates are those of the kernels there, bit for bit.
//
// What bounds it: the round trip through L2 (a store is seen by another SM's poll after about 700
// cycles): a half-step takes a store, the poll that finds it, the gathers and the row's adds. What the two
// kernels per step pay beside that (launch, ramp, a round trip for the operands, the drain of the last
// block) is gone. Measured per iteration, fp64: 10k x 15k random LP 6.6 -> 3.0 us, 30k 10.8 -> 4.2, 100k
// 12.9 -> 9.8; staircase T = 168 6.4 -> 2.7.
#pragma once

#include "resident_rule.hpp"
#include "spmv.cuh"

namespace b200 {

// A cell is one or two 8-byte words, each 32 bits of the value beside the tag: a word is read and written
// whole (relaxed accesses at device scope), so no tag is ever seen without its bits.
template <class T>
struct alignas(2 * sizeof(T)) Cell {
  unsigned long long w[sizeof(T) / 4];
};
template <class T>
struct CellRead {
  unsigned long long w[sizeof(T) / 4];
  __device__ __forceinline__ bool is(unsigned tag) const {
    bool ok = true;
#pragma unroll
    for (unsigned k = 0; k < sizeof(T) / 4; ++k) ok = ok && static_cast<unsigned>(w[k] >> 32) == tag;
    return ok;
  }
  __device__ __forceinline__ T value() const {
    if constexpr (sizeof(T) == 8)
      return __hiloint2double(static_cast<int>(static_cast<unsigned>(w[1])), static_cast<int>(static_cast<unsigned>(w[0])));
    else
      return __uint_as_float(static_cast<unsigned>(w[0]));
  }
};
// Reads the cell where `want` holds: a predicated load, so that the loads of a row issue back to back (as
// branches around the loads, a step of a 10k LP took 4.4 us instead of 3.2).
template <class T>
__device__ __forceinline__ void cell_load(CellRead<T>& r, const Cell<T>* p, bool want) {
  if constexpr (sizeof(T) == 8)
    asm volatile("{\n .reg .pred q;\n setp.ne.s32 q, %3, 0;\n @q ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];\n}"
                 : "+l"(r.w[0]), "+l"(r.w[1])
                 : "l"(p), "r"(static_cast<int>(want)));
  else
    asm volatile("{\n .reg .pred q;\n setp.ne.s32 q, %2, 0;\n @q ld.relaxed.gpu.global.b64 %0, [%1];\n}"
                 : "+l"(r.w[0])
                 : "l"(p), "r"(static_cast<int>(want)));
}
template <class T>
__device__ __forceinline__ void cell_store(Cell<T>* p, T v, unsigned tag) {
  const unsigned long long t = static_cast<unsigned long long>(tag) << 32;
  if constexpr (sizeof(T) == 8)
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(t | static_cast<unsigned>(__double2loint(v))),
                 "l"(t | static_cast<unsigned>(__double2hiint(v)))
                 : "memory");
  else
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(t | __float_as_uint(v)) : "memory");
}

// The lines of the rule, and what lies on both sides (fp64 / mixed, us per iteration, resident against the
// step kernels): random LPs of 10k rows 3.0 / 3.1 against 6.6 / 6.7, 30k 4.2 / 3.9 against 10.8 / 11.3,
// 100k 9.8 / 9.0 against 12.9 / 14.1. Past 194 KB a block the next carveout leaves the gathers too little
// L1: 112k rows (186 KB) 12.0 against 12.7, 121k (201 KB) 20.9 against 12.7. Past 2,560 columns and rows a
// block the polls crowd out the stores: mixed 150k rows (2,534) 13.6 against 14.1, 180k (3,040) 18.0
// against 16.9; the staircase T = 3600 (2,651) 6.7 against 9.1. LPs with long rows: resident_rule.hpp.
constexpr unsigned kResidentSmem = 194u * 1024u;
constexpr long long kResidentElements = 2688;

constexpr int kResidentPolls = 1 << 20;  // reads of one cell before a wait gives up (about half a second)

// r²HPDHG's updates (EpiPrimal / EpiDual). The vectors named by col_vec / row_vec are held in shared
// memory, vector k at v[k·stride].
template <class T>
struct ResidentR2h {
  T *x, *xh, *xb, *y, *yh, *yb;
  const T *x0, *c, *l, *u, *y0, *rl, *ru;
  T *xh0, *xb0, *yh0, *yb0;  // the points after the first step of a Halpern cycle (for its r⁰)
  double tau, sigma, rho;
  long long inner0;
  int K;
  static constexpr int kCol = 5, kRow = 4;
  __device__ const T* col_vec(int k) const { return k == 0 ? x : k == 1 ? x0 : k == 2 ? c : k == 3 ? l : u; }
  __device__ const T* row_vec(int k) const { return k == 0 ? y : k == 1 ? y0 : k == 2 ? rl : ru; }
  struct Step {
    T w, a, b;
    bool first, last;
  };
  __device__ Step step(int s) const {
    const long long k = inner0 + s;
    return {static_cast<T>(static_cast<double>(k + 1) / static_cast<double>(k + 2)), static_cast<T>(2 * rho),
            static_cast<T>(1 - 2 * rho), k == 0, s == K - 1};
  }
  // An update's operands and what can be done before its product is known; then the value the other side
  // gathers; then, once that is out, the rest.
  struct Col {
    T x, x0, c, l, u, h;
  };
  struct Row {
    T y, y0, rl, ru, q, h;
  };
  __device__ Col col_before(const T* v, int n) const { return {v[0], v[n], v[2 * n], v[3 * n], v[4 * n], T(0)}; }
  __device__ Row row_before(const T* v, int n) const {
    return {v[0], v[n], v[2 * n], v[3 * n], v[0] / static_cast<T>(sigma), T(0)};
  }
  __device__ T col(const Step&, double s, Col& o) const {
    const T aty = static_cast<T>(s);
    o.h = ref_clamp<T>(o.x - static_cast<T>(tau) * (o.c - aty), o.l, o.u);
    return static_cast<T>(static_cast<T>(2) * o.h - o.x);
  }
  __device__ void col_after(const Step& st, int j, const Col& o, T xbar, T* v, int) const {
    const T nx = st.w * (st.a * o.h + st.b * o.x) + (static_cast<T>(1) - st.w) * o.x0;
    v[0] = nx;
    if (st.first) xh0[j] = o.h, xb0[j] = xbar;
    if (st.last) xh[j] = o.h, xb[j] = xbar, x[j] = nx;
  }
  __device__ T row(const Step& st, double s, Row& o) const {
    const T ax = static_cast<T>(s), sg = static_cast<T>(sigma);
    const T d = ax - o.q;
    o.h = o.y - sg * ax + sg * ref_clamp<T>(d, o.rl, o.ru);
    return static_cast<T>(st.w * (st.a * o.h + st.b * o.y) + (static_cast<T>(1) - st.w) * o.y0);
  }
  __device__ void row_after(const Step& st, int i, const Row& o, T ny, T* v, int) const {
    v[0] = ny;
    if (st.first) yh0[i] = o.h, yb0[i] = static_cast<T>(2) * o.h - o.y;
    if (st.last) yh[i] = o.h, yb[i] = static_cast<T>(2) * o.h - o.y, y[i] = ny;
  }
};

// PDLP's steps and running averages (EpiPdlpPrimal / EpiPdlpDual): x, y in, x⁺, y⁺ out, with the point
// before the last step left in x_prev, y_prev.
template <class T>
struct ResidentPdlp {
  const T *x, *c, *l, *u, *y, *rl, *ru;
  T *xa, *ya, *x_out, *x_prev, *xb, *y_out, *y_prev;
  double tau, sigma;
  long long inner0;
  int K;
  static constexpr int kCol = 5, kRow = 4;
  __device__ const T* col_vec(int k) const { return k == 0 ? x : k == 1 ? xa : k == 2 ? c : k == 3 ? l : u; }
  __device__ const T* row_vec(int k) const { return k == 0 ? y : k == 1 ? ya : k == 2 ? rl : ru; }
  struct Step {
    T wa, wb;
    bool last;
  };
  __device__ Step step(int s) const {
    const double wa = 1.0 / static_cast<double>(inner0 + s + 1);
    return {static_cast<T>(wa), static_cast<T>(1.0 - wa), s == K - 1};
  }
  struct Col {
    T x, xa, c, l, u, h;
  };
  struct Row {
    T y, ya, rl, ru, q, h;
  };
  __device__ Col col_before(const T* v, int n) const { return {v[0], v[n], v[2 * n], v[3 * n], v[4 * n], T(0)}; }
  __device__ Row row_before(const T* v, int n) const {
    return {v[0], v[n], v[2 * n], v[3 * n], v[0] / static_cast<T>(sigma), T(0)};
  }
  __device__ T col(const Step&, double s, Col& o) const {
    const T aty = static_cast<T>(s);
    o.h = ref_clamp<T>(o.x - static_cast<T>(tau) * (o.c - aty), o.l, o.u);
    return static_cast<T>(static_cast<T>(-1.0) * o.x + static_cast<T>(2.0) * o.h);
  }
  __device__ void col_after(const Step& st, int j, const Col& o, T xbar, T* v, int n) const {
    const T avg = st.wa * o.h + st.wb * o.xa;
    if (st.last) x_prev[j] = o.x, x_out[j] = o.h, xb[j] = xbar, xa[j] = avg;
    v[0] = o.h;
    v[n] = avg;
  }
  __device__ T row(const Step&, double s, Row& o) const {
    const T ax = static_cast<T>(s), sg = static_cast<T>(sigma);
    const T d = ax - o.q;
    o.h = o.y - sg * ax + sg * ref_clamp<T>(d, o.rl, o.ru);
    return o.h;
  }
  __device__ void row_after(const Step& st, int i, const Row& o, T, T* v, int n) const {
    const T avg = st.wa * o.h + st.wb * o.ya;
    if (st.last) y_prev[i] = o.y, y_out[i] = o.h, ya[i] = avg;
    v[0] = o.h;
    v[n] = avg;
  }
};

// One LP of a launch: its matrix, cells and updates, and the blocks [first, first + blocks) that hold it.
template <class T, class Op>
struct ResidentPart {
  int m, n, first, blocks;
  const int *t_rp, *t_ri, *a_rp, *a_col;
  const T *t_val, *a_val;
  Cell<T>*xcell, *ycell;
  unsigned tag;  // y's at the start; step s makes x̄ with tag + s + 1 and y with tag + s + 1
  unsigned* err;
  Op op;
};

// Shared-memory bytes of one column or row and of one of its nonzeros: the measure by which the columns
// and the rows are dealt out to the blocks.
template <class T, class Op>
struct ResidentBytes {
  static constexpr long long kNz = 4 + sizeof(T), kColumn = 4 + Op::kCol * sizeof(T), kRowOf = 4 + Op::kRow * sizeof(T);
};
// Upper bound of a block's shared memory when `blocks` blocks share an LP: an even share of each side's
// bytes, one more column and row of the largest sizes, and the arrays' ends and alignment.
template <class T, class Op>
inline long long resident_bytes(long long m, long long n, long long nnz, long long max_row, long long max_col, int blocks) {
  using B = ResidentBytes<T, Op>;
  const long long cols = nnz * B::kNz + n * B::kColumn, rows = nnz * B::kNz + m * B::kRowOf;
  return cols / blocks + rows / blocks + max_col * B::kNz + B::kColumn + max_row * B::kNz + B::kRowOf + 256;
}

// The first row r of [0, rows] whose bytes before it, rp[r]·kNz + r·per, reach share g of `of` (one warp:
// 32 probes a round).
__device__ __forceinline__ int resident_cut(const int* __restrict__ rp, int rows, long long nz, long long per, int g, int of) {
  const int lane = threadIdx.x & 31;
  const long long total = static_cast<long long>(__ldg(rp + rows)) * nz + rows * per;
  const long long want = total / of * g + total % of * g / of;
  int lo = 0, hi = rows;
  while (lo < hi) {
    const int at = lo + static_cast<int>(static_cast<long long>(hi - lo) * lane / 32);
    const unsigned reached = __ballot_sync(kFull, static_cast<long long>(__ldg(rp + at)) * nz + at * per >= want);
    if (reached == 0) {
      lo = __shfl_sync(kFull, at, 31) + 1;
      continue;
    }
    const int f = __ffs(reached) - 1;
    hi = __shfl_sync(kFull, at, f);
    if (f > 0) lo = __shfl_sync(kFull, at, f - 1) + 1;
  }
  return hi;
}

constexpr int kResidentChunk = 64;  // entries of a long row gathered at a time

// One side of a block's part in shared memory.
template <class T>
struct ResidentSide {
  int from, count, stride;
  int *rp, *idx;  // rp rebased to the block's first nonzero
  T *val, *vec;
  double* chunk;  // the warps' buffers for long rows
};

// Both sides' places in a block's shared memory: columns [c0, c1) of a matrix with row pointers t_rp (of
// Ãᵀ), rows [r0, r1) of one with a_rp.
template <bool kLong, class T>
__device__ __forceinline__ void resident_layout(unsigned char* at, const int* t_rp, int c0, int c1, int col_vecs,
                                                const int* a_rp, int r0, int r1, int row_vecs, ResidentSide<T>& C,
                                                ResidentSide<T>& R) {
  auto take = [&](long long bytes) {
    unsigned char* r = at;
    at += (bytes + 7) & ~7LL;
    return r;
  };
  auto side = [&](ResidentSide<T>& S, const int* rp, int from, int to, int vecs) {
    S.from = from, S.count = to - from, S.stride = S.count;
    const int nz = __ldg(rp + to) - __ldg(rp + from);
    S.val = reinterpret_cast<T*>(take(static_cast<long long>(nz) * sizeof(T)));
    S.vec = reinterpret_cast<T*>(take(static_cast<long long>(vecs) * S.count * sizeof(T)));
    S.rp = reinterpret_cast<int*>(take((S.count + 1LL) * 4));
    S.idx = reinterpret_cast<int*>(take(nz * 4LL));
  };
  C.chunk = R.chunk = reinterpret_cast<double*>(take(kLong ? static_cast<long long>(blockDim.x) / 32 * kResidentChunk * 8 : 0));
  side(C, t_rp, c0, c1, col_vecs);
  side(R, a_rp, r0, r1, row_vecs);
}
// Brings a side's row pointers (rebased), indices and values in.
template <class T>
__device__ __forceinline__ void resident_fill(const ResidentSide<T>& S, const int* rp, const int* idx, const T* val) {
  const int tid = static_cast<int>(threadIdx.x), nt = static_cast<int>(blockDim.x);
  const int k0 = __ldg(rp + S.from), nz = __ldg(rp + S.from + S.count) - k0;
  for (int k = tid; k <= S.count; k += nt) S.rp[k] = __ldg(rp + S.from + k) - k0;
  for (int k = tid; k < nz; k += nt) S.idx[k] = __ldg(idx + k0 + k), S.val[k] = __ldg(val + k0 + k);
}

// A long row (resident_rule.hpp) walked by one thread would take a trip to L2 for every GB entries while the whole
// LP waits for it. Launches with one run kernels in which a warp sums such rows together (resident_long).
template <int GB>
constexpr int kResidentLong = resident_long_row(GB > 8 ? 0 : GB > 4 ? 1 : 2);
inline bool resident_is_long(int longest, int threads) { return longest > resident_long_row(resident_form(threads)); }
// Their shared memory beside the LP's part: a buffer for a chunk's products per warp.
inline long long resident_chunks(int longest, int threads) {
  return resident_is_long(longest, threads) ? threads / 32 * kResidentChunk * 8LL : 0;
}

// A thread's row: its entries [a, a + len) of the side's arrays, and the first GB of them. (With GB = 4,
// at 64 registers a thread, the values stay in shared memory until they are used.)
template <int GB, bool kLong, class T>
struct ResidentRow {
  static constexpr bool kVals = GB > 4;
  int a, len, longest;  // longest: of the warp's rows that have a thread each
  unsigned together;    // the lanes whose rows the warp sums together (kLong kernels)
  int idx[GB];
  T val[kVals ? GB : 1];
  // e < 0: the lane has no element (a row without entries)
  __device__ __forceinline__ void open(const ResidentSide<T>& S, int e) {
    a = e >= 0 ? S.rp[e] : 0, len = e >= 0 ? S.rp[e + 1] - a : 0;
    longest = __reduce_max_sync(kFull, len);
    together = 0;
    if (kLong && longest > kResidentLong<GB>) {
      const bool is = len > kResidentLong<GB>;
      if (__reduce_add_sync(kFull, is ? len : 0) < kResidentShare * longest) {
        together = __ballot_sync(kFull, is);
        longest = __reduce_max_sync(kFull, is ? 0 : len);
      }
    }
    load(S, 0);
  }
  __device__ __forceinline__ void load(const ResidentSide<T>& S, int k) {
#pragma unroll
    for (int q = 0; q < GB; ++q) {
      const int at = k + q < len ? a + k + q : 0;
      idx[q] = S.idx[at];
      if constexpr (kVals) val[q] = S.val[at];
    }
  }
  __device__ __forceinline__ double value(const ResidentSide<T>& S, int k, int q) const {
    if constexpr (kVals) return static_cast<double>(val[q]);
    else return static_cast<double>(S.val[k + q < len ? a + k + q : 0]);
  }
};

// The Σ of a long row, entries [0, n) at idx and val, by a whole warp: its lanes gather kResidentChunk entries at
// a time, the next ones while these are added, and every lane adds their products in CSR order from the warp's
// buffer `sh` (16-byte aligned). What bounds it: the chain of additions, 13 cycles each by itself (21 with shuffles in
// place of the buffer), 16 in blocks of 256 threads and 27 in those of 1,024, whose other warps poll beside it;
// chunks of 128, or two ahead, were no faster. Measured, us per iteration with one thread a long row / so / the
// step kernels' best variant: 10k rows and one of 512 26.6 / 7.4 / 9.9, of 4,096 190 / 36.9 / 29.7; 60k rows and
// one of 512 52.7 / 13.1 / 13.7, of 4,096 406 / 63.8 / 33.9.
struct ResidentLongSum {
  double s;
  bool dead;  // a lane's wait ran out
};
template <class T>
__device__ __noinline__ ResidentLongSum resident_long(const int* idx, const T* val, int n, const Cell<T>* cells, unsigned tag,
                                                      bool dead, double* sh) {
  constexpr int Q = kResidentChunk / 32;
  const int lane = static_cast<int>(threadIdx.x) & 31;
  CellRead<T> g[Q];
  const auto ask = [&](int k, bool again) {
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int e = k + 32 * q + lane;
      const bool in = e < n;
      if (!again) g[q] = CellRead<T>{};
      cell_load(g[q], cells + idx[in ? e : 0], in && !(again && g[q].is(tag)));
    }
  };
  double s = 0.0;
  ask(0, false);
  for (int k = 0; k < n; k += kResidentChunk) {
    for (int polls = 0;; ++polls) {
      bool late = false;
#pragma unroll
      for (int q = 0; q < Q; ++q) late = late || (k + 32 * q + lane < n && !g[q].is(tag));
      if (!__any_sync(kFull, late && !dead)) break;
      if (polls > kResidentPolls) dead = true;  // never expected
      ask(k, true);
    }
    __syncwarp();  // the chunk before has been added
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int e = k + 32 * q + lane;
      const double prod = static_cast<double>(val[e < n ? e : 0]) * static_cast<double>(g[q].value());
      sh[32 * q + lane] = e < n ? prod : -0.0;  // adding −0.0 leaves every sum as it is
    }
    __syncwarp();
    if (k + kResidentChunk < n) ask(k + kResidentChunk, false);
    const double2* p = reinterpret_cast<const double2*>(sh);
    double2 v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = p[q];
#pragma unroll
    for (int i = 0; i < kResidentChunk; i += 8) {  // 8 products ahead in registers (wrapping at the buffer's end)
      double2 w[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) w[q] = p[((i >> 1) + 4 + q) & (kResidentChunk / 2 - 1)];
#pragma unroll
      for (int q = 0; q < 4; ++q) s += v[q].x, s += v[q].y;
#pragma unroll
      for (int q = 0; q < 4; ++q) v[q] = w[q];
    }
  }
  return {s, __any_sync(kFull, dead) != 0};
}

// The row's Σ in CSR order, from cells of tag `tag`. `watch`: the warp's first element of this half-step.
// One lane then watches one cell until it is there before the warp gathers: polls of every gathered cell
// by every thread slow the stores that they wait for (a step of a 10k LP took 16.3 us that way, 4.4 with the
// watch). Cells that are late all the same are read again, by the whole warp in step. The warp's long rows come
// after the others.
template <int GB, bool kLong, class T>
__device__ __forceinline__ double resident_sum(ResidentRow<GB, kLong, T>& r, const ResidentSide<T>& S, const Cell<T>* cells,
                                               unsigned tag, bool watch, bool& dead) {
  if (watch && r.longest > 0) {
    const int who = __ffs(__ballot_sync(kFull, r.len > 0) & (kLong ? ~r.together : kFull)) - 1;
    if (static_cast<int>(threadIdx.x & 31) == who) {
      const Cell<T>* c = cells + r.idx[0];
      CellRead<T> g{};
      for (int polls = 0; !dead; ++polls) {
        cell_load(g, c, true);
        if (g.is(tag)) break;
        if (polls > kResidentPolls) dead = true;  // never expected
      }
    }
    __syncwarp();
  }
  double s = 0.0;
  const int lane = static_cast<int>(threadIdx.x) & 31, len = kLong && ((r.together >> lane) & 1u) ? 0 : r.len;
  for (int k = 0;;) {
    CellRead<T> g[GB];
    bool late[GB];
#pragma unroll
    for (int q = 0; q < GB; ++q) {
      late[q] = k + q < len;
      g[q] = CellRead<T>{};
      cell_load(g[q], cells + r.idx[q], late[q]);
    }
    for (int polls = 0;; ++polls) {
      bool any = false;
#pragma unroll
      for (int q = 0; q < GB; ++q) {
        late[q] = late[q] && !g[q].is(tag);
        any = any || late[q];
      }
      if (!__any_sync(kFull, any && !dead)) break;
      if (polls > kResidentPolls) dead = true;  // never expected
#pragma unroll
      for (int q = 0; q < GB; ++q) cell_load(g[q], cells + r.idx[q], late[q]);
    }
#pragma unroll
    for (int q = 0; q < GB; ++q) {  // in CSR order; adding −0.0 leaves every sum as it is
      const double prod = r.value(S, k, q) * static_cast<double>(g[q].value());
      s += k + q < len ? prod : -0.0;
    }
    k += GB;
    if (k >= r.longest) break;
    r.load(S, k);
  }
  if constexpr (kLong)
    for (unsigned left = r.together; left != 0; left &= left - 1) {
      const int who = __ffs(left) - 1, from = __shfl_sync(kFull, r.a, who);
      const ResidentLongSum t = resident_long(S.idx + from, S.val + from, __shfl_sync(kFull, r.len, who), cells, tag, dead,
                                              S.chunk + (threadIdx.x >> 5) * kResidentChunk);
      if (lane == who) s = t.s;
      dead = t.dead;
    }
  return dead ? __longlong_as_double(0x7ff8000000000000LL) : s;
}

template <int GB, bool kLong, class T, class Op>
__device__ __forceinline__ void resident_body(const ResidentPart<T, Op>& p, int g) {
  using B = ResidentBytes<T, Op>;
  extern __shared__ __align__(16) unsigned char resident_smem[];
  __shared__ int cut[4];
  const int tid = static_cast<int>(threadIdx.x), lane = tid & 31, warp = tid >> 5, warps = static_cast<int>(blockDim.x) >> 5;
  for (int q = warp; q < 4; q += warps) {  // columns [cut0, cut1), rows [cut2, cut3)
    const int r = q < 2 ? resident_cut(p.t_rp, p.n, B::kNz, B::kColumn, g + q, p.blocks)
                        : resident_cut(p.a_rp, p.m, B::kNz, B::kRowOf, g + q - 2, p.blocks);
    if (lane == 0) cut[q] = r;
  }
  __syncthreads();
  ResidentSide<T> C, R;
  resident_layout<kLong>(resident_smem, p.t_rp, cut[0], cut[1], Op::kCol, p.a_rp, cut[2], cut[3], Op::kRow, C, R);
  const int nt = static_cast<int>(blockDim.x);
  // y first, and out at once: the columns' first step waits for it
  for (int e = tid; e < R.count; e += nt) {
    const T v = p.op.row_vec(0)[R.from + e];
    R.vec[e] = v;
    cell_store(p.ycell + R.from + e, v, p.tag);
  }
  resident_fill(C, p.t_rp, p.t_ri, p.t_val);
  resident_fill(R, p.a_rp, p.a_col, p.a_val);
  for (int k = 0; k < Op::kCol; ++k)
    for (int e = tid; e < C.count; e += nt) C.vec[k * C.stride + e] = p.op.col_vec(k)[C.from + e];
  for (int k = 1; k < Op::kRow; ++k)
    for (int e = tid; e < R.count; e += nt) R.vec[k * R.stride + e] = p.op.row_vec(k)[R.from + e];
  __syncthreads();
  // the warps are shared out between columns and rows: one element a thread where there are enough
  const int wc_need = (C.count + 31) / 32, wr_need = (R.count + 31) / 32;
  int wc = wc_need;
  if (wc_need + wr_need > warps) wc = (warps * wc_need + (wc_need + wr_need) / 2) / (wc_need + wr_need);
  wc = max(1, min(wc, warps - 1));
  bool dead = false;
  const int K = p.op.K;
  // (the loops are the warp's: lanes without an element keep step. A warp with one element a thread and
  // rows of at most GB entries opens its rows once.)
  if (warp < wc) {
    const bool once = C.count <= 32 * wc;
    ResidentRow<GB, kLong, T> r;
    if (once) r.open(C, 32 * warp + lane < C.count ? 32 * warp + lane : -1);
    const bool held = once && r.longest <= GB;
    for (int s = 0; s < K; ++s) {
      const auto st = p.op.step(s);
      const unsigned tag = p.tag + static_cast<unsigned>(s);
      for (int e0 = 32 * warp; e0 < C.count; e0 += 32 * wc) {
        const int e = e0 + lane < C.count ? e0 + lane : -1;
        if (!held) r.open(C, e);
        T* v = C.vec + (e >= 0 ? e : 0);
        auto o = p.op.col_before(v, C.stride);
        const double sum = resident_sum(r, C, p.ycell, tag, e0 == 32 * warp, dead);
        if (e < 0) continue;
        const T xbar = p.op.col(st, sum, o);
        cell_store(p.xcell + C.from + e, xbar, tag + 1);
        p.op.col_after(st, C.from + e, o, xbar, v, C.stride);
      }
    }
  } else {
    const int wr = warps - wc, w = warp - wc;
    const bool once = R.count <= 32 * wr;
    ResidentRow<GB, kLong, T> r;
    if (once) r.open(R, 32 * w + lane < R.count ? 32 * w + lane : -1);
    const bool held = once && r.longest <= GB;
    for (int s = 0; s < K; ++s) {
      const auto st = p.op.step(s);
      const unsigned tag = p.tag + static_cast<unsigned>(s) + 1;
      for (int e0 = 32 * w; e0 < R.count; e0 += 32 * wr) {
        const int e = e0 + lane < R.count ? e0 + lane : -1;
        if (!held) r.open(R, e);
        T* v = R.vec + (e >= 0 ? e : 0);
        auto o = p.op.row_before(v, R.stride);
        const double sum = resident_sum(r, R, p.xcell, tag, e0 == 32 * w, dead);
        if (e < 0) continue;
        const T ny = p.op.row(st, sum, o);
        cell_store(p.ycell + R.from + e, ny, tag);
        p.op.row_after(st, R.from + e, o, ny, v, R.stride);
      }
    }
  }
  if (dead) count_stage_timeout(p.err);
}

// kLong: with the code for long rows, for LPs that have one (in the kernels of 64 registers it costs spills).
template <int kThreads, int GB, bool kLong, class T, class Op>
__global__ void __launch_bounds__(kThreads, 1) k_resident(const __grid_constant__ ResidentPart<T, Op> p) {
  resident_body<GB, kLong>(p, static_cast<int>(blockIdx.x));
}

// Several LPs in one launch (the request loop): blocks [0, blocks_d) are the fp64 LPs', the ones after them
// the fp32 LPs' (whose `first` counts from there). A block copies its LP's part to shared memory.
template <int kThreads, int GB, bool kLong, template <class> class Op>
__global__ void __launch_bounds__(kThreads, 1) k_resident_group(const ResidentPart<double, Op<double>>* __restrict__ pd, int nd,
                                                                int blocks_d, const ResidentPart<float, Op<float>>* __restrict__ pf,
                                                                int nf) {
  auto run = [](const auto* parts, int n, int b) {
    using Part = std::decay_t<decltype(*parts)>;
    __shared__ alignas(16) unsigned char held[sizeof(Part)];
    int k = 0;
    while (k + 1 < n && __ldg(&parts[k + 1].first) <= b) ++k;
    for (unsigned q = threadIdx.x; q < sizeof(Part) / 4; q += blockDim.x)
      reinterpret_cast<unsigned*>(held)[q] = __ldg(reinterpret_cast<const unsigned*>(parts + k) + q);
    __syncthreads();
    const Part& p = *reinterpret_cast<const Part*>(held);
    resident_body<GB, kLong>(p, b - p.first);
  };
  const int b = static_cast<int>(blockIdx.x);
  if (b < blocks_d) run(pd, nd, b);
  else run(pf, nf, b - blocks_d);
}
// false: refused (launch_cooperative).
template <template <class> class Op>
inline bool launch_resident_group(const ResidentPart<double, Op<double>>* pd, int nd, int blocks_d,
                                  const ResidentPart<float, Op<float>>* pf, int nf, int blocks, int threads, int longest,
                                  unsigned smem, cudaStream_t st) {
  const auto kernel = [&](auto is_long) {
    constexpr bool kLong = decltype(is_long)::value;
    return threads <= 256   ? reinterpret_cast<const void*>(&k_resident_group<256, 16, kLong, Op>)
           : threads <= 512 ? reinterpret_cast<const void*>(&k_resident_group<512, 8, kLong, Op>)
                            : reinterpret_cast<const void*>(&k_resident_group<1024, 4, kLong, Op>);
  };
  const void* f = resident_is_long(longest, threads) ? kernel(std::true_type{}) : kernel(std::false_type{});
  B200_CHECK(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kResidentSmem)));
  void* args[] = {&pd, &nd, &blocks_d, &pf, &nf};
  return launch_cooperative(f, blocks, threads, args, smem, st);
}

// How one LP's epochs are launched: blocks, threads and dynamic shared memory; blocks = 0: not this way.
struct ResidentShape {
  int blocks = 0, threads = 0;
  int longest = 0;  // entries of the longest row or column
  unsigned smem = 0;
};
// Threads for one column or row each, and a warp for uneven shares, as far as 1,024 go.
inline int resident_threads(long long m, long long n, int blocks) {
  const long long warps = (n / blocks + 32) / 32 + (m / blocks + 32) / 32 + 1;
  return static_cast<int>(32 * std::min(32LL, std::max(2LL, warps)));
}
// One block on each of sms SMs (fewer for tiny LPs: at least 8 elements a block).
template <class T, class Op>
inline ResidentShape resident_shape(long long m, long long n, long long nnz, long long max_row, long long max_col, int sms) {
  ResidentShape s;
  if (m < 1 || n < 1 || nnz < 1) return s;
  const int blocks = static_cast<int>(std::max(1LL, std::min<long long>(sms, (m + n + 7) / 8)));
  const int threads = resident_threads(m, n, blocks), longest = static_cast<int>(std::max(max_row, max_col));
  const long long bytes = resident_bytes<T, Op>(m, n, nnz, max_row, max_col, blocks) + resident_chunks(longest, threads);
  if (bytes > kResidentSmem || (m + n) / blocks > kResidentElements) return s;
  s.blocks = blocks;
  s.threads = threads;
  s.longest = longest;
  s.smem = static_cast<unsigned>(bytes);
  return s;
}
// Launches one epoch cooperatively on `st`; false: refused (launch_cooperative).
template <class T, class Op>
inline bool launch_resident(const ResidentPart<T, Op>& p, const ResidentShape& s, cudaStream_t st) {
  const auto kernel = [&](auto is_long) {
    constexpr bool kLong = decltype(is_long)::value;
    return s.threads <= 256   ? reinterpret_cast<const void*>(&k_resident<256, 16, kLong, T, Op>)
           : s.threads <= 512 ? reinterpret_cast<const void*>(&k_resident<512, 8, kLong, T, Op>)
                              : reinterpret_cast<const void*>(&k_resident<1024, 4, kLong, T, Op>);
  };
  const void* f = resident_is_long(s.longest, s.threads) ? kernel(std::true_type{}) : kernel(std::false_type{});
  B200_CHECK(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kResidentSmem)));
  void* args[] = {const_cast<ResidentPart<T, Op>*>(&p)};
  return launch_cooperative(f, s.blocks, s.threads, args, s.smem, st);
}

}  // namespace b200
