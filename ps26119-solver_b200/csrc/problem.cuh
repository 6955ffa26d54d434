// problem.cuh — the scaled problem resident on the device (≙ pdhg::ScaledProblem,
// reference src/pdhg/scaling.h:48-67) and the ‖Ã‖₂ estimate (la::estimate_norm2,
// src/la/csr.cpp:86-132), both computed on the device.
//
// HBM layout (m rows, n cols, nnz nonzeros; int32 indices):
//   A_orig  CSR  a_rp[m+1] a_col[nnz] a_v0[nnz]          (original values, rows sorted by col)
//   Aᵀ_orig CSC  the caller's col_start/row_index/value  (borrowed; original order)
//   Ãᵀ      CSR  col_start[n+1] t_ri[nnz] sat[nnz]       (CSC of Ã, rows sorted inside columns)
//   Ã       CSR  a_rp a_col sa[nnz]                      (shares A_orig's structure)
//   fp32 copies saf / satf and of the scaled vectors for mixed precision.
#pragma once

#include <algorithm>
#include <array>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

#include "engine.hpp"
#include "lanczos.cuh"
#include "reduce.cuh"
#include "setup.cuh"
#include "spmv.cuh"
#include "tune.hpp"

namespace b200 {

static __global__ void k_fill_d(long long n, double* v, double a) {
  B200_FOR(i, n) v[i] = a;
}
static __global__ void k_absmax(long long n, const double* v, unsigned long long* key) {
  double mx = 0.0;
  B200_FOR(i, n) mx = std_max(mx, fabs(v[i]));
  warp_max_atomic(key, mx);
}
// ---------------------------------------------------------------------- Lanczos
// The start vector is the reference's xorshift64* stream: entry j comes from the generator's state
// after j + 1 updates. An update is linear over GF(2), so a thread jumps to its place with the powers
// kStartRun·2^k of the update's matrix (the state's bits select columns to xor) and then steps through
// kStartRun entries; the reference walks the stream from its seed. terms receives v[j]².
constexpr int kStartRun = 32;
constexpr int kStartPowers = 27;  // 32·2^27 entries and more
static __global__ void k_lanczos_start(int n, const unsigned long long* jump, double* v, double* terms) {
  const long long run = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  const long long j0 = run * kStartRun;
  if (j0 >= n) return;
  unsigned long long s = 0x9E3779B97F4A7C15ULL;
  for (int k = 0; k < kStartPowers && (run >> k) != 0; ++k) {
    if (!((run >> k) & 1)) continue;
    unsigned long long to = 0;
    for (int b = 0; b < 64; ++b) to ^= ((s >> b) & 1ULL) ? __ldg(jump + k * 64 + b) : 0ULL;
    s = to;
  }
  for (long long j = j0; j < j0 + kStartRun && j < n; ++j) {
    s ^= s >> 12, s ^= s << 25, s ^= s >> 27;
    const double e = static_cast<double>((s * 0x2545F4914F6CDD1DULL) >> 11) / 9007199254740992.0 * 2.0 - 1.0;
    v[j] = e;
    terms[j] = e * e;
  }
}
// The jump matrices: column b of power k is the state that bit b becomes after kStartRun·2^k updates.
inline const std::vector<unsigned long long>& lanczos_jumps() {
  static const std::vector<unsigned long long> all = [] {
    using Cols = std::array<unsigned long long, 64>;
    auto apply = [](const Cols& m, unsigned long long x) {
      unsigned long long y = 0;
      for (int b = 0; b < 64; ++b)
        if ((x >> b) & 1) y ^= m[static_cast<std::size_t>(b)];
      return y;
    };
    Cols m;
    for (int b = 0; b < 64; ++b) {
      unsigned long long s = 1ULL << b;
      s ^= s >> 12, s ^= s << 25, s ^= s >> 27;
      m[static_cast<std::size_t>(b)] = s;
    }
    auto square = [&] {
      Cols q;
      for (std::size_t b = 0; b < 64; ++b) q[b] = apply(m, m[b]);
      m = q;
    };
    for (int k = 1; k < kStartRun; k <<= 1) square();
    std::vector<unsigned long long> out;
    for (int k = 0; k < kStartPowers; ++k, square()) out.insert(out.end(), m.begin(), m.end());
    return out;
  }();
  return all;
}
static __global__ void k_lanczos_normalise(int n, double* v, double* vprev, const double* sq) {
  const double nv = sqrt(*sq);
  B200_FOR(j, n) {
    v[j] = v[j] / nv;
    vprev[j] = 0.0;
  }
}
// After w = Ãᵀt: the terms of α = wᵀv and, where a slab is a tile of terms, their tile sums (reduce.cuh) on the
// way (stat: null otherwise, and the sum makes its own).
constexpr bool kLanczosStat = kSlabRows == kXTile;
struct EpiLanczosW : AlwaysActive {
  const double* v;
  double *w, *terms, *stat;
  struct Acc {
    double term = 0.0;
  };
  __device__ void operator()(int j, double s, Acc& acc) const {
    w[j] = s;
    acc.term = s * v[j];
    terms[j] = acc.term;
  }
  __device__ void flush(const Acc& acc) const { x_leave_stat(stat, acc.term); }
};
// w[j] -= al*v[j] + bprev*vprev[j]; terms[j] = w[j]² (csr.cpp:108-112), with α and β_prev² read
// from the device, where the sums left them (sqrt correctly rounded, as the host's std::sqrt).
// Launched with one thread per entry in blocks of kXTile, for the tile sums.
static __global__ void __launch_bounds__(kXTile) k_lanczos_update(int n, double* w, const double* v, const double* vprev,
                                                                  const double* ab, double* terms, double* stat) {
  const int j = blockIdx.x * kXTile + threadIdx.x;
  double term = 0.0;
  pdl_wait();
  if (j < n) {
    const double e = w[j] - (ab[0] * v[j] + sqrt(ab[1]) * vprev[j]);
    w[j] = e;
    term = e * e;
    terms[j] = term;
  }
  x_leave_stat(stat, term);
}
// The next Lanczos vector, w/β; hist receives (α, β²) of this step for the host's later replay.
static __global__ void k_lanczos_next(int n, const double* w, double* v, double* vprev, const double* ab, double* hist) {
  pdl_wait();
  const double bn = sqrt(ab[1]);
  if (blockIdx.x == 0 && threadIdx.x == 0) hist[0] = ab[0], hist[1] = ab[1];
  B200_FOR(j, n) {
    vprev[j] = v[j];
    v[j] = w[j] / bn;
  }
}

struct ScaledDevice {
  int m = 0, n = 0, sense = 1;
  long long nnz = 0;
  DeviceModel M;
  DevBuf<int> a_rp, a_col, t_ri;
  DevBuf<int> t_rp;  // this library's copy of the caller's col_start (Ãᵀ row pointers, TMA-staged)
  DevBuf<double> a_v0, t_v0, sa, sat;
  DevBuf<float> saf, satf;
  DevBuf<double> row_scale, col_scale;
  DevBuf<double> sc, scl, scu, srl, sru;
  DevBuf<float> scf, sclf, scuf, srlf, sruf;
  double bound_scale = 1.0, obj_scale = 1.0, log10_range = 0.0;
  bool gm_applied = false, have_f32 = false, exact = false;
  // original-space constants of kkt_general (cpu_backend.cpp:233-262): ‖b‖₂, ‖c‖₂, ‖c‖∞
  double b_norm = 0, c_norm = 0, c_inf = 0;
  long long kernels = 0;
  RowLengths lengths_[2];  // of the rows, of the columns
  bool have_lengths = false;
  int lanczos_launched = 0;  // Lanczos steps launched by the last lanczos() (counted or not)

  // Scratch for the setup reductions.
  DevBuf<double> tmp_m, tmp_n, fac_m, fac_n, sums;
  DevBuf<unsigned long long> keys;

  void build(const DeviceModel& dm, const ScalingOptions& so, bool exact_order, cudaStream_t st) {
    M = dm;
    m = dm.m, n = dm.n, sense = dm.sense, nnz = dm.nnz;
    exact = exact_order;
    have_lengths = false;
    const std::size_t mm = static_cast<std::size_t>(m), nn = static_cast<std::size_t>(n);
    const std::size_t nz = static_cast<std::size_t>(nnz);
    a_rp.alloc(mm + 1);
    t_rp.alloc(nn + 1);
    B200_CHECK(cudaMemcpyAsync(t_rp.get(), dm.col_start, (nn + 1) * sizeof(int), cudaMemcpyDeviceToDevice, st));
    a_col.alloc(nz);
    a_v0.alloc(nz);
    t_ri.alloc(nz);
    t_v0.alloc(nz);
    sa.alloc(nz);
    sat.alloc(nz);
    row_scale.alloc(mm);
    col_scale.alloc(nn);
    tmp_m.alloc(mm + 1);
    tmp_n.alloc(nn + 1);
    fac_m.alloc(mm + 1);
    fac_n.alloc(nn + 1);
    sums.alloc(16);
    keys.alloc(4);

    // ---- CSR of A (la::transpose of the CSC, csr.cpp:19-36)
    {
      DevBuf<int> counts(mm + 1), cursor(mm + 1), long_rows(std::max(mm, nn) + 1), n_long(1);
      B200_CHECK(cudaMemsetAsync(counts.get(), 0, (mm + 1) * sizeof(int), st));
      if (nnz > 0) k_count<<<grid_for(nnz), kBlock, 0, st>>>(nnz, dm.row_index, counts.get());
      B200_LAUNCH_CHECK();
      exclusive_scan(counts.get(), a_rp.get(), static_cast<long long>(mm) + 1, st);
      B200_CHECK(cudaMemcpyAsync(cursor.get(), a_rp.get(), (mm + 1) * sizeof(int), cudaMemcpyDeviceToDevice, st));
      if (n > 0)
        k_scatter<<<grid_for(n), kBlock, 0, st>>>(n, dm.col_start, dm.row_index, dm.value, cursor.get(), a_col.get(),
                                                  a_v0.get());
      B200_LAUNCH_CHECK();
      sort_segments(m, a_rp.get(), a_col.get(), a_v0.get(), long_rows.get(), n_long.get(), st);
      // canonical CSC of A (rows sorted inside each column) = CSR of Aᵀ as la::transpose makes it
      if (nnz > 0) {
        B200_CHECK(cudaMemcpyAsync(t_ri.get(), dm.row_index, nz * sizeof(int), cudaMemcpyDeviceToDevice, st));
        B200_CHECK(cudaMemcpyAsync(t_v0.get(), dm.value, nz * sizeof(double), cudaMemcpyDeviceToDevice, st));
      }
      sort_segments(n, dm.col_start, t_ri.get(), t_v0.get(), long_rows.get(), n_long.get(), st);
      B200_CHECK(cudaStreamSynchronize(st));
    }
    if (nnz > 0) {
      B200_CHECK(cudaMemcpyAsync(sa.get(), a_v0.get(), nz * sizeof(double), cudaMemcpyDeviceToDevice, st));
      B200_CHECK(cudaMemcpyAsync(sat.get(), t_v0.get(), nz * sizeof(double), cudaMemcpyDeviceToDevice, st));
    }
    k_fill_d<<<grid_for(mm), kBlock, 0, st>>>(static_cast<long long>(mm), row_scale.get(), 1.0);
    k_fill_d<<<grid_for(nn), kBlock, 0, st>>>(static_cast<long long>(nn), col_scale.get(), 1.0);
    B200_LAUNCH_CHECK();

    // ---- log10 range of |a| (scaling.cpp:51-56)
    {
      unsigned long long init[2] = {0x7ff0000000000000ULL /* +inf */, 0ULL};
      B200_CHECK(cudaMemcpyAsync(keys.get(), init, sizeof init, cudaMemcpyHostToDevice, st));
      if (nnz > 0)
        k_abs_range<<<std::min(grid_for(nnz), 8 * sm_count()), kBlock, 0, st>>>(nnz, a_v0.get(), keys.get(), keys.get() + 1);
      B200_LAUNCH_CHECK();
      unsigned long long got[2];
      B200_CHECK(cudaMemcpyAsync(got, keys.get(), sizeof got, cudaMemcpyDeviceToHost, st));
      B200_CHECK(cudaStreamSynchronize(st));
      double amin, amax;
      std::memcpy(&amin, &got[0], sizeof amin);
      std::memcpy(&amax, &got[1], sizeof amax);
      log10_range = amax > 0 ? std::log10(amax / amin) : 0.0;
    }
    gm_applied = so.geometric_mean_iterations > 0 && log10_range >= so.geometric_mean_min_log10_range;
    if (gm_applied) {  // scaling.cpp:57-80: factors from the ORIGINAL entries, applied once
      for (int it = 0; it < so.geometric_mean_iterations; ++it) {
        k_gm_pass<<<grid_for(mm), kBlock, 0, st>>>(m, a_rp.get(), a_col.get(), a_v0.get(), col_scale.get(),
                                                   row_scale.get());
        k_gm_pass<<<grid_for(nn), kBlock, 0, st>>>(n, dm.col_start, dm.row_index, dm.value, row_scale.get(),
                                                   col_scale.get());
        B200_LAUNCH_CHECK();
      }
    }
    scale_entries(so, st);

    sc.alloc(nn), scl.alloc(nn), scu.alloc(nn), srl.alloc(mm), sru.alloc(mm);
    k_scaled_cols<<<grid_for(nn), kBlock, 0, st>>>(n, sense, dm.c, dm.col_lower, dm.col_upper, col_scale.get(),
                                                   sc.get(), scl.get(), scu.get());
    k_scaled_rows<<<grid_for(mm), kBlock, 0, st>>>(m, dm.row_lower, dm.row_upper, row_scale.get(), srl.get(),
                                                   sru.get());
    B200_LAUNCH_CHECK();
    if (so.bound_objective_rescaling) {  // scaling.cpp:126-141
      double b2 = 0, c2 = 0;
      seq_sums(st, [&](double* tm, double* tn) {
        k_b2_terms<<<grid_for(mm), kBlock, 0, st>>>(m, srl.get(), sru.get(), tm);
        k_sq_terms<<<grid_for(nn), kBlock, 0, st>>>(static_cast<long long>(nn), sc.get(), tn);
      }, b2, c2);
      bound_scale = 1.0 / (std::sqrt(b2) + 1.0);
      obj_scale = 1.0 / (std::sqrt(c2) + 1.0);
      k_scale_vec<<<grid_for(mm), kBlock, 0, st>>>(static_cast<long long>(mm), srl.get(), bound_scale);
      k_scale_vec<<<grid_for(mm), kBlock, 0, st>>>(static_cast<long long>(mm), sru.get(), bound_scale);
      k_scale_vec<<<grid_for(nn), kBlock, 0, st>>>(static_cast<long long>(nn), scl.get(), bound_scale);
      k_scale_vec<<<grid_for(nn), kBlock, 0, st>>>(static_cast<long long>(nn), scu.get(), bound_scale);
      k_scale_vec<<<grid_for(nn), kBlock, 0, st>>>(static_cast<long long>(nn), sc.get(), obj_scale);
      B200_LAUNCH_CHECK();
    }
    // ---- original-space constants of kkt_general
    {
      double b2 = 0, c2 = 0;
      seq_sums(st, [&](double* tm, double* tn) {
        k_b2_terms<<<grid_for(mm), kBlock, 0, st>>>(m, dm.row_lower, dm.row_upper, tm);
        k_sq_terms<<<grid_for(nn), kBlock, 0, st>>>(static_cast<long long>(nn), dm.c, tn);
      }, b2, c2);
      b_norm = std::sqrt(b2);
      c_norm = std::sqrt(c2);
      B200_CHECK(cudaMemsetAsync(keys.get(), 0, sizeof(unsigned long long), st));
      k_absmax<<<std::min(grid_for(nn), 8 * sm_count()), kBlock, 0, st>>>(static_cast<long long>(nn), dm.c, keys.get());
      B200_LAUNCH_CHECK();
      unsigned long long key = 0;
      B200_CHECK(cudaMemcpyAsync(&key, keys.get(), sizeof key, cudaMemcpyDeviceToHost, st));
      B200_CHECK(cudaStreamSynchronize(st));
      std::memcpy(&c_inf, &key, sizeof c_inf);
    }
  }

  void make_f32(cudaStream_t st) {
    if (have_f32) return;
    const long long nz = nnz, nn = n, mm = m;
    saf.alloc(static_cast<std::size_t>(nz)), satf.alloc(static_cast<std::size_t>(nz));
    scf.alloc(n), sclf.alloc(n), scuf.alloc(n), srlf.alloc(m), sruf.alloc(m);
    k_convert<float, double><<<grid_for(nz), kBlock, 0, st>>>(nz, sa.get(), saf.get());
    k_convert<float, double><<<grid_for(nz), kBlock, 0, st>>>(nz, sat.get(), satf.get());
    k_convert<float, double><<<grid_for(nn), kBlock, 0, st>>>(nn, sc.get(), scf.get());
    k_convert<float, double><<<grid_for(nn), kBlock, 0, st>>>(nn, scl.get(), sclf.get());
    k_convert<float, double><<<grid_for(nn), kBlock, 0, st>>>(nn, scu.get(), scuf.get());
    k_convert<float, double><<<grid_for(mm), kBlock, 0, st>>>(mm, srl.get(), srlf.get());
    k_convert<float, double><<<grid_for(mm), kBlock, 0, st>>>(mm, sru.get(), sruf.get());
    B200_LAUNCH_CHECK();
    have_f32 = true;
  }

  // Scaled matrix views for SpMV in precision T.
  template <class T> const T* A_val() const;
  template <class T> const T* At_val() const;
  template <class T> const T* c() const;
  template <class T> const T* l() const;
  template <class T> const T* u() const;
  template <class T> const T* rl() const;
  template <class T> const T* ru() const;

  // The lengths of the rows [0] and of the columns [1] (cached by the problem; synchronises the stream the
  // first time).
  const RowLengths* lengths(cudaStream_t st) {
    if (!have_lengths) {
      static_assert(sizeof lengths_ == 6 * sizeof(int), "three numbers a side");
      DevBuf<int> d(6);
      B200_CHECK(cudaMemsetAsync(d.get(), 0, sizeof lengths_, st));
      if (m > 0) k_extents<<<std::min(grid_for(m), 8 * sm_count()), kBlock, 0, st>>>(m, a_rp.get(), d.get());
      if (n > 0) k_extents<<<std::min(grid_for(n), 8 * sm_count()), kBlock, 0, st>>>(n, t_rp.get(), d.get() + 3);
      B200_LAUNCH_CHECK();
      kernels += 2;
      B200_CHECK(cudaMemcpyAsync(lengths_, d.get(), sizeof lengths_, cudaMemcpyDeviceToHost, st));
      B200_CHECK(cudaStreamSynchronize(st));
      have_lengths = true;
    }
    return lengths_;
  }

  // ‖Ã‖₂ by Lanczos on ÃᵀÃ (csr.cpp:86-132), on the device: the reference's start vector, the
  // products, and α and β reduced in the reference's order. α and β stay on the device, where the
  // next step's update reads them; the host reads them back a batch of steps at a time (21, then 8)
  // and replays the reference's per-step decisions on them (Sturm bisection, breakdown and
  // stagnation tests) in step order while the device runs the next batch. The result and the number
  // of steps that count are the sequential loop's; steps run past the stopping one are discarded.
  // err: the caller's counter of waits that ran out on the device (nullptr: one of this call's own). When it
  // counts any the estimate ends there and throws.
  double lanczos(cudaStream_t st, unsigned* err = nullptr) {
    if (n == 0 || nnz == 0) return 0.0;
    DevBuf<unsigned> own;
    if (!err) {
      own.alloc(1);
      B200_CHECK(cudaMemsetAsync(own.get(), 0, sizeof(unsigned), st));
      err = own.get();
    }
    const int K = 400;
    const double rel_tol = 1e-12;
    lanczos_launched = 0;
    DevBuf<double> v(n), vprev(n), w(n), t(m), terms(n);
    DevBuf<double> out(2), hist(2 * static_cast<std::size_t>(K));
    DevBuf<unsigned long long> jump;
    jump.upload(lanczos_jumps().data(), lanczos_jumps().size(), st);
    SumPlan pal, pbn;
    pal.add(terms.get(), 0, n, 0.0, SumOrder::kSeq, out.get());
    pbn.add(terms.get(), 0, n, 0.0, SumOrder::kSeq, out.get() + 1);
    pbn.build(true, nullptr, st);  // α and β enter η = 0.998/‖Ã‖₂: always the reference's order
    k_lanczos_start<<<grid_for((n + kStartRun - 1) / kStartRun, 64), 64, 0, st>>>(n, jump.get(), v.get(), terms.get());
    B200_LAUNCH_CHECK();
    pbn.launch(st);
    k_lanczos_normalise<<<grid_for(n), kBlock, 0, st>>>(n, v.get(), vprev.get(), out.get() + 1);
    B200_LAUNCH_CHECK();
    B200_CHECK(cudaMemsetAsync(out.get() + 1, 0, sizeof(double), st));  // no β before the first step
    kernels += 2 + pbn.kernel_count();
    const int tiles = (n + kXTile - 1) / kXTile;
    // An LP that fits the SMs' shared memory takes a batch of steps in one launch (lanczos.cuh).
    const RowLengths* len = lengths(st);
    LanczosShape shape;
    if (tune_forced() < 0)  // a forced step-kernel variant: no cooperative launches
      shape = lanczos_shape(m, n, nnz, len[0].longest, len[1].longest, stream_sm_count(st));
    DevBuf<Cell<double>> cells;
    DevBuf<XFast> fast;
    DevBuf<XTileAgg> full;
    DevBuf<unsigned> count(1);
    unsigned tag = 1;
    const int polls = lanczos_polls();
    if (shape.blocks > 0) {
      cells.alloc(static_cast<std::size_t>(LanczosArgs::cells(m, n, shape.blocks)));
      fast.alloc(static_cast<std::size_t>(n / kXTile + shape.blocks));
      full.alloc(static_cast<std::size_t>(n / kXTile + shape.blocks));
      B200_CHECK(cudaMemsetAsync(cells.get(), 0, cells.size() * sizeof(Cell<double>), st));
      B200_CHECK(cudaMemsetAsync(fast.get(), 0, fast.size() * sizeof(XFast), st));
      B200_CHECK(cudaMemsetAsync(count.get(), 0, sizeof(unsigned), st));
    } else {
      pal.build(true, nullptr, st);
    }
    auto launch = [&](int from, int to) {
      if (shape.blocks > 0) {
        Cell<double>* c = cells.get();
        if (launch_lanczos({m, n, shape.blocks, t_rp.get(), t_ri.get(), a_rp.get(), a_col.get(), sat.get(), sa.get(),
                            c, c + n, c + n + m, c + n + m + shape.blocks, c + n + m + 2 * shape.blocks, v.get(), vprev.get(),
                            terms.get(), hist.get(), fast.get(), full.get(), count.get(), tag, from, to, polls, err},
                           shape, st)) {
          tag += 3u * static_cast<unsigned>(to - from) + 2u;
          ++kernels;
          lanczos_launched = to;
          return;
        }
        shape.blocks = 0;  // refused: the kernels' form, from here on
        pal.build(true, nullptr, st);
        if (from > 0)
          B200_CHECK(cudaMemcpyAsync(out.get() + 1, hist.get() + 2 * from - 1, sizeof(double), cudaMemcpyDeviceToDevice, st));
      }
      for (int k = from; k < to; ++k) {
        // every kernel of a step starts while the one before it ends (programmatic dependent launch)
        launch_slab_tma<double>(m, a_rp.get(), a_col.get(), sa.get(), v.get(), EpiStore<double>{{}, t.get()}, st,
                                nullptr, err, true);
        launch_slab_tma<double>(n, t_rp.get(), t_ri.get(), sat.get(), t.get(),
                                EpiLanczosW{{}, v.get(), w.get(), terms.get(), kLanczosStat ? pal.stat() : nullptr}, st,
                                nullptr, err, true);
        pal.launch(st, kLanczosStat);
        // β of the previous step is still in out[1]: this step's β² overwrites it only below
        launch_pdl(k_lanczos_update, tiles, kXTile, st, n, w.get(), v.get(), vprev.get(), out.get(), terms.get(), pbn.stat());
        pbn.launch(st, true);
        launch_pdl(k_lanczos_next, grid_for(n), kBlock, st, n, w.get(), v.get(), vprev.get(), out.get(), hist.get() + 2 * k);
        kernels += 5 + (kLanczosStat ? 1 : pal.kernel_count());
      }
      lanczos_launched = to;
    };
    PinnedBuf<double> h;
    PinnedBuf<unsigned> ran_out;
    h.alloc(2 * static_cast<std::size_t>(K)), ran_out.alloc(1);
    ran_out[0] = 0;
    Event landed[2];
    std::vector<double> alpha, beta;
    double theta = 0, theta_old = -1;
    int stagnant = 0;
    int from = 0, to = std::min(K, 21), slot = 0;
    const long long walk = static_cast<long long>(len[0].longest) + len[1].longest;
    auto fetch = [&](int a, int b, int s) {
      B200_CHECK(cudaMemcpyAsync(h.get() + 2 * a, hist.get() + 2 * a, 2 * static_cast<std::size_t>(b - a) * sizeof(double),
                                 cudaMemcpyDeviceToHost, st));
      B200_CHECK(cudaMemcpyAsync(ran_out.get(), err, sizeof(unsigned), cudaMemcpyDeviceToHost, st));
      B200_CHECK(cudaEventRecord(landed[s].get(), st));
    };
    launch(from, to);
    fetch(from, to, slot);
    for (bool done = false; !done;) {
      // The device goes on while the host looks at this batch, where a step is cheap against the
      // host's look or the run is long; else the steps past the stop would cost more than the wait. What a
      // step costs is in its columns, its nonzeros, and the longest row and column, which one thread walks each
      // (0.13 us an entry). Looking ahead regardless / so, ms: 20k rows of 300 columns, dense, 7,350 / 5,220; 2,000 of
      // 3,000, dense, 1,452 / 1,258; 20k rows of 200 17.2 / 12.4; 100k rows of 30 2.9 / 2.4; a band of 150k rows of 24
      // 2.8 / 2.2 (without these steps the first three took 5,550, 1,280 and 15.2 ms).
      const bool ahead = (n <= (1 << 18) && nnz <= (1 << 21) && walk <= 512) || (to >= 100 && nnz <= (1 << 24) && walk <= 4096);
      const int next = std::min(K, to + 8);
      auto go_on = [&] {
        if (next > to) launch(to, next), fetch(to, next, slot ^ 1);
      };
      if (ahead) go_on();
      B200_CHECK(cudaEventSynchronize(landed[slot].get()));
      if (ran_out[0]) break;
      for (int k = from; k < to; ++k) alpha.push_back(h[2 * k]), beta.push_back(std::sqrt(h[2 * k + 1]));
      double thetas[21];
      tridiag_max_eigs(alpha.data(), beta.data(), from + 1, to - from, thetas);
      for (int k = from; k < to && !done; ++k) {  // the reference's loop body, step by step
        const double bn = beta[static_cast<std::size_t>(k)];
        theta = thetas[k - from];
        if (bn <= 1e-14 * std_max(1.0, theta)) done = true;
        else if (theta - theta_old <= rel_tol * theta) done = ++stagnant >= 5 && k >= 20;
        else stagnant = 0;
        theta_old = theta;
      }
      if (to >= K) done = true;
      if (!done && !ahead) go_on();
      from = to, to = next, slot ^= 1;
    }
    B200_CHECK(cudaStreamSynchronize(st));  // the steps past the stop, before their buffers go back
    if (ran_out[0]) throw CudaError("a shared-memory staging wait timed out on the device");
    return std::sqrt(std_max(theta, 0.0)) * (1.0 + 1e-4);
  }

  // Largest eigenvalues of the leading k0, k0 + 1, …, k0 + count − 1 rows of the Lanczos tridiagonal
  // (a, b), each by the reference's Sturm bisection (csr.cpp:54-84). One bisection is a chain of
  // divisions; up to 8 of them go through the recurrence side by side.
  static void tridiag_max_eigs(const double* a, const double* b, int k0, int count, double* out) {
    constexpr int L = 8;
    for (int f = 0; f < count; f += L) {
      const int c = std::min(L, count - f);
      double lo[L], hi[L], mid[L], d[L];
      int k[L], it[L], neg[L];
      bool open[L];
      for (int q = 0; q < L; ++q) {
        k[q] = k0 + f + std::min(q, c - 1), it[q] = 0, lo[q] = 1e300, hi[q] = -1e300;
        for (int i = 0; i < k[q]; ++i) {
          const double r = (i > 0 ? std::fabs(b[i - 1]) : 0.0) + (i + 1 < k[q] ? std::fabs(b[i]) : 0.0);
          lo[q] = std_min(lo[q], a[i] - r);
          hi[q] = std_max(hi[q], a[i] + r);
        }
      }
      for (;;) {
        bool any = false;
        for (int q = 0; q < L; ++q) {
          open[q] = q < c && it[q] < 200 && hi[q] - lo[q] > 1e-15 * std_max(1.0, std::fabs(hi[q]));
          any = any || open[q];
          mid[q] = 0.5 * (lo[q] + hi[q]);
          neg[q] = 0, d[q] = 1.0;
        }
        if (!any) break;
        const int shortest = k[0], longest = k[c - 1];
        for (int i = 0; i < shortest; ++i) {
          const double ai = a[i], bb = i > 0 ? b[i - 1] * b[i - 1] : 0.0;
          for (int q = 0; q < L; ++q) {
            d[q] = (ai - mid[q]) - (i > 0 ? bb / d[q] : 0.0);
            d[q] = d[q] == 0.0 ? -1e-300 : d[q];
            neg[q] += d[q] < 0 ? 1 : 0;
          }
        }
        for (int i = shortest; i < longest; ++i) {
          const double ai = a[i], bb = i > 0 ? b[i - 1] * b[i - 1] : 0.0;
          for (int q = 0; q < c; ++q) {
            if (i >= k[q]) continue;
            d[q] = (ai - mid[q]) - (i > 0 ? bb / d[q] : 0.0);
            if (d[q] == 0.0) d[q] = -1e-300;
            if (d[q] < 0) ++neg[q];
          }
        }
        for (int q = 0; q < L; ++q) {
          if (!open[q]) continue;
          ++it[q];
          if (neg[q] == k[q]) hi[q] = mid[q];
          else lo[q] = mid[q];
        }
      }
      for (int q = 0; q < c; ++q) out[f + q] = hi[q];
    }
  }

 private:
  static void sort_segments(int rows, const int* rp, int* key, double* val, int* long_rows, int* n_long,
                                     cudaStream_t st) {
    if (rows <= 0) return;
    B200_CHECK(cudaMemsetAsync(n_long, 0, sizeof(int), st));
    k_sort_short<<<grid_for(rows), kBlock, 0, st>>>(rows, rp, key, val, long_rows, n_long);
    B200_LAUNCH_CHECK();
    k_sort_long<<<148, 512, 0, st>>>(rp, long_rows, n_long, key, val);
    B200_LAUNCH_CHECK();
  }

  // The geometric means' factors (if there are any: the scales so far), then the Ruiz (∞-norm) steps
  // (scaling.cpp:81-88) and the Pock–Chambolle (1-norm, α = 1) step (scaling.cpp:89-96): each step's factors
  // 1/√norm, applied to Ã and Ãᵀ by the next step's launches, accumulated into the scales. A step reads the
  // factors of the one before while it writes its own, so there are two buffers a side.
  void scale_entries(const ScalingOptions& so, cudaStream_t st) {
    double* rf[2] = {fac_m.get(), tmp_m.get()};
    double* cf[2] = {fac_n.get(), tmp_n.get()};
    int cur = 0;
    bool pending = gm_applied;
    if (pending) {
      B200_CHECK(cudaMemcpyAsync(rf[0], row_scale.get(), sizeof(double) * m, cudaMemcpyDeviceToDevice, st));
      B200_CHECK(cudaMemcpyAsync(cf[0], col_scale.get(), sizeof(double) * n, cudaMemcpyDeviceToDevice, st));
    }
    auto step = [&](auto kernel) {
      kernel<<<grid_for(m), kBlock, 0, st>>>(m, a_rp.get(), a_col.get(), sa.get(), rf[cur], cf[cur], rf[cur ^ 1],
                                             row_scale.get());
      kernel<<<grid_for(n), kBlock, 0, st>>>(n, M.col_start, t_ri.get(), sat.get(), cf[cur], rf[cur], cf[cur ^ 1],
                                             col_scale.get());
      B200_LAUNCH_CHECK();
      cur ^= 1, pending = true;
    };
    for (int it = 0; it < so.ruiz_iterations; ++it)
      step(pending ? &k_scale_step<true, RowNorm::kMax> : &k_scale_step<false, RowNorm::kMax>);
    if (so.pock_chambolle) step(pending ? &k_scale_step<true, RowNorm::kSum> : &k_scale_step<false, RowNorm::kSum>);
    if (pending) step(&k_scale_step<true, RowNorm::kNone>);
  }

  // Two sequential-order sums: terms over m (into tmp_m) and over n (into tmp_n).
  template <class F>
  void seq_sums(cudaStream_t st, F&& fill_terms, double& sm, double& sn) {
    fill_terms(tmp_m.get(), tmp_n.get());
    B200_LAUNCH_CHECK();
    SumPlan p;
    p.add(tmp_m.get(), 0, m, 0.0, SumOrder::kSeq, sums.get());
    p.add(tmp_n.get(), 0, n, 0.0, SumOrder::kSeq, sums.get() + 1);
    p.build(true, nullptr, st);  // norms that enter the scaled data: always the reference's order
    p.launch(st);
    double h[2];
    B200_CHECK(cudaMemcpyAsync(h, sums.get(), sizeof h, cudaMemcpyDeviceToHost, st));
    B200_CHECK(cudaStreamSynchronize(st));
    sm = h[0], sn = h[1];
  }

};

template <> inline const double* ScaledDevice::A_val<double>() const { return sa.get(); }
template <> inline const float* ScaledDevice::A_val<float>() const { return saf.get(); }
template <> inline const double* ScaledDevice::At_val<double>() const { return sat.get(); }
template <> inline const float* ScaledDevice::At_val<float>() const { return satf.get(); }
template <> inline const double* ScaledDevice::c<double>() const { return sc.get(); }
template <> inline const float* ScaledDevice::c<float>() const { return scf.get(); }
template <> inline const double* ScaledDevice::l<double>() const { return scl.get(); }
template <> inline const float* ScaledDevice::l<float>() const { return sclf.get(); }
template <> inline const double* ScaledDevice::u<double>() const { return scu.get(); }
template <> inline const float* ScaledDevice::u<float>() const { return scuf.get(); }
template <> inline const double* ScaledDevice::rl<double>() const { return srl.get(); }
template <> inline const float* ScaledDevice::rl<float>() const { return srlf.get(); }
template <> inline const double* ScaledDevice::ru<double>() const { return sru.get(); }
template <> inline const float* ScaledDevice::ru<float>() const { return sruf.get(); }

}  // namespace b200
