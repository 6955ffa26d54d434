// checks.cuh — the every-K-iterations work of r²HPDHG on the device: fixed-point residual,
// KKT statistics on the ORIGINAL problem, infeasibility ray tests, and the final unscaling.
//
// A check is three launches and a publication: k_check_points (the points, the residual's and the restart
// distances' terms), k_check_products (all products with A, Ã and Aᵀ that the check needs, over packed
// points), one launch of sums, k_check_publish; PDLP's the same with k_pdlp_points / k_pdlp_products.
//
// Each kernel writes per-element TERMS of the reference's sums into term arrays (reduced by a
// SumPlan in the reference's order or a fixed tree) and folds maxima into atomic slots.
// References:
//   residual  r2hpdhg.cpp:50-59 (Δ = x̄ − x̂ etc., dots via la::parallel_sum)
//   KKT       cpu_backend.cpp:226-284 (kkt_general) with unscaling scaling.cpp:144-155
//   ray test  engine.cpp:82-155
//   finish    engine.cpp:268-307 (z = c − Aᵀy, objective)
//   check     core/solution_checker.cpp:61-133 (in-process verification)
#pragma once

#include "spmv.cuh"

namespace b200 {

// Result slots (doubles; maxima stored as the bit pattern of a non-negative double).
enum Slot : int {
  kPx0 = 0, kPy0, kCross0,                  // fixed-point residual at the epoch's first step
  kPx, kPy, kCross, kDxn2, kDyn2,           // residual at the check + restart distances
  kRp2, kD, kRd2, kP,                       // KKT sums
  kRayObj, kRayMag, kRayCd, kRayCmag,       // ray test on T(z) − z
  kRayObj2, kRayMag2, kRayCd2, kRayCmag2,   // ray test on the drift z − z0
  kObjective, kChkDual, kChkPrimal,         // finish: objective; check sums
  kNumSums,
  kMaxPmax = 32, kMaxDmax, kMaxRmax, kMaxDviol, kMaxDabs, kMaxPviol,
  kMaxRmax2, kMaxDviol2, kMaxDabs2, kMaxPviol2,
  kMaxChkPrimal, kMaxChkDual,
  kNumSlots = 48
};

__device__ __forceinline__ unsigned long long* max_slot(double* res, int s) {
  return reinterpret_cast<unsigned long long*>(res + s);
}

// ---------------------------------------------------------------------- residual
// Of a Halpern cycle's first step: dx = x̄ − x̂ written as the reference's axpby(−1, x̂, 1, dx) with
// dx = x̄; terms Δx².
template <class T>
static __global__ void k_res_x(int n, const T* __restrict__ xb, const T* __restrict__ xh, T* __restrict__ dx,
                               double* t_px, const int* skip) {
  if (skip && *skip) return;
  B200_FOR(j, n) {
    const T d = static_cast<T>(-1.0) * xh[j] + static_cast<T>(1.0) * xb[j];
    dx[j] = d;
    t_px[j] = static_cast<double>(d) * static_cast<double>(d);
  }
}
// Epilogue after adx = Ã·dx: dy = ȳ − ŷ, terms Δy², Δyᵀ(AΔx).
template <class T>
struct EpiResY {
  const T *yb, *yh;
  double *t_py, *t_cross;
  const int* skip;
  __device__ bool active() const { return !(skip && *skip); }
  __device__ void operator()(int i, double s) const {
    const T ax = static_cast<T>(s);
    const T d = static_cast<T>(-1.0) * yh[i] + static_cast<T>(1.0) * yb[i];
    t_py[i] = static_cast<double>(d) * static_cast<double>(d);
    t_cross[i] = static_cast<double>(d) * static_cast<double>(ax);
  }
};

// ---------------------------------------------------------------------- unscale
// x = clamp(C x̃ / bs, l, u), y_min = R ỹ / os (scaling.cpp:144-155)
template <class T>
static __global__ void k_unscale_x(int n, const T* xs, const double* col_scale, double bound_scale, const double* cl,
                            const double* cu, double* xo) {
  B200_FOR(j, n) xo[j] = std_min(std_max(col_scale[j] * static_cast<double>(xs[j]) / bound_scale, cl[j]), cu[j]);
}
template <class T>
static __global__ void k_unscale_y(int m, const T* ys, const double* row_scale, double obj_scale, double* yo) {
  B200_FOR(i, m) yo[i] = row_scale[i] * static_cast<double>(ys[i]) / obj_scale;
}

__device__ __forceinline__ double elem_viol(double v, double lo, double up) {
  if (v < lo) return (lo - v) / (1.0 + fabs(lo));
  if (v > up) return (v - up) / (1.0 + fabs(up));
  return 0.0;
}

// ---------------------------------------------------------------------- KKT
// Row part of kkt_general after ax = A_orig·x (row-sequential). Term arrays have m+n entries:
// rows at [0, m), columns at [m, m+n) so that sums continuing over both loops are one chain.
struct EpiKktRows : AlwaysActive {
  const double *y, *rl, *ru;
  double *t_rp2, *t_d, *t_rd2;
  double* res;
  struct Acc {
    double pmax = 0.0, dmax = 0.0;
  };
  __device__ void operator()(int i, double ax, Acc& acc) const {
    const double lo = rl[i], up = ru[i];
    const double viol = ax < lo ? lo - ax : (ax > up ? ax - up : 0.0);
    t_rp2[i] = viol * viol;
    acc.pmax = elem_viol(ax, lo, up);
    const double yi = y[i];
    double d = 0.0, rd = 0.0;
    if (yi > 0) {
      if (isfinite(lo)) d = yi * lo;
      else rd = yi * yi, acc.dmax = yi;
    } else if (yi < 0) {
      if (isfinite(up)) d = yi * up;
      else rd = yi * yi, acc.dmax = -yi;
    }
    t_d[i] = d;
    t_rd2[i] = rd;
  }
  __device__ void flush(const Acc& a) const {
    warp_max_atomic(max_slot(res, kMaxPmax), a.pmax);
    warp_max_atomic(max_slot(res, kMaxDmax), a.dmax);
  }
};
// Column part after aty = Aᵀ_orig·y (the caller's CSC order).
struct EpiKktCols : AlwaysActive {
  const double *x, *c, *cl, *cu;
  double sense;
  int m;
  double *t_p, *t_d, *t_rd2;
  double* res;
  struct Acc {
    double pmax = 0.0, dmax = 0.0;
  };
  __device__ void operator()(int j, double aty, Acc& acc) const {
    const double cj = sense * c[j];
    t_p[m + j] = cj * x[j];
    const double lo = cl[j], up = cu[j];
    acc.pmax = elem_viol(x[j], lo, up);
    const double lam = cj - aty;
    double z;
    if (isfinite(lo) && isfinite(up)) z = lam;
    else if (isfinite(lo)) z = std_max(lam, 0.0);
    else if (isfinite(up)) z = std_min(lam, 0.0);
    else z = 0.0;
    t_rd2[m + j] = (lam - z) * (lam - z);
    acc.dmax = fabs(lam - z);
    t_d[m + j] = z > 0 ? z * lo : (z < 0 ? z * up : 0.0);
  }
  __device__ void flush(const Acc& a) const {
    warp_max_atomic(max_slot(res, kMaxPmax), a.pmax);
    warp_max_atomic(max_slot(res, kMaxDmax), a.dmax);
  }
};

// ---------------------------------------------------------------------- a check in three kernels
// Everything a check evaluates on the way to its sums, for r²HPDHG: the residual's Δ, the unscaled point,
// the ray directions (kRays ≥ 1: of the last step; 2: of the drift since the restart anchor as well) and
// their products. k_check_points makes the points, one thread per column and per row, and packs what the
// products gather: X[j] = {x, Δx̃, d, d₂}, Y[i] = {y, r, r₂, 0}, 32 bytes, one sector. k_check_products then
// walks every row and every column once for all of them. Each value is the one that the kernels above
// compute, sums in the same order; the terms go to the same arrays.
// PDLP's check has the same two kernels (k_pdlp_points, k_pdlp_products): the KKT statistics of the current
// point and of the average, and the rays of the last step and of the drift; X[j] = {x, x_avg, d, d₂},
// Y[i] = {y, y_avg, r, r₂}.
// What bounds it: for LPs up to some 100k rows the number of dependent launches (up to 15 in the longest
// chain before, 4 now); for large ones the gathers (one of 32 bytes per nonzero and side, against five to
// seven of 8). A check with the host's part, fp64: 10k rows 87 -> 33 us, 100k 157 -> 71, 1M 560 -> 389.
// kkt_general's terms of one row and of one column (EpiKktRows, EpiKktCols).
struct KktTerms {
  double *rp2, *d, *rd2, *p;  // rows at [0, m), columns at [m, m + n)
};
__device__ __forceinline__ void kkt_row(const KktTerms& t, int k, double ax, double yi, double lo, double up, double& pmax,
                                        double& dmax) {
  const double out = ax < lo ? lo - ax : (ax > up ? ax - up : 0.0);
  t.rp2[k] = out * out;
  pmax = elem_viol(ax, lo, up);
  double d = 0.0, rd = 0.0;
  dmax = 0.0;
  if (yi > 0) {
    if (isfinite(lo)) d = yi * lo;
    else rd = yi * yi, dmax = yi;
  } else if (yi < 0) {
    if (isfinite(up)) d = yi * up;
    else rd = yi * yi, dmax = -yi;
  }
  t.d[k] = d;
  t.rd2[k] = rd;
}
__device__ __forceinline__ void kkt_col(const KktTerms& t, long long at, double aty, double cj, double x, double lo, double up,
                                        double& pmax, double& dmax) {
  t.p[at] = cj * x;
  pmax = elem_viol(x, lo, up);
  const double lam = cj - aty;
  double z;
  if (isfinite(lo) && isfinite(up)) z = lam;
  else if (isfinite(lo)) z = std_max(lam, 0.0);
  else if (isfinite(up)) z = std_min(lam, 0.0);
  else z = 0.0;
  t.rd2[at] = (lam - z) * (lam - z);
  dmax = fabs(lam - z);
  t.d[at] = z > 0 ? z * lo : (z < 0 ? z * up : 0.0);
}
template <class T>
struct CheckVecs {
  int n, m;
  const T *xb, *xh, *x0, *yb, *yh, *y0;
  const double *col_scale, *row_scale;
  double bound_scale, obj_scale, sense;
  const double *c, *cl, *cu, *rl, *ru;
  double4 *X, *Y;
  double *t_px, *t_dxn, *t_py, *t_cross, *t_dyn;  // residual and restart distances
  KktTerms kkt;
  double *r_obj, *r_mag, *r_cd, *r_cmag;          // rays
  double *q_obj, *q_mag, *q_cd, *q_cmag;          // drift rays
  double* res;
};
__device__ __forceinline__ double ray_dual(double v, double lo, double up) {  // engine.cpp:88-96
  if (!isfinite(lo)) v = std_min(v, 0.0);
  if (!isfinite(up)) v = std_max(v, 0.0);
  return v;
}
__device__ __forceinline__ double ray_primal(double v, double lo, double up) {  // engine.cpp:130-137
  if (isfinite(lo)) v = std_max(v, 0.0);
  if (isfinite(up)) v = std_min(v, 0.0);
  return v;
}
template <class T, int kRays>
static __global__ void __launch_bounds__(kBlock) k_check_points(const __grid_constant__ CheckVecs<T> v, int col_blocks) {
  const bool cols = static_cast<int>(blockIdx.x) < col_blocks;
  const int k = (static_cast<int>(blockIdx.x) - (cols ? 0 : col_blocks)) * kBlock + static_cast<int>(threadIdx.x);
  double mx = 0.0, mx2 = 0.0;
  if (cols) {
    if (k < v.n) {
      const T xh = v.xh[k], x0 = v.x0[k];
      const T d = static_cast<T>(-1.0) * xh + static_cast<T>(1.0) * v.xb[k];
      const double e = static_cast<double>(xh) - static_cast<double>(x0), dd = static_cast<double>(d);
      const double sc = v.col_scale[k], lo = v.cl[k], up = v.cu[k];
      double4 X;
      X.x = std_min(std_max(sc * static_cast<double>(xh) / v.bound_scale, lo), up);
      X.y = dd, X.z = X.w = 0.0;
      v.t_px[k] = dd * dd;
      v.t_dxn[k] = e * e;
      if constexpr (kRays >= 1) {
        X.z = ray_primal(sc * dd / v.bound_scale, lo, up);
        mx = fabs(X.z);
      }
      if constexpr (kRays == 2) {
        const T g = static_cast<T>(-1.0) * x0 + static_cast<T>(1.0) * xh;
        X.w = ray_primal(sc * static_cast<double>(g) / v.bound_scale, lo, up);
        mx2 = fabs(X.w);
      }
      v.X[k] = X;
    }
    if constexpr (kRays >= 1) warp_max_atomic(max_slot(v.res, kMaxDabs), mx);
    if constexpr (kRays == 2) warp_max_atomic(max_slot(v.res, kMaxDabs2), mx2);
  } else {
    if (k < v.m) {
      const T yh = v.yh[k], y0 = v.y0[k];
      const T d = static_cast<T>(-1.0) * yh + static_cast<T>(1.0) * v.yb[k];
      const double e = static_cast<double>(yh) - static_cast<double>(y0), dd = static_cast<double>(d);
      const double sc = v.row_scale[k];
      double4 Y;
      Y.x = sc * static_cast<double>(yh) / v.obj_scale;
      Y.y = Y.z = 0.0, Y.w = 0.0;
      v.t_py[k] = dd * dd;
      v.t_dyn[k] = e * e;
      if constexpr (kRays >= 1) {
        Y.y = ray_dual(sc * dd / v.obj_scale, v.rl[k], v.ru[k]);
        mx = fabs(Y.y);
      }
      if constexpr (kRays == 2) {
        const T g = static_cast<T>(-1.0) * y0 + static_cast<T>(1.0) * yh;
        Y.z = ray_dual(sc * static_cast<double>(g) / v.obj_scale, v.rl[k], v.ru[k]);
        mx2 = fabs(Y.z);
      }
      v.Y[k] = Y;
    }
    if constexpr (kRays >= 1) warp_max_atomic(max_slot(v.res, kMaxRmax), mx);
    if constexpr (kRays == 2) warp_max_atomic(max_slot(v.res, kMaxRmax2), mx2);
  }
}

// A packed point: its first two values, or all four.
template <bool kAll>
__device__ __forceinline__ double4 load_packed(const double4* p) {
  const double2 a = __ldg(reinterpret_cast<const double2*>(p));
  double2 b = make_double2(0.0, 0.0);
  if constexpr (kAll) b = __ldg(reinterpret_cast<const double2*>(p) + 1);
  return make_double4(a.x, a.y, b.x, b.y);
}
// A ray's row terms and violation, and its column terms and violation (engine.cpp:97-128).
__device__ __forceinline__ double ray_row(double ad, double r, double lo, double up, double& obj, double& mag) {
  double viol = 0.0;
  if (isfinite(lo)) viol = std_max(viol, -ad);
  if (isfinite(up)) viol = std_max(viol, ad);
  obj = r > 0 ? lo * r : (r < 0 ? up * r : 0.0);
  mag = fabs(obj);
  return viol;
}
__device__ __forceinline__ double ray_col(double g, double gabs, double lo, double up, double& obj, double& mag) {
  const double lam = -g;
  double viol = 0.0;
  obj = mag = 0.0;
  if (lam > 0) {
    if (isfinite(lo)) obj = lo * lam, mag = gabs * fabs(lo);
    else viol = lam;
  } else if (lam < 0) {
    if (isfinite(up)) obj = up * lam, mag = gabs * fabs(up);
    else viol = -lam;
  }
  return viol;
}
// A long row or column would hold up the check: its thread makes two trips to memory (the indices, then the
// points there) for every four entries. The check of an LP that has one (kLong) sums the long ones of a warp's
// rows with the whole warp, one after the other, where their entries together are fewer than kCheckShare times
// the longest's. (A thread takes 0.2 us an entry, so 25 us for 128, no more than a check's launches; the warp 0.01,
// so that 16 rows one after the other are still quicker than one by its thread.) Ten checks and the first residuals of
// their cycles, ms, without / with: 60k rows of 6 and one of 4,000 entries 7.5 / 2.8, of 60,000 99 / 28; a column of
// 60,000 54 / 6.7; 300k rows and one of 300,000 665 / 136. The kernel for LPs without is as it was.
constexpr int kCheckLong = 128, kCheckShare = 16;
constexpr int kCheckChunk = 64, kCheckPitch = kCheckChunk + 2;  // entries at a time; of a buffer (free of bank conflicts)
inline bool check_is_long(int longest) { return longest > kCheckLong; }
// The lanes whose rows, of len entries each, the warp sums.
__device__ __forceinline__ unsigned check_together(int len) {
  const bool is = len > kCheckLong;
  const long long longest = __reduce_max_sync(kFull, is ? len : 0);
  return static_cast<long long>(__reduce_add_sync(kFull, is ? len : 0)) < kCheckShare * longest ? __ballot_sync(kFull, is) : 0u;
}
// The sums of a long row, entries [b, e) with their indices at idx, by a whole warp: the lanes form kCheckChunk
// entries' products (load: what those of an entry need; mul: the kSums products of it) while the next ones are
// on their way, and a lane for each sum adds them in storage order. Lane k < kSums returns the k-th sum, lane kSums + k
// the sum of the (k + 1)-th products' absolute values. sh: kSums buffers of kCheckPitch.
template <int kSums, int kAbs, class Load, class Mul>
__device__ __forceinline__ double check_long(int b, int e, const int* __restrict__ idx, double* sh, const Load& load,
                                             const Mul& mul) {
  constexpr int Q = kCheckChunk / 32;
  const int lane = static_cast<int>(threadIdx.x) & 31;
  const bool magnitude = lane >= kSums;
  const double* mine = sh + (lane < kSums ? lane : lane < kSums + kAbs ? lane - kSums + 1 : 0) * kCheckPitch;
  const auto place = [&](unsigned k, int q) {
    return static_cast<int>(min(k + static_cast<unsigned>(32 * q + lane), static_cast<unsigned>(e - 1)));
  };
  int at[Q];
  decltype(load(0, 0)) in[Q];
#pragma unroll
  for (int q = 0; q < Q; ++q) at[q] = idx[place(b, q)];
#pragma unroll
  for (int q = 0; q < Q; ++q) in[q] = load(place(b, q), at[q]), at[q] = idx[place(static_cast<unsigned>(b) + kCheckChunk, q)];
  double s = 0.0;
  const auto add = [&](int k) { s += magnitude ? fabs(mine[k]) : mine[k]; };
  const unsigned end = static_cast<unsigned>(e);
  for (unsigned k = static_cast<unsigned>(b); k < end; k += kCheckChunk) {
    __syncwarp();  // the chunk before has been added
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      double prod[kSums];
      mul(in[q], prod);
#pragma unroll
      for (int t = 0; t < kSums; ++t) sh[t * kCheckPitch + 32 * q + lane] = prod[t];
    }
    __syncwarp();
    if (k + kCheckChunk < end) {
#pragma unroll
      for (int q = 0; q < Q; ++q) in[q] = load(place(k + kCheckChunk, q), at[q]);
#pragma unroll
      for (int q = 0; q < Q; ++q) at[q] = idx[place(k + 2 * kCheckChunk, q)];
#pragma unroll 16
      for (int i = 0; i < kCheckChunk; ++i) add(i);
    } else {
      for (int i = 0; i < static_cast<int>(end - k); ++i) add(i);
    }
  }
  return s;
}
// Rows of A (blocks [0, row_blocks)): original values a0 and scaled values as on one index list; columns
// (the blocks after them): the caller's CSC.
template <class T, int kRays, bool kLong>
static __global__ void __launch_bounds__(kBlock) k_check_products(const __grid_constant__ CheckVecs<T> v, int row_blocks,
                                                                  const int* __restrict__ rp, const int* __restrict__ col,
                                                                  const double* __restrict__ a0, const T* __restrict__ as,
                                                                  const int* __restrict__ cp, const int* __restrict__ ri,
                                                                  const double* __restrict__ av) {
  constexpr int GB = 4;  // entries whose gathers are in flight together
  __shared__ double sh_long[kLong ? kBlock / 32 : 1][kLong ? (kRays + 2) * kCheckPitch : 1];
  const bool rows = static_cast<int>(blockIdx.x) < row_blocks;
  const int k = (static_cast<int>(blockIdx.x) - (rows ? 0 : row_blocks)) * kBlock + static_cast<int>(threadIdx.x);
  const int lane = static_cast<int>(threadIdx.x) & 31;
  double* sh = sh_long[kLong ? threadIdx.x >> 5 : 0];
  const bool mine = k < (rows ? v.m : v.n);
  const int* __restrict__ ptr = rows ? rp : cp;
  const int b = mine ? ptr[k] : 0, all = mine ? ptr[k + 1] : 0;
  const unsigned together = kLong ? check_together(all - b) : 0u;
  const int e = kLong && ((together >> lane) & 1u) ? b : all;  // the thread's own walk
  double pmax = 0.0, dmax = 0.0, viol = 0.0, viol2 = 0.0;
  if (rows) {
    double ax = 0.0, adx = 0.0, ad = 0.0, ad2 = 0.0;
    for (int p = b; p < e; p += GB) {
      double4 g[GB];
      double w[GB], ws[GB];
#pragma unroll
      for (int q = 0; q < GB; ++q) {
        const int at = p + q < e ? p + q : p;
        g[q] = load_packed<(kRays >= 1)>(v.X + col[at]);
        w[q] = a0[at], ws[q] = static_cast<double>(as[at]);
      }
#pragma unroll
      for (int q = 0; q < GB; ++q)
        if (p + q < e) {  // each sum in CSR order
          ax += w[q] * g[q].x;
          adx += ws[q] * g[q].y;
          if constexpr (kRays >= 1) ad += w[q] * g[q].z;
          if constexpr (kRays == 2) ad2 += w[q] * g[q].w;
        }
    }
    if constexpr (kLong) {
      struct In {
        double4 g;
        double w, ws;
      };
      for (unsigned left = together; left != 0; left &= left - 1) {
        const int who = __ffs(left) - 1;
        const double s = check_long<kRays + 2, 0>(
            __shfl_sync(kFull, b, who), __shfl_sync(kFull, all, who), col, sh,
            [&](int p, int at) { return In{load_packed<(kRays >= 1)>(v.X + at), a0[p], static_cast<double>(as[p])}; },
            [&](const In& in, double* prod) {
              prod[0] = in.w * in.g.x, prod[1] = in.ws * in.g.y;
              if constexpr (kRays >= 1) prod[2] = in.w * in.g.z;
              if constexpr (kRays == 2) prod[3] = in.w * in.g.w;
            });
        const double s0 = __shfl_sync(kFull, s, 0), s1 = __shfl_sync(kFull, s, 1), s2 = __shfl_sync(kFull, s, 2),
                     s3 = __shfl_sync(kFull, s, 3);
        if (lane == who) ax = s0, adx = s1, ad = s2, ad2 = s3;
      }
    }
    if (mine) {
      const double lo = v.rl[k], up = v.ru[k];
      const double4 Y = v.Y[k];
      const T dy = static_cast<T>(-1.0) * v.yh[k] + static_cast<T>(1.0) * v.yb[k];
      v.t_cross[k] = static_cast<double>(dy) * static_cast<double>(static_cast<T>(adx));
      kkt_row(v.kkt, k, ax, Y.x, lo, up, pmax, dmax);
      if constexpr (kRays >= 1) {
        double obj, mag;
        viol = ray_row(ad, Y.y, lo, up, obj, mag);
        v.r_obj[k] = obj, v.r_mag[k] = mag;
        if constexpr (kRays == 2) {
          viol2 = ray_row(ad2, Y.z, lo, up, obj, mag);
          v.q_obj[k] = obj, v.q_mag[k] = mag;
        }
      }
    }
    if constexpr (kRays >= 1) warp_max_atomic(max_slot(v.res, kMaxPviol), viol);
    if constexpr (kRays == 2) warp_max_atomic(max_slot(v.res, kMaxPviol2), viol2);
  } else {
    double aty = 0.0, gr = 0.0, ga = 0.0, gr2 = 0.0, ga2 = 0.0;
    for (int p = b; p < e; p += GB) {
      double4 g[GB];
      double w[GB];
#pragma unroll
      for (int q = 0; q < GB; ++q) {
        const int at = p + q < e ? p + q : p;
        g[q] = load_packed<kRays == 2>(v.Y + ri[at]);
        w[q] = av[at];
      }
#pragma unroll
      for (int q = 0; q < GB; ++q)
        if (p + q < e) {
          aty += w[q] * g[q].x;
          if constexpr (kRays >= 1) {
            const double t = w[q] * g[q].y;
            gr += t, ga += fabs(t);
          }
          if constexpr (kRays == 2) {
            const double t = w[q] * g[q].z;
            gr2 += t, ga2 += fabs(t);
          }
        }
    }
    if constexpr (kLong) {
      struct In {
        double4 g;
        double w;
      };
      for (unsigned left = together; left != 0; left &= left - 1) {
        const int who = __ffs(left) - 1;
        constexpr int S = kRays + 1;
        const double s = check_long<S, kRays>(
            __shfl_sync(kFull, b, who), __shfl_sync(kFull, all, who), ri, sh,
            [&](int p, int at) { return In{load_packed<kRays == 2>(v.Y + at), av[p]}; },
            [&](const In& in, double* prod) {
              prod[0] = in.w * in.g.x;
              if constexpr (kRays >= 1) prod[1] = in.w * in.g.y;
              if constexpr (kRays == 2) prod[2] = in.w * in.g.z;
            });
        const double s0 = __shfl_sync(kFull, s, 0), s1 = __shfl_sync(kFull, s, 1), a1 = __shfl_sync(kFull, s, S),
                     s2 = __shfl_sync(kFull, s, 2), a2 = __shfl_sync(kFull, s, S + 1);
        if (lane == who) aty = s0, gr = s1, ga = a1, gr2 = s2, ga2 = a2;
      }
    }
    if (mine) {
      const double lo = v.cl[k], up = v.cu[k], c = v.c[k];
      const double4 X = v.X[k];
      const long long at = static_cast<long long>(v.m) + k;
      kkt_col(v.kkt, at, aty, v.sense * c, X.x, lo, up, pmax, dmax);
      if constexpr (kRays >= 1) {
        double obj, mag;
        viol = ray_col(gr, ga, lo, up, obj, mag);
        v.r_obj[at] = obj, v.r_mag[at] = mag;
        v.r_cd[k] = v.sense * c * X.z;
        v.r_cmag[k] = fabs(c * X.z);
        if constexpr (kRays == 2) {
          viol2 = ray_col(gr2, ga2, lo, up, obj, mag);
          v.q_obj[at] = obj, v.q_mag[at] = mag;
          v.q_cd[k] = v.sense * c * X.w;
          v.q_cmag[k] = fabs(c * X.w);
        }
      }
    }
    if constexpr (kRays >= 1) warp_max_atomic(max_slot(v.res, kMaxDviol), viol);
    if constexpr (kRays == 2) warp_max_atomic(max_slot(v.res, kMaxDviol2), viol2);
  }
  warp_max_atomic(max_slot(v.res, kMaxPmax), pmax);
  warp_max_atomic(max_slot(v.res, kMaxDmax), dmax);
}
template <class T>
struct PdlpVecs {
  int n, m;
  const T *xc, *xa, *xp, *x0, *yc, *ya, *yp, *y0;  // current, average, the step before, the restart anchor
  const double *col_scale, *row_scale;
  double bound_scale, obj_scale, sense;
  const double *c, *cl, *cu, *rl, *ru;
  double4 *X, *Y;
  KktTerms cur, avg;
  double *r_obj, *r_mag, *r_cd, *r_cmag;  // rays
  double *q_obj, *q_mag, *q_cd, *q_cmag;  // drift rays
  double *res, *res_cur;                  // results: of the average and the rays, of the current point
};
template <class T, int kRays>
static __global__ void __launch_bounds__(kBlock) k_pdlp_points(const __grid_constant__ PdlpVecs<T> v, int col_blocks) {
  const bool cols = static_cast<int>(blockIdx.x) < col_blocks;
  const int k = (static_cast<int>(blockIdx.x) - (cols ? 0 : col_blocks)) * kBlock + static_cast<int>(threadIdx.x);
  double mx = 0.0, mx2 = 0.0;
  if (cols) {
    if (k < v.n) {
      const T x = v.xc[k];
      const double sc = v.col_scale[k], lo = v.cl[k], up = v.cu[k];
      double4 X;
      X.x = std_min(std_max(sc * static_cast<double>(x) / v.bound_scale, lo), up);
      X.y = std_min(std_max(sc * static_cast<double>(v.xa[k]) / v.bound_scale, lo), up);
      X.z = X.w = 0.0;
      if constexpr (kRays >= 1) {  // Δ = z_k − z_{k−1}: axpby(1, x, −1, x_prev) (pdlp.cpp:83-85)
        const T d = static_cast<T>(1.0) * x + static_cast<T>(-1.0) * v.xp[k];
        X.z = ray_primal(sc * static_cast<double>(d) / v.bound_scale, lo, up);
        mx = fabs(X.z);
      }
      if constexpr (kRays == 2) {  // the drift z − z0: copy + axpby(−1, x0, 1, ·) (pdlp.cpp:89-93)
        const T d = static_cast<T>(-1.0) * v.x0[k] + static_cast<T>(1.0) * x;
        X.w = ray_primal(sc * static_cast<double>(d) / v.bound_scale, lo, up);
        mx2 = fabs(X.w);
      }
      v.X[k] = X;
    }
    if constexpr (kRays >= 1) warp_max_atomic(max_slot(v.res, kMaxDabs), mx);
    if constexpr (kRays == 2) warp_max_atomic(max_slot(v.res, kMaxDabs2), mx2);
  } else {
    if (k < v.m) {
      const T y = v.yc[k];
      const double sc = v.row_scale[k];
      double4 Y;
      Y.x = sc * static_cast<double>(y) / v.obj_scale;
      Y.y = sc * static_cast<double>(v.ya[k]) / v.obj_scale;
      Y.z = Y.w = 0.0;
      if constexpr (kRays >= 1) {
        const T d = static_cast<T>(1.0) * y + static_cast<T>(-1.0) * v.yp[k];
        Y.z = ray_dual(sc * static_cast<double>(d) / v.obj_scale, v.rl[k], v.ru[k]);
        mx = fabs(Y.z);
      }
      if constexpr (kRays == 2) {
        const T d = static_cast<T>(-1.0) * v.y0[k] + static_cast<T>(1.0) * y;
        Y.w = ray_dual(sc * static_cast<double>(d) / v.obj_scale, v.rl[k], v.ru[k]);
        mx2 = fabs(Y.w);
      }
      v.Y[k] = Y;
    }
    if constexpr (kRays >= 1) warp_max_atomic(max_slot(v.res, kMaxRmax), mx);
    if constexpr (kRays == 2) warp_max_atomic(max_slot(v.res, kMaxRmax2), mx2);
  }
}
template <class T, int kRays>
static __global__ void __launch_bounds__(kBlock) k_pdlp_products(const __grid_constant__ PdlpVecs<T> v, int row_blocks,
                                                                 const int* __restrict__ rp, const int* __restrict__ col,
                                                                 const double* __restrict__ a0, const int* __restrict__ cp,
                                                                 const int* __restrict__ ri, const double* __restrict__ av) {
  constexpr int GB = 4;
  const bool rows = static_cast<int>(blockIdx.x) < row_blocks;
  const int k = (static_cast<int>(blockIdx.x) - (rows ? 0 : row_blocks)) * kBlock + static_cast<int>(threadIdx.x);
  const bool mine = k < (rows ? v.m : v.n);
  const int* __restrict__ ptr = rows ? rp : cp;
  const int* __restrict__ idx = rows ? col : ri;
  const double* __restrict__ val = rows ? a0 : av;
  const double4* from = rows ? v.X : v.Y;
  double sx = 0.0, sy = 0.0, sz = 0.0, sw = 0.0, tz = 0.0, tw = 0.0;  // the four sums, and Σ|·| of the rays'
  const int b = mine ? ptr[k] : 0, e = mine ? ptr[k + 1] : 0;
  for (int p = b; p < e; p += GB) {
    double4 g[GB];
    double w[GB];
#pragma unroll
    for (int q = 0; q < GB; ++q) {
      const int at = p + q < e ? p + q : p;
      g[q] = load_packed<(kRays >= 1)>(from + idx[at]);
      w[q] = val[at];
    }
#pragma unroll
    for (int q = 0; q < GB; ++q)
      if (p + q < e) {  // each sum in storage order
        sx += w[q] * g[q].x;
        sy += w[q] * g[q].y;
        if constexpr (kRays >= 1) {
          const double t = w[q] * g[q].z;
          sz += t, tz += fabs(t);
        }
        if constexpr (kRays == 2) {
          const double t = w[q] * g[q].w;
          sw += t, tw += fabs(t);
        }
      }
  }
  double pc = 0.0, dc = 0.0, pa = 0.0, da = 0.0, viol = 0.0, viol2 = 0.0;
  if (mine && rows) {
    const double lo = v.rl[k], up = v.ru[k];
    const double4 Y = v.Y[k];
    kkt_row(v.cur, k, sx, Y.x, lo, up, pc, dc);
    kkt_row(v.avg, k, sy, Y.y, lo, up, pa, da);
    double obj, mag;
    if constexpr (kRays >= 1) viol = ray_row(sz, Y.z, lo, up, obj, mag), v.r_obj[k] = obj, v.r_mag[k] = mag;
    if constexpr (kRays == 2) viol2 = ray_row(sw, Y.w, lo, up, obj, mag), v.q_obj[k] = obj, v.q_mag[k] = mag;
  } else if (mine) {
    const double lo = v.cl[k], up = v.cu[k], c = v.c[k];
    const double4 X = v.X[k];
    const long long at = static_cast<long long>(v.m) + k;
    kkt_col(v.cur, at, sx, v.sense * c, X.x, lo, up, pc, dc);
    kkt_col(v.avg, at, sy, v.sense * c, X.y, lo, up, pa, da);
    double obj, mag;
    if constexpr (kRays >= 1) {
      viol = ray_col(sz, tz, lo, up, obj, mag), v.r_obj[at] = obj, v.r_mag[at] = mag;
      v.r_cd[k] = v.sense * c * X.z, v.r_cmag[k] = fabs(c * X.z);
    }
    if constexpr (kRays == 2) {
      viol2 = ray_col(sw, tw, lo, up, obj, mag), v.q_obj[at] = obj, v.q_mag[at] = mag;
      v.q_cd[k] = v.sense * c * X.w, v.q_cmag[k] = fabs(c * X.w);
    }
  }
  if constexpr (kRays >= 1) warp_max_atomic(max_slot(v.res, rows ? kMaxPviol : kMaxDviol), viol);
  if constexpr (kRays == 2) warp_max_atomic(max_slot(v.res, rows ? kMaxPviol2 : kMaxDviol2), viol2);
  warp_max_atomic(max_slot(v.res_cur, kMaxPmax), pc);
  warp_max_atomic(max_slot(v.res_cur, kMaxDmax), dc);
  warp_max_atomic(max_slot(v.res, kMaxPmax), pa);
  warp_max_atomic(max_slot(v.res, kMaxDmax), da);
}

// The results go to the host's pinned block, and the maxima back to zero for the next check. (PDLP: a second
// set, in the second block of threads.)
static __global__ void k_check_publish(double* res, double* host, double* res2, double* host2) {
  const int k = threadIdx.x;
  if (k >= kNumSlots) return;
  double* r = blockIdx.x ? res2 : res;
  (blockIdx.x ? host2 : host)[k] = r[k];
  if (k >= kMaxPmax) r[k] = 0.0;
}
// One packed component as a vector (an infeasibility ray).
static __global__ void k_unpack(int len, const double4* P, int which, double* out) {
  B200_FOR(i, len) out[i] = which == 0 ? P[i].x : which == 1 ? P[i].y : which == 2 ? P[i].z : P[i].w;
}

// ---------------------------------------------------------------------- finish
// y = sense · y_min; z_j = c_j − Σ a_ij y_i with the subtractions in CSC order (engine.cpp:283-286)
static __global__ void k_dual_out(int m, double sense, const double* ymin, double* y) {
  B200_FOR(i, m) y[i] = sense * ymin[i];
}
static __global__ void k_reduced_costs(int n, const int* cp, const int* ri, const double* v, const double* c,
                                const double* y, double* z) {
  B200_FOR(j, n) {
    double zz = c[j];
    for (int k = cp[j]; k < cp[j + 1]; ++k) zz -= v[k] * y[ri[k]];
    z[j] = zz;
  }
}
static __global__ void k_obj_terms(int n, const double* c, const double* x, double* t) {
  B200_FOR(j, n) t[j] = c[j] * x[j];
}

// In-process check (solution_checker.cpp:61-133) on the device, for the device-resident path.
__device__ __forceinline__ double bound_violation(double val, double lo, double up) {
  double v = 0.0;
  if (lo != -INFINITY) v = std_max(v, (lo - val) / (1.0 + fabs(lo)));
  if (up != INFINITY) v = std_max(v, (val - up) / (1.0 + fabs(up)));
  return v;
}
__device__ __forceinline__ void multiplier(double mult, double lo, double up, double& viol, double& contrib) {
  viol = 0.0, contrib = 0.0;
  if (mult > 0.0) {
    if (lo == -INFINITY) viol = mult;
    else contrib = mult * lo;
  } else if (mult < 0.0) {
    if (up == INFINITY) viol = -mult;
    else contrib = mult * up;
  }
}
struct EpiCheckRows : AlwaysActive {  // after ax = A·x; y = min-form duals (sense · reported y)
  const double *y, *rl, *ru;
  double c_scale;
  double* t_dual;  // [0, m) rows, [m, m+n) cols
  double* res;
  struct Acc {
    double primal = 0.0, dual = 0.0;
  };
  __device__ void operator()(int i, double ax, Acc& acc) const {
    acc.primal = bound_violation(ax, rl[i], ru[i]);
    double viol, contrib;
    multiplier(y[i], rl[i], ru[i], viol, contrib);
    acc.dual = viol / c_scale;
    t_dual[i] = contrib;
  }
  __device__ void flush(const Acc& a) const {
    warp_max_atomic(max_slot(res, kMaxChkPrimal), a.primal);
    warp_max_atomic(max_slot(res, kMaxChkDual), a.dual);
  }
};
struct EpiCheckCols : AlwaysActive {  // after aty = Aᵀ·y_min (CSC order)
  const double *x, *c, *cl, *cu;
  double sense, c_scale;
  int m;
  double *t_dual, *t_primal;
  double* res;
  struct Acc {
    double primal = 0.0, dual = 0.0;
  };
  __device__ void operator()(int j, double aty, Acc& acc) const {
    acc.primal = bound_violation(x[j], cl[j], cu[j]);
    const double cj = sense * c[j];
    const double d = cj - aty;
    double viol, contrib;
    multiplier(d, cl[j], cu[j], viol, contrib);
    acc.dual = viol / c_scale;
    t_dual[m + j] = contrib;
    t_primal[j] = cj * x[j];
  }
  __device__ void flush(const Acc& a) const {
    warp_max_atomic(max_slot(res, kMaxChkPrimal), a.primal);
    warp_max_atomic(max_slot(res, kMaxChkDual), a.dual);
  }
};
static __global__ void k_scale_copy(long long n, const double* src, double s, double* dst) {
  B200_FOR(i, n) dst[i] = s * src[i];
}

// ---------------------------------------------------------------------- vector helpers
template <class T>
static __global__ void k_fill(long long n, T* v, T a) {
  B200_FOR(i, n) v[i] = a;
}
template <class T>
static __global__ void k_axpby(long long n, T a, const T* x, T b, T* y) {
  B200_FOR(i, n) y[i] = a * x[i] + b * y[i];
}
// x = proj_[l,u](0 − 0·(c − 0)), the reference's primal_step(dx=0, aty=0, τ=0) start point
template <class T>
static __global__ void k_init_x(int n, const T* c, const T* l, const T* u, T* x) {
  B200_FOR(j, n) {
    const T zero = static_cast<T>(0.0);
    x[j] = ref_clamp<T>(zero - zero * (c[j] - zero), l[j], u[j]);
  }
}
// restart at T(z): x = x0 = x̂, y = y0 = ŷ (r2hpdhg.cpp:155-158)
template <class T>
static __global__ void k_restart(int n, int m, const T* xh, T* x, T* x0, const T* yh, T* y, T* y0) {
  B200_FOR(i, (n > m ? n : m)) {
    if (i < n) x[i] = xh[i], x0[i] = xh[i];
    if (i < m) y[i] = yh[i], y0[i] = yh[i];
  }
}

}  // namespace b200
