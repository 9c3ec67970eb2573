// FP64 Lopez-Sancho decimation with its products on the 5th-generation tensor
// cores (Ndim FP64_SPLIT_MIN_N .. FP64_SPLIT_MAX_N; other sizes run in
// wtg_decimate.cu).
//
// GB300 issues two FP64 FMAs a clock per SM: the FP64 pipe at 91-95 % was the
// bound of the whole form, 20 M cycles an iteration at Ndim 112.  Here every
// complex product of surfgreen_1985 (src/surfgreen.f90:92-116, zgemm at
// src/mat_mul.f90:23) is an exactly split product (split_gemm of wtg_split.cuh
// with DigF8 digits): 55-bit operands against a shared exponent per row /
// column, seven base-256 digits, the slice orders 2..9 in one exact integer
// accumulator each.  Its error is the operands' rounding against their row's or
// column's maximum, real and imaginary parts together: below an FP64 product's,
// whose partial sums round K times, where the terms reach those maxima (against
// exact products of normal random complex matrices 3-6 times smaller at Ndim
// 40..320), above it for operands graded along k and for imaginary parts far below
// the real ones.  Points of that kind run on the FP64 pipe (split_suits).
//
// Inverses (zgesv with identity, src/inverse.f90:43-55): an FP32 Gauss-Jordan
// with partial pivoting gives a starting point, and Newton-Schulz steps
// X <- X + X (I - M X) with the residual as a split product are taken until
// |I - M X|_F <= 1e-8 before a step, so that the step leaves its square, below
// the residual's own rounding: an FP64 inverse with a right residual as small
// as a pivoted elimination's.  Where the residual does not get there (condition
// beyond ~1e7, an FP32 zero pivot, infinities), the FP64 Gauss-Jordan of the
// plain form runs instead, with its singular flag.
#include <mutex>

#include "../../include/wtgpu.h"
#include "wtg_common.cuh"

namespace wtg {

namespace {

#include "wtg_fp64_dev.cuh"
#include "wtg_split.cuh"
#include "wtg_split_inverse.cuh"
#include "wtg_fp64_solve.cuh"
#include "wtg_small_dev.cuh"

// Whether a point may run on split products: operands rounded against their row's or
// column's maximum (2^-55 of it, for real and imaginary parts together) lose what an
// FP64 product keeps
//   - where orbitals have very different scales (M = w - H00 and H01): an inner index of
//     the products then joins large columns to small rows;
//   - where eta is very small: off the bands the imaginary parts, which the spectral sums
//     read, are about eta / |M| of the real ones.
// The largest elements of the orbitals' rows and columns have to lie within a factor of
// 2^6 and eta within 2^20 of the largest of all.  Relative errors of the sums, split
// against FP64 arithmetic (emulated, Ndim 27..40, against 64-bit mantissas): scales within
// 2^5 median 1e-13 and 1e-13, at 2^6 at most 3.4e-12 and 5.7e-12, at 2^9 4e-12 (worst
// 6e-11) and 2e-13, on-site 1e12 beside hopping 1e6 5e-8 and 4e-13; energies 20 eV off the
// bands at eta 1e-3 eV (2^-15) 3e-13 and 1e-14, 1e-6 eV 2e-10 and 1e-11, 1e-10 eV 5e-6 and
// 1e-7 (a real H keeps 1e-16 in FP64).  One pass over H00 and H01 that also makes alpha's
// exponents (as exps_of); E and Al are workspace matrices 0 and 3; all threads.
__device__ __noinline__ bool split_suits(const double2* __restrict__ W, double2 w, int N, MxShared s) {
  constexpr int Al = 3;
  const double2* const A = W + (size_t)Al * N * N;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int* const top = s.t().prow;                      // exponent of an orbital's largest element
  int* const er = s.rows(Al, N);
  int* const ec = s.cols(Al, N);
  for (int i = threadIdx.x; i < N; i += SP_T) {
    er[i] = EXP_MIN;
    top[i] = 0;
  }
  __syncthreads();
  constexpr int ROWS = FP64_SPLIT_MAX_N / 32;
  int amax[ROWS], tmax[ROWS];
#pragma unroll
  for (int q = 0; q < ROWS; ++q) amax[q] = tmax[q] = 0;
  for (int j = warp; j < N; j += SP_T / 32) {
    int ca = EXP_MIN, ct = 0;
#pragma unroll
    for (int q = 0; q < ROWS; ++q) {
      const int i = lane + 32 * q;
      if (i < N) {
        const double2 a = A[i + (size_t)j * N];
        double2 m = W[i + (size_t)j * N];
        if (i == j) m = make_double2(w.x - m.x, w.y - m.y);
        const int ea = max(bexp(a.x), bexp(a.y)), et = max(ea, max(bexp(m.x), bexp(m.y)));
        amax[q] = max(amax[q], ea);
        tmax[q] = max(tmax[q], et);
        ca = max(ca, ea);
        ct = max(ct, et);
      }
    }
    ca = __reduce_max_sync(0xffffffffu, ca);
    ct = __reduce_max_sync(0xffffffffu, ct);
    if (lane == 0) {
      ec[j] = ca;
      atomicMax(&top[j], ct);
    }
  }
#pragma unroll
  for (int q = 0; q < ROWS; ++q) {
    const int i = lane + 32 * q;
    if (i < N) {
      atomicMax(&er[i], amax[q]);
      atomicMax(&top[i], tmax[q]);
    }
  }
  __syncthreads();
  int hi = 0, lo = 2047;
  for (int i = lane; i < N; i += 32) {
    hi = max(hi, top[i]);
    lo = min(lo, top[i]);
  }
  hi = __reduce_max_sync(0xffffffffu, hi);
  lo = __reduce_min_sync(0xffffffffu, lo);
  __syncthreads();
  // (infinities and NaN: no form has a result)
  return hi == 2047 || (hi - lo <= 6 && hi - bexp(w.y) <= 20);
}

// a point on the FP64 pipe in the shared memory of the split products
template <class O, class Emit>
__device__ __forceinline__ void pipe_solve(int N, double2 w, const O& o, double2* gll, double2* grr,
                                           double2* gb, double2* W, int gi, Emit emit) {
  constexpr int KC = 16;
  if (N <= MX_SMEM_GJ_N && !gi)
    fp64_solve<13, false>(N, KC, w, o, gll, grr, gb, W, fp64_layout(MxShared::base(), N, KC, true), emit);
  else
    fp64_solve<13, true>(N, KC, w, o, gll, grr, gb, W, fp64_layout(MxShared::base(), N, KC, false), emit);
}

// Decimation of one instance whose eps, eps_s, eps_t (= H00), alpha (= H01, with
// its exponents) and beta (= H01^dagger) already sit in workspace matrices 0..4 of
// W (11 N x N matrices), as fp64_solve; all threads.
template <class O, class Emit>
__device__ __forceinline__ void s64_solve(const MxPlan& pl, double2 w, const O& o, double2* gll,
                                          double2* grr, double2* gb, double2* W, int gi,
                                          const MxShared s, Emit emit) {
  const int N = pl.N, NN = N * N, tid = threadIdx.x;
  int Al = 3, Be = 4, G = 5, R = 9, Gn = 10;          // workspace matrices by index
  constexpr int iE = 0, iES = 1, iET = 2, M1 = 6, M2 = 7, iMi = 8;
  int stat = 0, it = 0;
  bool conv = false;
  split_tables<F8x7, F8x4>(pl, s);
  exps_dagger(Be, Al, N, s);
  for (int itc = 1; itc <= o.itermax && !s.t().abort; ++itc) {   // src/surfgreen.f90:86-122
    it = itc;
    if (s64_inverse(iE, w, W, pl, G, Gn, iMi, R, Al, Be, gi, s)) stat |= PT_SINGULAR;
    // the six products (:92-116), row-stacked where that takes fewer 128-row
    // tiles; eps still receives M1 beta before M2 alpha
    float part;
    if ((2 * N + 127) / 128 < 2 * ((N + 127) / 128)) {
      f8_gemm7(W, ops(Al, G, M1, 0, Be, M2), OZ_STORE, OZ_STORE, pl, s);               // :92, :95
      f8_gemm7(W, ops(M1, Be, iE, iES, M2, R), OZ_ADD2, OZ_STORE, pl, s);              // :98-102, :116
      part = f8_gemm7(W, ops(M1, Al, Gn, 0, M2, iE, iET), OZ_STORE_NORM, OZ_ADD2, pl, s);  // :113, :107-110
    } else {
      f8_gemm7(W, ops(Al, G, M1), OZ_STORE, -1, pl, s);                                // :92
      f8_gemm7(W, ops(Be, G, M2), OZ_STORE, -1, pl, s);                                // :95
      f8_gemm7(W, ops(M1, Be, iE, iES), OZ_ADD2, -1, pl, s);                           // :98-102
      part = f8_gemm7(W, ops(M1, Al, Gn), OZ_STORE_NORM, -1, pl, s);                   // :113
      f8_gemm7(W, ops(M2, Al, iE, iET), OZ_ADD2, -1, pl, s);                           // :107-110
      f8_gemm7(W, ops(M2, Be, R), OZ_STORE, -1, pl, s);                                // :116
    }
    swap_mat(Al, Gn);
    swap_mat(Be, R);
    if (converged(part, W + (size_t)Al * NN, N, o.tol, s)) {     // :120-122
      conv = true;
      break;
    }
  }
  if (!conv) stat |= PT_NOT_CONVERGED;

  double sums[9];                                   // dl, dr, db, then the six spin sums
  if (split_finals(w, W, pl, o, G, Gn, iMi, R, gll, grr, gb, gi, sums, s)) stat |= PT_SINGULAR;
  if (tid == 0) {
    if (s.t().abort) stat |= PT_TIMEOUT;
    if (!isfinite(sums[0]) || !isfinite(sums[1]) || !isfinite(sums[2])) stat |= PT_NONFINITE;
    emit(sums[0], sums[1], sums[2], sums + 3, it, stat);
  }
  __syncthreads();
}

// an instance's outputs
__device__ __forceinline__ void put_point(const DecimArgs& a, int inst, double dl, double dr, double db,
                                          const double* spin, int it, int stat) {
  const size_t oidx = (size_t)(a.k_offset + inst / a.nomega) + (size_t)(inst % a.nomega) * a.nk_total;
  a.dos_l[oidx] = dl;
  a.dos_r[oidx] = dr;
  a.dos_bulk[oidx] = db;
  if (a.spin[0])
    for (int c = 0; c < 6; ++c) a.spin[c][oidx] = spin[c];
  if (a.iters) a.iters[oidx] = it;
  if (a.status) a.status[oidx] = (uint8_t)stat;
}

// an instance that split products do not suit; a function of its own, so that the split
// path shares no registers or stack with it (inlined, a product-bound point was 0.7 % slower)
__device__ __noinline__ void pipe_point(const DecimArgs& a, int inst, double2* W, int gi) {
  const size_t NN = (size_t)a.N * a.N;
  pipe_solve(a.N, make_double2(a.omega[inst % a.nomega], a.eta), a, a.gll ? a.gll + inst * NN : nullptr,
             a.grr ? a.grr + inst * NN : nullptr, a.gb ? a.gb + inst * NN : nullptr, W, gi,
             [&](double dl, double dr, double db, const double* spin, int it, int stat) {
               put_point(a, inst, dl, dr, db, spin, it, stat);
             });
}

__global__ void __launch_bounds__(SP_T, 1) k_decimate_split64(const __grid_constant__ DecimArgs a,
                                                              int gi, unsigned spin_limit) {
  const int N = a.N, NN = N * N, T = blockDim.x, tid = threadIdx.x;
  const MxPlan pl = s64_plan(N);
  const MxShared s = mx_layout(pl.wb);
  mx_setup(s, spin_limit);
  double2* W = a.ws + (size_t)blockIdx.x * 11 * NN;
  for (;;) {
    if (tid == 0) s.t().misc[0] = atomicAdd(a.counter, 1);
    __syncthreads();
    const int inst = s.t().misc[0];
    __syncthreads();
    if (inst >= a.n_inst) break;
    const int ik = inst / a.nomega, iw = inst % a.nomega;
    if (s.t().abort) {       // a wait gave up earlier: the rest of this CTA's points are not computed
      if (tid == 0) {
        const double nan = __longlong_as_double(0x7FF8000000000000LL);
        const double spin[6] = {nan, nan, nan, nan, nan, nan};
        put_point(a, inst, nan, nan, nan, spin, 0, PT_TIMEOUT);
      }
      continue;
    }
    const double2* H00 = a.h + (size_t)ik * 2 * NN;
    const double2* H01 = H00 + NN;
    const double2 w = make_double2(a.omega[iw], a.eta);      // src/surfgreen.f90:82
    for (int e = tid; e < NN; e += T) {                       // :74-78
      const double2 h = H00[e];
      W[e] = h;
      W[NN + e] = h;
      W[2 * NN + e] = h;
      const double2 t = H01[e];
      W[3 * NN + e] = t;
      const int i = e % N, j = e / N;
      W[4 * NN + j + (size_t)i * N] = make_double2(t.x, -t.y);
    }
    __syncthreads();
    if (!split_suits(W, w, N, s)) {
      pipe_point(a, inst, W, gi);
      continue;
    }
    s64_solve(pl, w, a, a.gll ? a.gll + (size_t)inst * NN : nullptr,
              a.grr ? a.grr + (size_t)inst * NN : nullptr,
              a.gb ? a.gb + (size_t)inst * NN : nullptr, W, gi, s,
              [&](double dl, double dr, double db, const double* spin, int it, int stat) {
                put_point(a, inst, dl, dr, db, spin, it, stat);
              });
  }
  mx_teardown(s);
}

// Uneven batch (several models, eta per point) in one persistent launch, as
// k_batch_fp64 of wtg_decimate.cu: points outside the split range, or that split
// products do not suit, run on the FP64 pipe, the others as k_decimate_split64.
__global__ void __launch_bounds__(SP_T, 1) k_batch_split64(const __grid_constant__ BatchArgs a,
                                                           unsigned spin_limit) {
  extern __shared__ __align__(1024) unsigned char smem_dyn[];
  const int tid = threadIdx.x;
  const MxShared s = mx_layout(a.wb);
  mx_setup(s, spin_limit);
  double2* W = a.ws + (size_t)blockIdx.x * a.ws_stride;
  const int npts = a.run ? a.run->npts : a.npts;
  const double tol = a.run ? a.run->tol : a.tol;
  const int itermax = a.run ? a.run->itermax : a.itermax;
  const int divide_by_pi = a.run ? a.run->divide_by_pi : a.divide_by_pi;
  for (;;) {
    if (tid == 0) {
      const int q = atomicAdd(a.counter, 1);
      s.t().misc[0] = q < npts ? a.order[q] : -1;
    }
    __syncthreads();
    const int p = s.t().misc[0];
    __syncthreads();
    if (p < 0) break;
    if (s.t().abort) {                // a wait gave up earlier: not computed
      if (tid == 0) {
        const double nan = __longlong_as_double(0x7FF8000000000000LL);
        a.dos_l[p] = nan;
        a.dos_r[p] = nan;
        a.dos_bulk[p] = nan;
        if (a.iters) a.iters[p] = 0;
        if (a.status) a.status[p] = PT_TIMEOUT;
      }
      continue;
    }
    const BatchModel& m = a.models[a.pmodel[p]];
    fourier_fill(m, a.k[p], a.k[p + a.npts], W, reinterpret_cast<double2*>(smem_dyn + a.ph_off));
    SolveOpts o;
    o.nw = m.nw;
    o.tol = tol;
    o.itermax = itermax;
    o.divide_by_pi = divide_by_pi;
    o.ntop = m.ntop;
    o.nbot = m.nbot;
    o.top = m.top;
    o.bot = m.bot;
    for (int c = 0; c < 6; ++c) o.spin[c] = nullptr;
    o.spin_right_bottom = 0;
    const double2 w = make_double2(a.omega[p], a.eta[p]);
    auto emit = [&](double dl, double dr, double db, const double*, int it, int st) {
      a.dos_l[p] = dl;
      a.dos_r[p] = dr;
      a.dos_bulk[p] = db;
      if (a.iters) a.iters[p] = it;
      if (a.status) a.status[p] = (uint8_t)st;
    };
    if (m.N <= SMALL_MAX_N) {                // one warp, as k_decimate_small
      if (tid < 32) small_point(m.N, w, o, W, emit);
      __syncthreads();
    } else if (m.N < FP64_SPLIT_MIN_N || m.N > FP64_SPLIT_MAX_N || !split_suits(W, w, m.N, s)) {
      pipe_solve(m.N, w, o, nullptr, nullptr, nullptr, W, 0, emit);
    } else {
      MxPlan pl = s64_plan(m.N);
      pl.wb = a.wb;
      s64_solve(pl, w, o, nullptr, nullptr, nullptr, W, 0, s, emit);
    }
  }
  mx_teardown(s);
}

// Whether a split product X Y (workspace matrices 0 and 1 with their exponents) is as
// accurate as an FP64 one in every element.  Its operands are rounded against their
// row's (X) or column's (Y) maximum, so an element's error is K 2^-55 2^(er_i + ec_j)
// whatever its terms are, an FP64 product's K 2^-53 sum_k |x_ik y_kj|.  With operands
// graded along k (X D, D^-1 Y), or with sparse ones, the terms can lie far below the
// product of the maxima (at n = 40, scales of 1e+-4 lose 2e-10 of the product, 1e+-8
// all of it).  Required: sum_k |x_ik y_kj| >= 2^(er_i + ec_j), summed from exponents
// alone, at most 4 times too small; an element without terms is an exact zero.  (Normal
// random operands: at least 2.5 at n = 25, growing with n.)  Infinities and NaN fail:
// a split product makes NaN of their whole row or column.  All threads.
__device__ __noinline__ bool terms_reach_scales(const double2* W, int N, MxShared s) {
  const double2* const X = W;
  const double2* const Y = W + (size_t)N * N;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  bool low = false;
  for (int j = warp; j < N; j += SP_T / 32) {
    const int ec = s.cols(1, N)[j];
    for (int i = lane; i < N; i += 32) {
      const int er = s.rows(0, N)[i];
      float sum = 0.f;
      for (int k = 0; k < N; ++k) {
        const double2 x = X[i + (size_t)k * N], y = Y[k + (size_t)j * N];
        const bool none = (x.x == 0.0 && x.y == 0.0) || (y.x == 0.0 && y.y == 0.0);
        const int e = max(bexp(x.x), bexp(x.y)) - er + max(bexp(y.x), bexp(y.y)) - ec;
        if (!none) sum += __int_as_float((max(e, -100) + 127) << 23);      // e <= 0
      }
      low = low || (sum > 0.f && sum < 1.f) || max(er, ec) == 2047;
    }
  }
  return !__syncthreads_or(low);
}

// Whether the split residual I - X G (workspace matrices 0 and iG, both with their
// exponents) resolves what an inverse of X owes: its rounding, 2^-55 2^(er_i + ec_j), is
// to stay within 2^5 of the largest term x_ik g_kj a row has, taking G's largest column.
// Graded columns of X put its terms far below: scales of 1e+-2 to 1e+-3 still meet the
// residual's limit and left 1e-12 to 5e-10 in the rows of G, where an FP64 elimination
// has 1e-14.  Up to 5 bits the split inverse is the closer one (random, row-graded and
// ill-conditioned X: 0 to 2 bits).  All threads.
__device__ __noinline__ bool residual_resolves(const double2* X, int iG, int N, MxShared s) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int* const top = s.t().prow;                       // per row: exponent of its largest term
  for (int i = threadIdx.x; i < N; i += SP_T) top[i] = 0;
  __syncthreads();
  for (int k = warp; k < N; k += SP_T / 32) {
    const int eg = s.rows(iG, N)[k];
    for (int i = lane; i < N; i += 32) {
      const double2 x = X[i + (size_t)k * N];
      if (x.x != 0.0 || x.y != 0.0) atomicMax(&top[i], max(bexp(x.x), bexp(x.y)) + eg);
    }
  }
  __syncthreads();
  int ec = 0;
  for (int j = lane; j < N; j += 32) ec = max(ec, s.cols(iG, N)[j]);
  ec = __reduce_max_sync(0xffffffffu, ec);
  bool low = false;
  for (int i = threadIdx.x; i < N; i += SP_T) low = low || s.rows(0, N)[i] + ec > top[i] + 5;
  return !__syncthreads_or(low);
}

// one product (op 0) or inverse (op 1) by one CTA: W holds X, Y, the result and
// five work matrices
__global__ void __launch_bounds__(SP_T, 1) k_split64_unit(int op, int N, double2* W, int* status) {
  const MxPlan pl = s64_plan(N);
  const int NN = N * N, tid = threadIdx.x;
  const MxShared s = mx_layout(pl.wb);
  mx_setup(s, 0u);
  split_tables<F8x7, F8x4>(pl, s);
  int sing = 0;
  if (op == 0) {
    exps_of(W, 0, N, s);
    exps_of(W + NN, 1, N, s);
    if (terms_reach_scales(W, N, s)) {
      f8_gemm7(W, ops(0, 1, 2), OZ_STORE, -1, pl, s);
    } else {                                    // the FP64 pipe; its stages alias the split ones
      const Shared f = fp64_layout(MxShared::base(), N, GJ_PANEL, false);
      cta_gemm<13, EPI_STORE>(W, W + NN, N, GJ_PANEL, f.sX, f.sY, W + 2 * (size_t)NN, nullptr);
    }
  } else {
    // C = X^-1: X given directly, so pass -X with w = 0 (M = 0*I - (-X) = X)
    double2* negX = W + 7 * (size_t)NN;
    for (int e = tid; e < NN; e += blockDim.x) negX[e] = make_double2(-W[e].x, -W[e].y);
    __syncthreads();
    int G = 3, Gn = 4;
    sing = s64_inverse(7, make_double2(0.0, 0.0), W, pl, G, Gn, 6, 5, -1, -1, 0, s);
    __syncthreads();
    exps_of(W, 0, N, s);
    if (!sing && !s.t().abort && !residual_resolves(W, G, N, s))
      sing = gj64(negX, make_double2(0.0, 0.0), N, W + (size_t)G * NN, W + 6 * (size_t)NN, 0);
    double2* C = W + 2 * (size_t)NN;
    for (int e = tid; e < NN; e += blockDim.x) C[e] = W[(size_t)G * NN + e];
  }
  if (tid == 0) *status = (s.t().abort ? PT_TIMEOUT : 0) | (sing ? PT_SINGULAR : 0);
  mx_teardown(s);
}

static_assert(fp64_gi_smem_bytes(MX_MAXN) <= MX_FP64_AREA, "the FP64 pipe's stages fit the area");

size_t s64_smem(int wb) {
  // at least 116 KB so that two CTAs never share an SM (each allocates all 512 TMEM columns)
  const size_t b = split_smem(wb);
  return b > (size_t)(116 << 10) ? b : (size_t)(116 << 10);
}

}  // namespace

cudaError_t split64_config(int N, DecimConfig* cfg) {
  if (N > MX_MAXN) return cudaErrorInvalidValue;
  cfg->threads = SP_T;
  cfg->KC = 0;
  cfg->RP = 0;
  cfg->split = 1;
  cfg->smem = s64_smem(s64_plan(N).wb);
  cudaError_t e = cudaFuncSetAttribute(k_decimate_split64,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cfg->smem);
  if (e != cudaSuccess) return e;
  int occ = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_decimate_split64, SP_T, cfg->smem);
  if (e != cudaSuccess) return e;
  cfg->ctas_per_sm = occ > 1 ? 1 : occ;       // tensor memory is allocated whole (512 columns)
  return cudaSuccess;
}

cudaError_t batch_split64_config(int max_n, int* wb, DecimConfig* cfg) {
  if (max_n > MX_MAXN) return cudaErrorInvalidValue;
  int w = 8;
  for (int n = FP64_SPLIT_MIN_N; n <= max_n && n <= FP64_SPLIT_MAX_N; ++n)
    w = w > s64_plan(n).wb ? w : s64_plan(n).wb;
  *wb = w;
  cfg->threads = SP_T;
  cfg->KC = 0;
  cfg->RP = 0;
  cfg->split = 1;
  cfg->smem = s64_smem(w);
  cfg->ph_room = planes_bytes_of(w);
  cfg->ctas_per_sm = 1;
  return cudaSuccess;
}

// the batch kernel's dynamic shared-memory limit raised to the opt-in maximum
cudaError_t batch_split64_prepare() {
  int dev = 0, optin = 0;
  cudaError_t err = cudaGetDevice(&dev);
  cudaFuncAttributes fa;
  if (err == cudaSuccess)
    err = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (err == cudaSuccess) err = cudaFuncGetAttributes(&fa, k_batch_split64);
  if (err == cudaSuccess)
    err = cudaFuncSetAttribute(k_batch_split64, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               optin - (int)fa.sharedSizeBytes);
  return err;
}

cudaError_t launch_batch_split64(const BatchArgs& a, const DecimConfig& cfg, int grid,
                                 cudaStream_t s) {
  k_batch_split64<<<grid, cfg.threads, cfg.smem, s>>>(
      a, (unsigned)test_option(WTG_TEST_MIXED_SPIN_LIMIT));
  return cudaGetLastError();
}

cudaError_t launch_split64_unit(int op, int N, double2* W, int* status, cudaStream_t s) {
  const size_t smem = s64_smem(s64_plan(N).wb);
  cudaError_t e =
      cudaFuncSetAttribute(k_split64_unit, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  k_split64_unit<<<1, SP_T, smem, s>>>(op, N, W, status);
  return cudaGetLastError();
}

cudaError_t launch_split64(const DecimArgs& a, const DecimConfig& cfg, int grid, cudaStream_t s) {
  k_decimate_split64<<<grid, cfg.threads, cfg.smem, s>>>(
      a, cfg.inv_global, (unsigned)test_option(WTG_TEST_MIXED_SPIN_LIMIT));
  return cudaGetLastError();
}

}  // namespace wtg
