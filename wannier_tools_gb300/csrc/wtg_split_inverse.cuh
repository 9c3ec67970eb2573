// FP64 inverses on exactly split products, and the spectral sums of the three
// final ones: the FP64 form's split kernels and the end of the mixed form.
// Included inside an anonymous namespace after wtg_split.cuh.
#pragma once

using F8x7 = DigF8<7>;
using F8x4 = DigF8<4>;

__host__ __device__ inline MxPlan s64_plan(int N) { return split_plan(N, split_wmax<F8x7>()); }

__device__ __forceinline__ float f8_gemm7(double2* W, uint32_t op, int epi, int epi2, const MxPlan& p,
                                       const MxShared s) {
  return split_gemm<F8x7>(W, op, epi, epi2, p.N, p.NP, p.w0, s);
}
__device__ __forceinline__ void f8_gemm4(double2* W, uint32_t op, int epi, const MxPlan& p7,
                                      const MxShared s) {
  const MxPlan p = split_plan4(p7);
  split_gemm<F8x4>(W, op, epi, -1, p.N, p.NP, p.w0, s);
}

// the FP64 Gauss-Jordan of the plain form, un-permuted into dst; its area
// aliases the stages and the exponents.  Mg: work for the global-memory variant.
__device__ __noinline__ int gj64(const double2* X, double2 w, int N, double2* dst, double2* Mg,
                                 int gi) {
  extern __shared__ __align__(1024) unsigned char smem_dyn[];
  const bool gsm = N <= MX_SMEM_GJ_N && !gi;
  const Shared fs = fp64_layout(smem_dyn, N, GJ_PANEL, gsm);
  __syncthreads();
  int sing;
  if (gsm) {
    sing = gj_invert(X, w, N, fs);
    gj_store(N, fs, dst);
  } else {
    sing = gj_invert_global(X, w, N, Mg, fs);
    gj_store_global(N, Mg, fs, dst);
  }
  __syncthreads();
  return sing;
}

// (w I - W[iX])^-1 into workspace matrix G with its exponents: an FP32
// Gauss-Jordan with partial pivoting, then Newton-Schulz steps until |I - M G|_F
// <= 1e-8 before a step, or the FP64 Gauss-Jordan where that is not reached.  Uses matrices Mi, R, Gn as work; swaps G and Gn.  live0 / live1:
// matrices whose exponents a fallback has to make again (-1: none).
__device__ int s64_inverse(int iX, double2 w, double2* W, const MxPlan& pl, int& G, int& Gn, int Mi,
                           int R, int live0, int live1, int gi, const MxShared s) {
  const int N = pl.N;
  const size_t NN = (size_t)N * N;
  bool good = false;
  if (!gj32(W + iX * NN, w, N, W, Mi, G, R, s)) {
    float prev = 3.0e38f;
    for (int t = 0; t < 8 && !s.t().abort; ++t) {
      // R = I - M G; the sum is |R|_F^2
      const float res = sqrtf(block_sum_f(f8_gemm7(W, ops(Mi, G, R), OZ_IMINUS, -1, pl, s), s));
      if (!(res < 0.25f * prev)) break;               // no longer converging (or NaN)
      // Gn = G + G R: 30 bits of R keep the step's own error below |R| 2^-30
      f8_gemm4(W, ops(G, R, Gn, G), OZ_ADDTO, pl, s);
      swap_mat(G, Gn);
      if (res <= 1e-8f) {                             // the step left at most 1e-16
        good = true;
        break;
      }
      prev = res;
    }
  }
  if (good || s.t().abort) return 0;
  const int sing = gj64(W + iX * NN, w, N, W + G * NN, W + Mi * NN, gi);
  exps_of(W + G * NN, G, N, s);
  if (live0 >= 0) exps_of(W + live0 * NN, live0, N, s);
  if (live1 >= 0) exps_of(W + live1 * NN, live1, N, s);
  return sing;
}

// sum over q = 0 .. n-1 of f(q), subtracted term by term in order (as the
// reference's loops), the terms evaluated by all threads; result in thread 0
template <class F>
__device__ double list_sum(int n, F f, const MxShared s) {
  double* buf = reinterpret_cast<double*>(s.base());
  constexpr int NB = 4096;
  double acc = 0.0;
  for (int q0 = 0; q0 < n; q0 += NB) {
    const int m = min(NB, n - q0);
    __syncthreads();
    for (int q = threadIdx.x; q < m; q += blockDim.x) buf[q] = f(q0 + q);
    __syncthreads();
    if (threadIdx.x == 0)
      for (int q = 0; q < m; ++q) acc = acc - buf[q];
  }
  __syncthreads();
  return acc;
}

// spin terms of orbital io (1-based list entry + offset - 1): see spin_sums
__device__ __forceinline__ double spin_term(const double2* G, int N, int nw, int io, int c) {
  const int nwh = nw / 2, jl = io % nw;
  int partner = -1;
  double sgn = 0.0;
  if (jl < nwh) {
    partner = io + nwh;
    sgn = 1.0;
  } else if (jl < 2 * nwh) {
    partner = io - nwh;
    sgn = -1.0;
  }
  if (partner < 0) return 0.0;
  if (c == 2) return sgn * G[io + (size_t)io * N].y;
  const double2 gp = G[io + (size_t)partner * N];
  return c == 0 ? gp.y : sgn * gp.x;
}

// GLL = (w - eps_s)^-1, GRR = (w - eps_t)^-1, GB = (w - eps)^-1 (src/surfgreen.f90:
// 127-134; eps, eps_s, eps_t in workspace matrices 0..2) and their spectral sums:
// dos_l, dos_r, dos_bulk, then sx, sy, sz of the left and the right surface, in
// thread 0's sums.  G, Gn, Mi, R: work matrices.  Returns whether one was singular.
template <class O>
__device__ int split_finals(double2 w, double2* W, const MxPlan& pl, const O& o, int G, int Gn,
                            int Mi, int R, double2* gll, double2* grr, double2* gb, int gi,
                            double (&sums)[9], const MxShared s) {
  const int N = pl.N, NN = N * N, tid = threadIdx.x;
  constexpr int iE = 0, iES = 1, iET = 2;
  int singular = 0;
  for (int k = 0; k < 3; ++k) {
    const int iX = k == 0 ? iES : k == 1 ? iET : iE;
    double2* const dst = k == 0 ? gll : k == 1 ? grr : gb;
    if (s64_inverse(iX, w, W, pl, G, Gn, Mi, R, -1, -1, gi, s)) singular = 1;
    __syncthreads();
    const double2* const g = W + (size_t)G * NN;
    if (dst)
      for (int e = tid; e < NN; e += blockDim.x) dst[e] = g[e];
    const int n = k == 0 ? o.ntop : k == 1 ? o.nbot : N;
    auto idx = [&](int q) {
      return k == 0 ? o.top[q] - 1 : k == 1 ? N - o.nw + o.bot[q] - 1 : q;
    };
    auto scaled = [&](double v) { return o.divide_by_pi ? v / PI_REF : v; };
    sums[k] = list_sum(n, [&](int q) {
      const int io = idx(q);
      return scaled(g[io + (size_t)io * N].y);
    }, s);
    if (k < 2 && o.spin[0]) {                       // src/surfstat.f90:162-192
      // surfstat's right sums run over the top list (as the reference's do)
      const bool top = k == 0 || !o.spin_right_bottom;
      const int off = top ? 0 : N - o.nw;
      for (int c = 0; c < 3; ++c)
        sums[3 + 3 * k + c] = list_sum(top ? o.ntop : o.nbot, [&](int q) {
          return scaled(spin_term(g, N, o.nw, off + (top ? o.top[q] : o.bot[q]) - 1, c));
        }, s);
    }
  }
  return singular;
}
