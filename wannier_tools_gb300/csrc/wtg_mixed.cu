// Mixed-precision Lopez-Sancho decimation on the 5th-generation tensor cores.
//
// Every complex product of surfgreen_1985 (src/surfgreen.f90:92-116, zgemm at
// src/mat_mul.f90:23) runs as an exactly-split BF16 product on tcgen05
// (split_gemm of wtg_split.cuh with DigB7 digits): 49-bit operands in seven
// balanced base-128 digits, one FP32 accumulator in tensor memory for each of
// the slice orders 2..6 and one for the orders 7 and 8.  49 bits are needed
// because the Newton-Schulz refinement below can only be as accurate as its
// residual product.
// Inverses in the loop (zgesv with identity, src/inverse.f90:43-55) are an
// FP32 Gauss-Jordan (shared memory up to Ndim 112, global memory in panels
// above) followed by Newton-Schulz refinement X <- X + X (I - M X): the
// residual I - M X is a 7-digit split product, the correction X R a 4-digit
// one (R is small).  The three final inverses (src/surfgreen.f90:127-134) are
// FP64 (the FP64 form's own), and the convergence test
// sum |alpha_ij| (src/surfgreen.f90:120) takes each |alpha_ij| and the sum in
// FP64 wherever the FP32 bounds of the sum do not decide it.
#include <mutex>

#include "../../include/wtgpu.h"
#include "wtg_common.cuh"

namespace wtg {

namespace {

#include "wtg_fp64_dev.cuh"
#include "wtg_split.cuh"
#include "wtg_split_inverse.cuh"

// 7-digit products, and the 4-digit corrections of the refinement
using Dig7 = DigB7<7>;
using Dig4 = DigB7<4>;
constexpr int MX_T = SP_T;

// widest pass: both components side by side, 2 x 6 accumulators of w columns in
// the 512 tensor-memory columns
__host__ __device__ inline int mx_wmax() { return split_wmax<Dig7>(); }

__host__ __device__ inline MxPlan mx_plan(int N, int w0_req = 0) {
  return split_plan(N, mx_wmax(), w0_req);
}

__device__ __forceinline__ float gemm7(double2* W, uint32_t op, int epi, int epi2, const MxPlan& p,
                                       const MxShared s) {
  return split_gemm<Dig7>(W, op, epi, epi2, p.N, p.NP, p.w0, s);
}
__device__ __forceinline__ void gemm4(double2* W, uint32_t op, int epi, const MxPlan& p7,
                                      const MxShared s) {
  const MxPlan p = split_plan4(p7);
  split_gemm<Dig4>(W, op, epi, -1, p.N, p.NP, p.w0, s);
}

// (w I - X)^-1 into workspace matrix G: FP32 Gauss-Jordan, then Newton-Schulz
// steps G <- G + G (I - M G) on the split tensor-core products until the
// residual sum_ij |I - M G|_1 stops shrinking quadratically, or is at most brk N
// before an update (after which it is ~(brk N)^2; brk = 1e-7 puts it below the
// products' own rounding); at most ns_max steps.  Uses matrices Mi, R, Gn as
// work; swaps G and Gn.
__device__ int mixed_inverse(const double2* X, double2 w, double2* W, const MxPlan& pl, int ns_max,
                             int& G, int& Gn, int Mi, int R, const MxShared s, float brk = 1e-7f) {
  const int N = pl.N;
  const int sing = gj32(X, w, N, W, Mi, G, R, s);
  float prev = 3.0e38f;
  for (int t = 0; t < ns_max && !s.t().abort; ++t) {
    // R = I - M G
    const float res = block_sum_f(gemm7(W, ops(Mi, G, R), OZ_IMINUS, -1, pl, s), s);
    if (!(res < 0.25f * prev)) break;                 // no longer converging (or NaN)
    // Gn = G + G R: R is small, so 4 digits (28 bits) keep G R far below G's own error
    gemm4(W, ops(G, R, Gn, G), OZ_ADDTO, pl, s);
    swap_mat(G, Gn);
    if (res <= brk * (float)N) break;                 // G + G R is then accurate enough
    prev = res;
  }
  return sing;
}

// Decimation of one instance whose eps, eps_s, eps_t (= H00), alpha (= H01)
// and beta (= H01^dagger) already sit in workspace matrices 0..4 of W (11
// N x N matrices); the spectral sums go to emit(dl, dr, db, spin[6],
// iterations, status) in thread 0, the final inverses to gll / grr / gb when
// those are not null.  o has DecimArgs' member names (lists, tolerance, ...).
// The loop's products and inverses are the split-BF16 forms; the three final
// inverses (src/surfgreen.f90:127-134) are FP64 (split_finals).
template <class O, class Emit>
__device__ __forceinline__ void mixed_solve(const MxPlan& pl, double2 w, const O& o, int ns_iter,
                                            double2* gll, double2* grr, double2* gb, double2* W,
                                            const MxShared s, Emit emit) {
  const int N = pl.N, NN = N * N, tid = threadIdx.x;
  int Al = 3, Be = 4, G = 5, R = 9, Gn = 10;         // workspace matrices by index
  constexpr int iE = 0, iES = 1, iET = 2, M1 = 6, M2 = 7, iMi = 8;
  int stat = 0, it = 0;
  bool conv = false;
  split_tables<Dig7, Dig4>(pl, s);
  exps_of(W + (size_t)Al * NN, Al, N, s);
  exps_dagger(Be, Al, N, s);
  for (int itc = 1; itc <= o.itermax && !s.t().abort; ++itc) {   // src/surfgreen.f90:86-122
    it = itc;
    // the refinement stops at a residual sum of 1e-4 Ndim (then ~1e-8 after its
    // update): the dense Fermi-arc check stays below 2e-6 against the FP64 oracle
    if (mixed_inverse(W, w, W, pl, ns_iter, G, Gn, iMi, R, s, 1e-4f)) stat |= PT_SINGULAR;
    // the reference's six products (:92-116); eps still receives M1 beta before
    // M2 alpha.  Where it takes fewer 128-row tiles (Ndim mod 128 in 1..64: up to
    // Ndim 64, or 129..192, 257..320), the products with a common right factor
    // run as one product whose rows are those of the first and then those of the
    // second: three products instead of six.
    float part;
    if ((2 * N + 127) / 128 < 2 * ((N + 127) / 128)) {
      gemm7(W, ops(Al, G, M1, 0, Be, M2), OZ_STORE, OZ_STORE, pl, s);               // :92, :95
      gemm7(W, ops(M1, Be, iE, iES, M2, R), OZ_ADD2, OZ_STORE, pl, s);              // :98-102, :116
      part = gemm7(W, ops(M1, Al, Gn, 0, M2, iE, iET), OZ_STORE_NORM, OZ_ADD2, pl, s);  // :113, :107-110
    } else {
      gemm7(W, ops(Al, G, M1), OZ_STORE, -1, pl, s);                                // :92
      gemm7(W, ops(Be, G, M2), OZ_STORE, -1, pl, s);                                // :95
      gemm7(W, ops(M1, Be, iE, iES), OZ_ADD2, -1, pl, s);                           // :98-102
      part = gemm7(W, ops(M1, Al, Gn), OZ_STORE_NORM, -1, pl, s);                   // :113
      gemm7(W, ops(M2, Al, iE, iET), OZ_ADD2, -1, pl, s);                           // :107-110
      gemm7(W, ops(M2, Be, R), OZ_STORE, -1, pl, s);                                // :116
    }
    swap_mat(Al, Gn);
    swap_mat(Be, R);
    if (converged(part, W + (size_t)Al * NN, N, o.tol, s)) {     // :120-122
      conv = true;
      break;
    }
  }
  if (!conv) stat |= PT_NOT_CONVERGED;

  // the three final inverses in FP64, refined on 55-bit products (Ndim 112:
  // eliminations on the FP64 pipe took 17 % of a solve, 112 against 103.5 ms for 912
  // points; Ndim 40: 64.4 and 65.9 ms for 5151)
  MxPlan pf = split_plan(N, min(split_wmax<F8x7>(), pl.wb));
  pf.wb = pl.wb;
  split_tables<F8x7, F8x4>(pf, s);
  double sums[9];                                   // dl, dr, db, then the six spin sums
  if (split_finals(w, W, pf, o, G, Gn, iMi, R, gll, grr, gb, 0, sums, s)) stat |= PT_SINGULAR;
  if (tid == 0) {
    if (s.t().abort) stat |= PT_TIMEOUT;
    if (!isfinite(sums[0]) || !isfinite(sums[1]) || !isfinite(sums[2])) stat |= PT_NONFINITE;
    emit(sums[0], sums[1], sums[2], sums + 3, it, stat);
  }
  __syncthreads();
}

__global__ void __launch_bounds__(MX_T, 1) k_decimate_mixed(const __grid_constant__ DecimArgs a,
                                                            int ns_iter, unsigned spin_limit) {
  const int N = a.N, NN = N * N, T = blockDim.x, tid = threadIdx.x;
  const MxPlan pl = mx_plan(N, a.w0);
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
    if (s.t().abort) {        // a wait gave up earlier: the rest of this CTA's points are not computed
      if (tid == 0) {
        const size_t oidx = (size_t)(a.k_offset + ik) + (size_t)iw * a.nk_total;
        const double nan = __longlong_as_double(0x7FF8000000000000LL);
        a.dos_l[oidx] = nan;
        a.dos_r[oidx] = nan;
        a.dos_bulk[oidx] = nan;
        if (a.spin[0])
          for (int c = 0; c < 6; ++c) a.spin[c][oidx] = nan;
        if (a.iters) a.iters[oidx] = 0;
        if (a.status) a.status[oidx] = (uint8_t)PT_TIMEOUT;
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
      W[3 * NN + e] = H01[e];
      const int i = e % N, j = e / N;
      const double2 t = H01[j + (size_t)i * N];
      W[4 * NN + e] = make_double2(t.x, -t.y);
    }
    __syncthreads();
    const size_t oidx = (size_t)(a.k_offset + ik) + (size_t)iw * a.nk_total;
    mixed_solve(pl, w, a, ns_iter, a.gll ? a.gll + (size_t)inst * NN : nullptr,
                a.grr ? a.grr + (size_t)inst * NN : nullptr,
                a.gb ? a.gb + (size_t)inst * NN : nullptr, W, s,
                [&](double dl, double dr, double db, const double* spin, int it, int stat) {
                  a.dos_l[oidx] = dl;
                  a.dos_r[oidx] = dr;
                  a.dos_bulk[oidx] = db;
                  if (a.spin[0])
                    for (int c = 0; c < 6; ++c) a.spin[c][oidx] = spin[c];
                  if (a.iters) a.iters[oidx] = it;
                  if (a.status) a.status[oidx] = (uint8_t)stat;
                });
  }
  mx_teardown(s);
}

// options of one batch instance, with DecimArgs' member names
struct MxOpts {
  int nw;
  double tol;
  int itermax;
  int divide_by_pi;
  int ntop, nbot;
  const int* top;
  const int* bot;
  double* spin[6];
  int spin_right_bottom;
};

// Uneven batch in one persistent launch (mixed form): as k_batch_fp64, with the
// shared-memory layout sized for the widest B plane of the batch (a.wb).
__global__ void __launch_bounds__(MX_T, 1) k_batch_mixed(const __grid_constant__ BatchArgs a,
                                                         int ns_iter, unsigned spin_limit) {
  extern __shared__ __align__(1024) unsigned char smraw[];
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
    if (p < 0 || s.t().abort) {
      if (p >= 0 && tid == 0) {       // a wait gave up earlier: not computed
        const double nan = __longlong_as_double(0x7FF8000000000000LL);
        a.dos_l[p] = nan;
        a.dos_r[p] = nan;
        a.dos_bulk[p] = nan;
        if (a.iters) a.iters[p] = 0;
        if (a.status) a.status[p] = PT_TIMEOUT;
      }
      if (p < 0) break;
      continue;
    }
    const BatchModel& m = a.models[a.pmodel[p]];
    MxPlan pl = mx_plan(m.N, m.w0);
    pl.wb = a.wb;
    fourier_fill(m, a.k[p], a.k[p + a.npts], W, reinterpret_cast<double2*>(smraw + a.ph_off));
    MxOpts o;
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
    mixed_solve(pl, make_double2(a.omega[p], a.eta[p]), o, ns_iter, nullptr, nullptr,
                nullptr, W, s,
                [&](double dl, double dr, double db, const double*, int it, int stat) {
                  a.dos_l[p] = dl;
                  a.dos_r[p] = dr;
                  a.dos_bulk[p] = db;
                  if (a.iters) a.iters[p] = it;
                  if (a.status) a.status[p] = (uint8_t)stat;
                });
  }
  mx_teardown(s);
}

// single complex product / inverse through the same device code (one CTA): W
// holds X, Y, the result and five work matrices
__global__ void __launch_bounds__(MX_T, 1) k_mixed_unit(int op, int N, double2* W, int ns,
                                                        int* status) {
  const MxPlan pl = mx_plan(N);
  const int NN = N * N, tid = threadIdx.x;
  const MxShared s = mx_layout(pl.wb);
  mx_setup(s, 0u);
  split_tables<Dig7, Dig4>(pl, s);
  int sing = 0;
  if (op == 0) {
    exps_of(W, 0, N, s);
    exps_of(W + NN, 1, N, s);
    gemm7(W, ops(0, 1, 2), OZ_STORE, -1, pl, s);
  } else {
    // C = X^-1: X given directly, so pass -X with w = 0 (M = 0*I - (-X) = X)
    double2* negX = W + 7 * (size_t)NN;
    for (int e = tid; e < NN; e += blockDim.x) negX[e] = make_double2(-W[e].x, -W[e].y);
    __syncthreads();
    int G = 3, Gn = 4;
    sing = mixed_inverse(negX, make_double2(0.0, 0.0), W, pl, ns, G, Gn, 6, 5, s);
    double2* C = W + 2 * (size_t)NN;
    for (int e = tid; e < NN; e += blockDim.x) C[e] = W[(size_t)G * NN + e];
  }
  if (tid == 0) *status = (s.t().abort ? PT_TIMEOUT : 0) | (sing ? PT_SINGULAR : 0);
  mx_teardown(s);
}

size_t mixed_smem(int N, int wb = 0) {     // wb = 0: the built-in plan's width
  return split_smem(wb > 0 ? wb : mx_plan(N).w0);
}

}  // namespace

int decim_mixed_max_n() { return MX_MAXN; }

size_t decim_mixed_ws_matrices() { return 11; }

cudaError_t decim_mixed_config(int N, DecimConfig* cfg) {
  cfg->threads = MX_T;
  cfg->KC = 0;
  cfg->RP = 0;
  cfg->split = 1;
  cfg->w0 = mx_plan(N, tile_value(1, N)).w0;
  // at least 116 KB so that two CTAs never share an SM (each allocates all 512 TMEM columns)
  const size_t sm = mixed_smem(N, cfg->w0);
  cfg->smem = sm > (size_t)(116 << 10) ? sm : (size_t)(116 << 10);
  cudaError_t e = cudaFuncSetAttribute(k_decimate_mixed, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)cfg->smem);
  if (e != cudaSuccess) return e;
  int occ = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_decimate_mixed, MX_T, cfg->smem);
  if (e != cudaSuccess) return e;
  cfg->ctas_per_sm = occ > 1 ? 1 : occ;     // tensor memory is allocated whole (512 columns)
  return cudaSuccess;
}

cudaError_t launch_decimate_mixed(const DecimArgs& a, const DecimConfig& cfg, int grid,
                                  cudaStream_t s) {
  k_decimate_mixed<<<grid, cfg.threads, cfg.smem, s>>>(
      a, 6, (unsigned)test_option(WTG_TEST_MIXED_SPIN_LIMIT));
  return cudaGetLastError();
}

cudaError_t batch_mixed_config(int max_n, int* wb, DecimConfig* cfg) {
  if (max_n > MX_MAXN) return cudaErrorInvalidValue;
  int w = 16;
  size_t smem = 0;
  for (int n = 1; n <= max_n; ++n) {
    const int wn = mx_plan(n, tile_value(1, n)).w0;
    w = w > wn ? w : wn;
  }
  for (int n = 1; n <= max_n; ++n) {
    const size_t t = mixed_smem(n, w);
    smem = smem > t ? smem : t;
  }
  *wb = w;
  cfg->split = 1;
  cfg->threads = MX_T;
  cfg->KC = 0;
  cfg->RP = 0;
  cfg->inv_global = 0;
  cfg->smem = smem > (size_t)(116 << 10) ? smem : (size_t)(116 << 10);
  cfg->ctas_per_sm = 1;
  return cudaSuccess;
}

// as batch_fp64_prepare
cudaError_t batch_mixed_prepare() {
  static std::mutex mu;
  static bool done[64];
  int dev = 0, optin = 0;
  cudaError_t err = cudaGetDevice(&dev);
  if (err != cudaSuccess) return err;
  std::lock_guard<std::mutex> lk(mu);
  if (dev < 64 && done[dev]) return cudaSuccess;
  cudaFuncAttributes fa;
  err = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (err == cudaSuccess) err = cudaFuncGetAttributes(&fa, k_batch_mixed);
  if (err == cudaSuccess)
    err = cudaFuncSetAttribute(k_batch_mixed, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               optin - (int)fa.sharedSizeBytes);
  if (err == cudaSuccess && dev < 64) done[dev] = true;
  return err;
}

cudaError_t launch_batch_mixed(const BatchArgs& a, const DecimConfig& cfg, int grid,
                               cudaStream_t s) {
  k_batch_mixed<<<grid, cfg.threads, cfg.smem, s>>>(
      a, 6, (unsigned)test_option(WTG_TEST_MIXED_SPIN_LIMIT));
  return cudaGetLastError();
}

int batch_mixed_w0(int N) { return mx_plan(N, tile_value(1, N)).w0; }

int mixed_w0_default(int N) { return mx_plan(N).w0; }

int mixed_w0_max(int) { return mx_wmax(); }

cudaError_t launch_mixed_unit(int op, int N, double2* W, int ns, int* status, cudaStream_t s) {
  const size_t smem = mixed_smem(N) > (size_t)(116 << 10) ? mixed_smem(N) : (size_t)(116 << 10);
  cudaError_t e =
      cudaFuncSetAttribute(k_mixed_unit, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  k_mixed_unit<<<1, MX_T, smem, s>>>(op, N, W, ns, status);
  return cudaGetLastError();
}

}  // namespace wtg
