// All-FP64 Lopez-Sancho decimation (surfgreen_1985) for a batch of (k, omega)
// instances, one CTA per instance, persistent over an atomic work counter.
//
// Restates src/surfgreen.f90:74-134 per instance:
//   eps = eps_s = eps_t = H00, alpha = H01, beta = H01^dagger, w = omega + i eta
//   repeat (<= itermax):
//     g = (w - eps)^-1                           (Gauss-Jordan, shared memory)
//     m1 = alpha g ; m2 = beta g
//     t = m1 beta ; eps += t ; eps_s += t
//     t = m2 alpha; eps += t ; eps_t += t
//     alpha = m1 alpha ; beta = m2 beta
//     stop when sum_ij |alpha_ij| <= tol
//   GLL = (w - eps_s)^-1, GRR = (w - eps_t)^-1, GB = (w - eps)^-1
// followed by the spectral sums of src/surfstat.f90:149-160 /
// src/fermiarc.f90:237-248.
//
// This file: the kernels on the FP64 pipe (Ndim <= 8 a few lanes of a warp per
// instance, up to 24 and above 256 a CTA) and the routing; Ndim 25..256 runs on
// exactly split tensor-core products (wtg_split64.cu).
//
// GB300 notes.  FP64 runs at 2 DFMA/clk/SM on this part (1.2 TFLOP/s measured,
// with FP64 mma.sync slower still), so the CTA kernel is bound by the FP64 pipe,
// not by memory: the eight N x N matrices of an instance live in a per-CTA
// global workspace (L2-resident), GEMM operands are staged through shared
// memory in k-chunks, and the inverse runs in shared memory.  What matters is
// the count of FP64 instructions (exactly 4 DFMA per complex multiply-add)
// and keeping the pipe fed; pivot searches compare magnitudes as integers.
#include <algorithm>

#include <mutex>

#include "wtg_common.cuh"

namespace wtg {

namespace {

#include "wtg_fp64_dev.cuh"

#include "wtg_fp64_solve.cuh"
#include "wtg_small_dev.cuh"

template <int RP, bool GI>
__global__ void __launch_bounds__(GI ? 256 : 512, 1) k_decimate_fp64(const __grid_constant__ DecimArgs a) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const int N = a.N, NN = N * N, T = blockDim.x, tid = threadIdx.x;
  const Shared s = fp64_layout(smraw, N, a.KC, !GI);
  double2* W = a.ws + (size_t)blockIdx.x * (GI ? 9 : 8) * NN;

  for (;;) {
    if (tid == 0) s.misc[0] = atomicAdd(a.counter, 1);
    __syncthreads();
    const int inst = s.misc[0];
    __syncthreads();
    if (inst >= a.n_inst) break;
    const int ik = inst / a.nomega, iw = inst % a.nomega;
    const double2* H00 = a.h + (size_t)ik * 2 * NN;
    const double2* H01 = H00 + NN;
    const double2 w = make_double2(a.omega[iw], a.eta);     // src/surfgreen.f90:82
    for (int e = tid; e < NN; e += T) {                       // src/surfgreen.f90:74-78
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
    fp64_solve<RP, GI>(N, a.KC, w, a, a.gll ? a.gll + (size_t)inst * NN : nullptr,
                       a.grr ? a.grr + (size_t)inst * NN : nullptr,
                       a.gb ? a.gb + (size_t)inst * NN : nullptr, W, s,
                       [&](double dl, double dr, double db, const double* spin, int it, int st) {
                         a.dos_l[oidx] = dl;
                         a.dos_r[oidx] = dr;
                         a.dos_bulk[oidx] = db;
                         if (a.spin[0])
                           for (int c = 0; c < 6; ++c) a.spin[c][oidx] = spin[c];
                         if (a.iters) a.iters[oidx] = it;
                         if (a.status) a.status[oidx] = (uint8_t)st;
                       });
  }
}

// Ndim <= 8: a group of lanes per instance (small_solve), warps striding over the
// instances
template <int P>
__global__ void __launch_bounds__(128) k_decimate_small(const __grid_constant__ DecimArgs a) {
  constexpr int PER = 32 / Small<P>::G;            // instances a warp
  const int N = a.N, NN = N * N;
  const long long nwarp = (long long)gridDim.x * 4;
  const int sub = (threadIdx.x & 31) / Small<P>::G;
  for (long long q = ((long long)blockIdx.x * 4 + (threadIdx.x >> 5)) * PER; q < a.n_inst;
       q += nwarp * PER) {
    const bool valid = q + sub < a.n_inst;
    const int inst = valid ? (int)(q + sub) : 0;
    const int ik = inst / a.nomega, iw = inst % a.nomega;
    const double2* H00 = a.h + (size_t)ik * 2 * NN;
    const double2 w = make_double2(a.omega[iw], a.eta);     // src/surfgreen.f90:82
    const size_t oidx = (size_t)(a.k_offset + ik) + (size_t)iw * a.nk_total;
    small_solve<P>(N, w, a, H00, H00 + NN, valid,
                   [&](double dl, double dr, double db, const double* spin, int it, int st) {
                     a.dos_l[oidx] = dl;
                     a.dos_r[oidx] = dr;
                     a.dos_bulk[oidx] = db;
                     if (a.spin[0])
                       for (int c = 0; c < 6; ++c) a.spin[c][oidx] = spin[c];
                     if (a.iters) a.iters[oidx] = it;
                     if (a.status) a.status[oidx] = (uint8_t)st;
                   });
  }
}

// Uneven batch: points of several models (different Ndim, eta per point) in
// one persistent launch.  CTAs take points in the host's cost order (largest
// first); each point runs its own Fourier sum, then the shared-memory or the
// global-memory inverse variant by its Ndim, and stops at its own convergence.
__global__ void __launch_bounds__(256, 1) k_batch_fp64(const __grid_constant__ BatchArgs a) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const int tid = threadIdx.x;
  double2* W = a.ws + (size_t)blockIdx.x * a.ws_stride;
  __shared__ int sinst;
  const int npts = a.run ? a.run->npts : a.npts;
  const double tol = a.run ? a.run->tol : a.tol;
  const int itermax = a.run ? a.run->itermax : a.itermax;
  const int divide_by_pi = a.run ? a.run->divide_by_pi : a.divide_by_pi;
  for (;;) {
    if (tid == 0) {
      const int q = atomicAdd(a.counter, 1);
      sinst = q < npts ? a.order[q] : -1;
    }
    __syncthreads();
    const int p = sinst;
    __syncthreads();
    if (p < 0) break;
    const BatchModel& m = a.models[a.pmodel[p]];
    const int N = m.N;
    const bool gi = N > a.smem_gj_max;
    const Shared s = fp64_layout(smraw, N, a.KC, !gi);
    fourier_fill(m, a.k[p], a.k[p + a.npts], W, reinterpret_cast<double2*>(smraw + a.ph_off));
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
    if (N <= SMALL_MAX_N) {                  // one warp, as k_decimate_small
      if (tid < 32) small_point(N, w, o, W, emit);
      __syncthreads();
    } else if (gi) fp64_solve<13, true>(N, a.KC, w, o, nullptr, nullptr, nullptr, W, s, emit);
    else fp64_solve<13, false>(N, a.KC, w, o, nullptr, nullptr, nullptr, W, s, emit);
  }
}

// one product (op 0) or inverse (op 1) on the FP64 pipe by one CTA (Ndim below
// FP64_SPLIT_MIN_N): W holds X, Y, the result and work matrices
__global__ void __launch_bounds__(512, 1) k_fp64_unit(int op, int N, int KC, double2* W,
                                                      int* status) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const int NN = N * N;
  const Shared s = fp64_layout(smraw, N, KC, true);
  double2* const C = W + 2 * NN;
  if (op == 0) {
    cta_gemm<13, EPI_STORE>(W, W + NN, N, KC, s.sX, s.sY, C, nullptr);
    if (threadIdx.x == 0) *status = 0;
  } else {
    double2* const negX = W + 3 * NN;
    for (int e = threadIdx.x; e < NN; e += blockDim.x) negX[e] = make_double2(-W[e].x, -W[e].y);
    __syncthreads();
    const int sing = gj_invert(negX, make_double2(0.0, 0.0), N, s);   // (0 I - (-X))^-1
    gj_store(N, s, C);
    if (threadIdx.x == 0) *status = sing ? PT_SINGULAR : 0;
  }
}

size_t smem_bytes(int N, int KC, bool inv_in_smem) {
  const size_t big = inv_in_smem ? (size_t)(N * N > 2 * N * KC ? N * N : 2 * N * KC)
                                 : (size_t)2 * N * KC;
  return big * 16 + (size_t)N * 32 + 16 * GJ_PANEL + 32 * 8 + (size_t)N * 8 + 16;
}

}  // namespace

int decim_fp64_max_n() {
  int n = 8;
  while (smem_bytes(n + 1, (n + 1) / 2, true) <= 227 * 1024) ++n;
  return n;
}

int decim_fp64_large_max_n() { return 32 * GJ_ROWS; }

int fp64_threads_default(int N) { return N <= 48 ? 128 : (N <= 80 ? 256 : 512); }

int fp64_threads_for(int N, long long n_inst, int nsm) {
  const int tile = tile_value(0, N);
  if (tile > 0) return tile;
  // from timings at Ndim 12 / 16 / 20 / 24: with no more instances than SMs a wider
  // CTA shortens each (0.77 -> 0.67, 0.95 -> 0.85, 1.94 -> 1.52, 2.33 -> 2.15 ms a
  // point against 128 threads); with many, narrow ones keep more instances in
  // flight (20 000, 16 875 and 8 639 points: 38.6 -> 32.1, 43.5 -> 43.3, 52.5 ->
  // 46.7 ms with 64 threads)
  if (N >= 12 && n_inst <= nsm) return 256;
  if (N <= 20 && n_inst >= 8LL * nsm) return 64;
  return fp64_threads_default(N);
}

size_t decim_fp64_ws_matrices(const DecimConfig& cfg) {
  return cfg.small ? 0 : cfg.split ? 11 : cfg.inv_global ? 9 : 8;
}

// launch shape of the kernel on the FP64 pipe (Ndim 9..24, above 256 and in the unit
// kernel; any with force_global)
static cudaError_t dfma_config(int N, int threads_override, DecimConfig* cfg, bool force_global) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  int smem_optin = 0;
  e = cudaDeviceGetAttribute(&smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e != cudaSuccess) return e;
  const bool gi = force_global || N > decim_fp64_max_n();
  if (gi && N > decim_fp64_large_max_n()) return cudaErrorInvalidValue;
  if (threads_override <= 0) threads_override = tile_value(0, N);
  int T = threads_override > 0 ? threads_override : fp64_threads_default(N);
  if (gi) T = 256;                 // 255 registers: a lane keeps 10 rows of a column
  const int KC = gi ? 16 : N;
  if (smem_bytes(N, KC, !gi) > (size_t)smem_optin) return cudaErrorInvalidValue;
  const int rounds = (N * N + T - 1) / T;      // at most 7 where not gi
  const int RP = gi ? 13 : rounds <= 4 ? 4 : 8;
  cfg->threads = T;
  cfg->KC = KC;
  cfg->RP = RP;
  cfg->inv_global = gi ? 1 : 0;
  cfg->smem = smem_bytes(N, KC, !gi);
  int occ = 0;
  const void* fn = gi ? (const void*)k_decimate_fp64<13, true>
                   : RP == 4 ? (const void*)k_decimate_fp64<4, false> : (const void*)k_decimate_fp64<8, false>;
  e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cfg->smem);
  if (e != cudaSuccess) return e;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, T, cfg->smem);
  if (e != cudaSuccess) return e;
  cfg->ctas_per_sm = occ;
  return cudaSuccess;
}

// Ndim <= SMALL_MAX_N without full-matrix outputs: warps without a workspace (the
// CTA-wide kernel stays for full matrices and the forced global-memory inverse)
static cudaError_t small_config(int N, DecimConfig* cfg) {
  cfg->small = 1;
  cfg->threads = 128;
  cfg->smem = 0;
  const void* fn = N <= 4 ? (const void*)k_decimate_small<4> : (const void*)k_decimate_small<8>;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&cfg->ctas_per_sm, fn, cfg->threads, 0);
}

cudaError_t decim_fp64_config(int N, int threads_override, DecimConfig* cfg, bool force_global,
                              bool full_out) {
  if (N <= SMALL_MAX_N && !force_global && !full_out) return small_config(N, cfg);
  if (fp64_split(N)) {
    const cudaError_t e = split64_config(N, cfg);
    cfg->inv_global = force_global ? 1 : 0;       // of the FP64 fallback inverse
    return e;
  }
  return dfma_config(N, threads_override, cfg, force_global);
}

cudaError_t launch_decimate_fp64(const DecimArgs& a, const DecimConfig& cfg, int grid,
                                 cudaStream_t s) {
  if (cfg.split) return launch_split64(a, cfg, grid, s);
  if (cfg.small) {
    if (a.N <= 4) k_decimate_small<4><<<grid, cfg.threads, 0, s>>>(a);
    else k_decimate_small<8><<<grid, cfg.threads, 0, s>>>(a);
    return cudaGetLastError();
  }
  if (cfg.inv_global) k_decimate_fp64<13, true><<<grid, cfg.threads, cfg.smem, s>>>(a);
  else if (cfg.RP == 4) k_decimate_fp64<4, false><<<grid, cfg.threads, cfg.smem, s>>>(a);
  else k_decimate_fp64<8, false><<<grid, cfg.threads, cfg.smem, s>>>(a);
  return cudaGetLastError();
}

size_t batch_ws_matrices(const DecimConfig& cfg) { return cfg.split ? 11 : 9; }

static size_t batch_fp64_smem(int max_n, int max_smem_gj_n, int KC) {
  size_t b = smem_bytes(max_n, KC, false);
  if (max_smem_gj_n > 0) {
    const size_t t = smem_bytes(max_smem_gj_n, KC, true);
    if (t > b) b = t;
  }
  return b;
}

cudaError_t batch_fp64_config(int max_n, size_t extra_smem, int* smem_gj_max, int* wb,
                              DecimConfig* cfg) {
  // the split kernel wherever the phase table fits its stages (206 KB: 12 864 R vectors); more
  // take the FP64 pipe, whose shared memory leaves room for a few hundred to 1 300 others
  if (max_n >= FP64_SPLIT_MIN_N) {
    *smem_gj_max = 0;
    const cudaError_t e = batch_split64_config(max_n, wb, cfg);
    if (e != cudaSuccess || extra_smem <= cfg->ph_room) return e;
    *cfg = DecimConfig();
  }
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  int smem_optin = 0;
  e = cudaDeviceGetAttribute(&smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e != cudaSuccess) return e;
  if (max_n > decim_fp64_large_max_n()) return cudaErrorInvalidValue;
  const int KC = 16;
  // the shared-memory inverse up to the largest Ndim that fits beside the stages
  int g = 0;
  while (g + 1 <= decim_fp64_max_n() && smem_bytes(g + 1, KC, true) + extra_smem + 16 <= (size_t)smem_optin)
    ++g;
  *smem_gj_max = g;
  cfg->threads = 256;
  cfg->KC = KC;
  cfg->RP = 13;
  cfg->inv_global = 1;
  cfg->smem = batch_fp64_smem(max_n, std::min(g, max_n), KC);
  if (cfg->smem + extra_smem + 16 > (size_t)smem_optin) return cudaErrorInvalidValue;
  cfg->ctas_per_sm = 1;
  return cudaSuccess;
}

// the batch kernel's dynamic shared-memory limit raised once per device to the
// opt-in maximum (engines of any size launch it, also from captured graphs)
cudaError_t batch_fp64_prepare() {
  static std::mutex mu;
  static bool done[64];
  int dev = 0, optin = 0;
  cudaError_t err = cudaGetDevice(&dev);
  if (err != cudaSuccess) return err;
  std::lock_guard<std::mutex> lk(mu);
  if (dev < 64 && done[dev]) return cudaSuccess;
  cudaFuncAttributes fa;
  err = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (err == cudaSuccess) err = cudaFuncGetAttributes(&fa, k_batch_fp64);
  if (err == cudaSuccess)
    err = cudaFuncSetAttribute(k_batch_fp64, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               optin - (int)fa.sharedSizeBytes);
  if (err == cudaSuccess) err = batch_split64_prepare();
  if (err == cudaSuccess && dev < 64) done[dev] = true;
  return err;
}

cudaError_t launch_batch_fp64(const BatchArgs& a, const DecimConfig& cfg, int grid, cudaStream_t s) {
  if (cfg.split) return launch_batch_split64(a, cfg, grid, s);
  k_batch_fp64<<<grid, cfg.threads, cfg.smem, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_fp64_unit(int op, int N, double2* W, int* status, cudaStream_t st) {
  if (N >= FP64_SPLIT_MIN_N) return launch_split64_unit(op, N, W, status, st);
  DecimConfig cfg;
  cudaError_t e = dfma_config(N, 512, &cfg, false);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(k_fp64_unit, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cfg.smem);
  if (e != cudaSuccess) return e;
  k_fp64_unit<<<1, 512, cfg.smem, st>>>(op, N, cfg.KC, W, status);
  return cudaGetLastError();
}

}  // namespace wtg
