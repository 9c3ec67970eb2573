// One decimation on the FP64 pipe (surfgreen_1985, src/surfgreen.f90:74-134),
// shared by the per-model and the batch kernels.  Included inside an anonymous
// namespace after wtg_fp64_dev.cuh.
#pragma once

// Options of one solve for the batch kernel, with the member names of
// DecimArgs (whose kernel parameter the plain kernel passes directly, so its
// lists are read from parameter space).  Orbital lists are 1-based.
struct SolveOpts {
  int nw;
  double tol;
  int itermax;
  int divide_by_pi;
  int ntop, nbot;
  const int* top;
  const int* bot;
  double* spin[6];             // null: no spin-resolved sums
  int spin_right_bottom;
};

// The products of one decimation step.  At the large Ndim of the global-memory
// inverse the eight workspaces of all resident CTAs no longer fit the L2, so
// operands come from DRAM and their staging is double-buffered.
template <int RP, int EPI, bool GI>
__device__ __forceinline__ double gemm(const double2* X, const double2* Y, int N, int KC,
                                       const Shared& s, double2* out0, double2* out1) {
  if (GI) return cta_gemm_db<RP, EPI>(X, Y, N, KC, s.sX, out0, out1);
  return cta_gemm<RP, EPI>(X, Y, N, KC, s.sX, s.sY, out0, out1);
}

// Decimation of one instance whose eps, eps_s, eps_t (= H00), alpha (= H01)
// and beta (= H01^dagger) already sit in workspace matrices 0..4 of W; the
// spectral sums of the three final inverses are handed to emit(dl, dr, db,
// spin[6], iterations, status) in thread 0, the inverses themselves go to
// gll / grr / gb when those are not null.
// GI = false: the inverse runs in shared memory (Ndim <= decim_fp64_max_n());
// GI = true: it runs in workspace matrix 8 in global memory, in panels
// (gj_invert_global; Ndim <= 320).
template <int RP, bool GI, class O, class Emit>
__device__ void fp64_solve(int N, int KC, double2 w, const O& o, double2* gll, double2* grr,
                           double2* gb, double2* W, const Shared& s, Emit emit) {
  const int NN = N * N, tid = threadIdx.x;
  double2* Mg = GI ? W + (size_t)8 * NN : nullptr;   // global-memory inverse work
  double2* E = W;
  double2* ES = W + (size_t)NN;
  double2* ET = W + (size_t)2 * NN;
  double2* Al = W + (size_t)3 * NN;
  double2* Be = W + (size_t)4 * NN;
  double2* G = W + (size_t)5 * NN;
  double2* M1 = W + (size_t)6 * NN;
  double2* M2 = W + (size_t)7 * NN;
  // (w - X)^-1, optionally stored un-permuted to dst; ginv reads the result
  // blk 1 / 2: only the leading / trailing Num_wann block of the inverse (one
  // principal layer), from the Schur complement of the rest, where the spectral
  // sums read nothing else (schur_block_invert); a zero pivot there takes the
  // full inverse.  With GI the block's inverse needs its Num_wann^2 area within
  // the stage area every launch of this Ndim has (KC = 16).
  const int m = N - o.nw;
  const bool gblk = !GI || schur_area_bytes(N, o.nw) <= fp64_gi_smem_bytes(N);
  const Shared fb = schur_layout(reinterpret_cast<unsigned char*>(s.big), N, o.nw);
  int blk = 0;
  auto invert = [&](const double2* X, double2* dst, int want_blk) -> int {
    blk = (gblk && !dst && m > 0) ? want_blk : 0;
    if (blk && !(GI ? schur_block_invert_global(X, w, N, o.nw, blk == 1, Mg, fb)
                    : schur_block_invert(X, w, N, o.nw, blk == 1, s)))
      return 0;
    blk = 0;
    int sing;
    if (GI) {
      sing = gj_invert_global(X, w, N, Mg, s);
      if (dst) gj_store_global(N, Mg, s, dst);
    } else {
      sing = gj_invert(X, w, N, s);
      if (dst) gj_store(N, s, dst);
    }
    return sing;
  };
  auto ginv = [&](int i, int j) {
    if (blk) {                        // block entry (i, j): local indices in the block
      const int li = blk == 1 ? o.nw - 1 - i : i - m;
      const int lj = blk == 1 ? o.nw - 1 - j : j - m;
      return GI ? fb.big[li + (size_t)fb.cols[lj] * o.nw]
                : s.big[m + li + (size_t)(m + s.cols[lj]) * N];
    }
    return GI ? Mg[i + (size_t)s.cols[j] * N] : s.big[i + s.cols[j] * N];
  };

  int st = 0, it = 0;
  bool conv = false;
  for (int itc = 1; itc <= o.itermax; ++itc) {                // src/surfgreen.f90:86
    it = itc;
    if (invert(E, G, 0)) st |= PT_SINGULAR;                   // :88-89
    __syncthreads();
    gemm<RP, EPI_STORE, GI>(Al, G, N, KC, s, M1, nullptr);              // :92
    gemm<RP, EPI_STORE, GI>(Be, G, N, KC, s, M2, nullptr);              // :95
    gemm<RP, EPI_ADD2, GI>(M1, Be, N, KC, s, E, ES);                    // :98-102
    gemm<RP, EPI_ADD2, GI>(M2, Al, N, KC, s, E, ET);                    // :107-110
    double part = gemm<RP, EPI_STORE_NORM, GI>(M1, Al, N, KC, s, G, nullptr);  // :113
    gemm<RP, EPI_STORE, GI>(M2, Be, N, KC, s, M1, nullptr);             // :116
    // rotate buffers: alpha <- G, beta <- M1
    double2* t0 = Al;
    Al = G;
    G = t0;
    double2* t1 = Be;
    Be = M1;
    M1 = t1;
    const double nrm = block_sum(part, s);                    // :120
    if (nrm <= o.tol) {                                       // :121
      conv = true;
      break;
    }
  }
  if (!conv) st |= PT_NOT_CONVERGED;

  double dl = 0.0, dr = 0.0, db = 0.0;
  double spin[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  // GLL = (w - eps_s)^-1                                     // :127-128
  if (invert(ES, gll, 1)) st |= PT_SINGULAR;
  if (tid == 0) {
    for (int q = 0; q < o.ntop; ++q) {
      const int io = o.top[q] - 1;
      const double v = ginv(io, io).y;
      dl = o.divide_by_pi ? dl - v / PI_REF : dl - v;
    }
    if (o.spin[0])                                            // src/surfstat.f90:162-177
      spin_sums(ginv, o.nw, o.ntop, o.top, 0, o.divide_by_pi, spin[0], spin[1], spin[2]);
  }
  __syncthreads();
  // GRR = (w - eps_t)^-1                                     // :130-131
  // surfstat's spin sums read GRR's leading block as well (src/surfstat.f90:178-192)
  if (invert(ET, grr, (o.spin[0] && !o.spin_right_bottom) ? 0 : 2)) st |= PT_SINGULAR;
  if (tid == 0) {
    for (int q = 0; q < o.nbot; ++q) {
      const int io = N - o.nw + o.bot[q] - 1;
      const double v = ginv(io, io).y;
      dr = o.divide_by_pi ? dr - v / PI_REF : dr - v;
    }
    if (o.spin[0]) {                                          // src/surfstat.f90:178-192
      if (o.spin_right_bottom)                                // src/fermiarc.f90:300-327
        spin_sums(ginv, o.nw, o.nbot, o.bot, N - o.nw, o.divide_by_pi, spin[3], spin[4], spin[5]);
      else
        spin_sums(ginv, o.nw, o.ntop, o.top, 0, o.divide_by_pi, spin[3], spin[4], spin[5]);
    }
  }
  __syncthreads();
  // GB = (w - eps)^-1                                        // :133-134
  if (invert(E, gb, 0)) st |= PT_SINGULAR;
  if (tid == 0) {
    for (int i = 0; i < N; ++i) {
      const double v = ginv(i, i).y;
      db = o.divide_by_pi ? db - v / PI_REF : db - v;
    }
    if (!isfinite(dl) || !isfinite(dr) || !isfinite(db)) st |= PT_NONFINITE;
    emit(dl, dr, db, spin, it, st);
  }
  __syncthreads();
}

