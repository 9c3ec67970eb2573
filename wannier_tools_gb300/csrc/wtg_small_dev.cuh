// Lopez-Sancho decimation of a small matrix (Ndim <= 8) by a group of lanes of
// one warp: every matrix lives in registers, one element (Ndim <= 4: 16 lanes, two
// instances a warp) or two (Ndim <= 8: the whole warp) per lane, and lanes read
// each other's elements with shuffles.  No shared memory, no barriers.  A CTA of
// 128 threads per instance kept 16 of its threads busy at Ndim 4 and met three
// barriers per pivot step.  What bounds it: the FP64 pipe (a warp-wide FP64
// instruction takes it 64 cycles per sub-partition whatever lanes take part).
// Every element sees the operations of fp64_solve in the same order, so results
// are those of the CTA-wide kernel bit for bit.
// Included inside an anonymous namespace after wtg_fp64_dev.cuh.
#pragma once

constexpr int SMALL_MAX_N = 8;

// P: padded size (4 or 8).  Element (i, j) sits in lane i + P (j & 3) of the
// group, register j >> 2.
template <int P>
struct Small {
  static constexpr int G = 4 * P;            // lanes of a group
  static constexpr int R = P / 4;            // elements a lane
  typedef double2 Mat[R];

  int N, i, jl, base;                        // this lane's row, column & 3, group's first lane
  __device__ __forceinline__ explicit Small(int n) {
    const int lane = threadIdx.x & 31, l = lane % G;
    N = n;
    i = l % P;
    jl = l / P;
    base = lane - l;
  }
  __device__ __forceinline__ int col(int r) const { return jl + 4 * r; }
  __device__ __forceinline__ static double2 shfl(double2 v, int src) {
    return make_double2(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
  }
  // element (row, column c) where the column is the same for the whole group
  __device__ __forceinline__ double2 at_col(const Mat& m, int row, int c) const {
    const double2 v = R == 1 || c < 4 ? m[0] : m[R - 1];
    return shfl(v, base + row + P * (c & 3));
  }
  // element (row, this lane's column of register r)
  __device__ __forceinline__ double2 at_row(const Mat& m, int row, int r) const {
    return shfl(m[r], base + row + P * jl);
  }
  // any element
  __device__ __forceinline__ double2 at(const Mat& m, int row, int c) const {
    const int src = base + row + P * (c & 3);
    const double2 v0 = shfl(m[0], src);
    if (R == 1) return v0;
    const double2 v1 = shfl(m[R - 1], src);
    return c < 4 ? v0 : v1;
  }
  // out = x y (cta_gemm's order: k ascending, four FMAs a term)
  __device__ __forceinline__ void mul(const Mat& x, const Mat& y, Mat& out) const {
#pragma unroll
    for (int r = 0; r < R; ++r) out[r] = make_double2(0.0, 0.0);
#pragma unroll
    for (int k = 0; k < P; ++k) {
      if (k >= N) break;
      const double2 a = at_col(x, i, k);
#pragma unroll
      for (int r = 0; r < R; ++r) cfma(out[r], a, at_row(y, k, r));
    }
  }
  // w - x, with rev: x's indices in reverse order (gj_load)
  __device__ __forceinline__ void load(const Mat& x, double2 w, bool rev, Mat& m) const {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int j = col(r);
      double2 v = x[r];
      const double2 u = at(x, max(N - 1 - i, 0), max(N - 1 - j, 0));
      if (rev) v = u;
      m[r] = i == j ? make_double2(w.x - v.x, w.y - v.y) : make_double2(-v.x, -v.y);
    }
  }
  // the first maximal |re| + |im| of column c over rows r0 .. r1-1; key 0: all zero
  __device__ __forceinline__ long long pivot(const Mat& m, int c, int r0, int r1, int& p) const {
    const long long own = cabs1_key(R == 1 || c < 4 ? m[0] : m[R - 1]);
    long long best = -1;
    p = r0;
#pragma unroll
    for (int q = 0; q < P; ++q) {
      const long long k = __shfl_sync(0xffffffffu, own, base + q + P * (c & 3));
      if (q >= r0 && q < r1 && k > best) {
        best = k;
        p = q;
      }
    }
    return best;
  }
  __device__ __forceinline__ static void sub(double2& v, double2 f, double2 rk) {
    v.x = fma(-f.x, rk.x, v.x);
    v.x = fma(f.y, rk.y, v.x);
    v.y = fma(-f.x, rk.y, v.y);
    v.y = fma(-f.y, rk.x, v.y);
  }
  // gj_core on rows and columns [o, o + n): inverse (i, j) = m(o + i, o + cols[j]),
  // cols as nibbles.  Returns whether a pivot was exactly zero (m is then the
  // identity there).
  __device__ __forceinline__ bool gj(Mat& m, int o, int n, unsigned& cols) const {
    bool sing = false;
    unsigned perm = 0;
    for (int k = 0; k < n; ++k) {
      const int kk = o + k;
      int p;
      const long long best = pivot(m, kk, kk, o + n, p);
      sing = sing || best == 0;
      perm |= (unsigned)(p - o) << (4 * k);
      const double2 r = crecip(at_col(m, p, kk));
      const double2 f = at_col(m, i == p ? kk : i, kk);
      Mat v;
#pragma unroll
      for (int s = 0; s < R; ++s) {
        const int j = col(s);
        const double2 akj = at_row(m, kk, s), apj = at_row(m, p, s);
        const double2 nk = j == kk ? r : cmul(apj, r);
        double2 x = j == kk ? make_double2(0.0, 0.0) : (i == p ? akj : m[s]);
        sub(x, f, nk);
        v[s] = i == kk ? nk : x;
      }
#pragma unroll
      for (int s = 0; s < R; ++s) {
        const int j = col(s);
        if (!sing && i >= o && i < o + n && j >= o && j < o + n) m[s] = v[s];
      }
    }
    cols = 0x76543210u;
    for (int k = n - 1; k >= 0; --k) {         // undo the row swaps as column swaps
      const int p = (perm >> (4 * k)) & 15;
      const unsigned d = ((cols >> (4 * k)) ^ (cols >> (4 * p))) & 15u;
      cols ^= (d << (4 * k)) | (d << (4 * p));
    }
    if (sing) {
      cols = 0x76543210u;
#pragma unroll
      for (int s = 0; s < R; ++s) m[s] = make_double2(i == col(s) ? 1.0 : 0.0, 0.0);
    }
    return sing;
  }
  // schur_block_invert: the trailing nb x nb block of m^-1 at offset N - nb; false
  // on an exact zero pivot
  __device__ __forceinline__ bool schur(Mat& m, int nb, unsigned& cols) const {
    const int mm = N - nb;
    bool ok = true;
    for (int k = 0; k < mm; ++k) {
      int p;
      ok = pivot(m, k, k, mm, p) != 0 && ok;
      const double2 r = crecip(at_col(m, p, k));
      const double2 f = cmul(at_col(m, i == p ? k : i, k), r);
      Mat v;
#pragma unroll
      for (int s = 0; s < R; ++s) {
        const double2 rk = at_row(m, p, s), mk = at_row(m, k, s);
        double2 x = i == p ? mk : m[s];
        sub(x, f, rk);
        v[s] = x;
      }
#pragma unroll
      for (int s = 0; s < R; ++s)
        if (i > k && col(s) > k) m[s] = v[s];
    }
    return !gj(m, mm, nb, cols) && ok;
  }
};

// One decimation a group, as fp64_solve: H00, H01 column-major, Ndim <= P; a group
// without a point (valid false) takes part in the shuffles only.  Whole warps.
// The results go to emit(dl, dr, db, spin[6], iterations, status) in the group's
// first lane.
template <int P, class O, class Emit>
__device__ __noinline__ void small_solve(int N, double2 w, const O& o, const double2* H00,
                                         const double2* H01, bool valid, Emit emit) {
  typedef Small<P> S;
  typedef typename S::Mat Mat;
  constexpr int R = S::R;
  const S g(N);
  Mat E, ES, ET, Al, Be, G, M1, M2;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int i = g.i, j = g.col(r);
    double2 h = make_double2(0.0, 0.0), a = h, b = h;
    if (valid && i < N && j < N) {
      h = H00[i + j * N];
      a = H01[i + j * N];
      b = H01[j + i * N];
      b.y = -b.y;
    }
    E[r] = ES[r] = ET[r] = h;
    Al[r] = a;
    Be[r] = b;
  }
  int st = 0, it = 0;
  bool conv = false, run = valid;
  for (int itc = 1; itc <= o.itermax; ++itc) {                // src/surfgreen.f90:86
    if (!__any_sync(0xffffffffu, run)) break;
    unsigned cols;
    Mat m;
    g.load(E, w, false, m);
    const bool sing = g.gj(m, 0, N, cols);                    // :88-89
#pragma unroll
    for (int r = 0; r < R; ++r) G[r] = g.at(m, g.i, (cols >> (4 * min(g.col(r), N - 1))) & 15);
    g.mul(Al, G, M1);                                         // :92
    g.mul(Be, G, M2);                                         // :95
    Mat t, u, an, bn;
    g.mul(M1, Be, t);                                         // :98-102
    g.mul(M2, Al, u);                                         // :107-110
    g.mul(M1, Al, an);                                        // :113
    g.mul(M2, Be, bn);                                        // :116
    float part = 0.f;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (run) {
        E[r] = make_double2(E[r].x + t[r].x, E[r].y + t[r].y);
        ES[r] = make_double2(ES[r].x + t[r].x, ES[r].y + t[r].y);
        E[r] = make_double2(E[r].x + u[r].x, E[r].y + u[r].y);
        ET[r] = make_double2(ET[r].x + u[r].x, ET[r].y + u[r].y);
        Al[r] = an[r];
        Be[r] = bn[r];
      }
      if (g.i < N && g.col(r) < N) part += fabsf(d2f_bits(an[r].x)) + fabsf(d2f_bits(an[r].y));
    }
    // the convergence norm (:120-122): FP32 bounds, in FP64 where they do not decide
#pragma unroll
    for (int off = S::G / 2; off > 0; off >>= 1) part += __shfl_xor_sync(0xffffffffu, part, off);
    const double ub = (double)part;
    bool done = ub * (1.0 + 1e-4) + 64 * 3e-38 <= o.tol;
    const bool open = !done && !(ub * 0.7071 * (1.0 - 1e-4) > o.tol);
    if (__any_sync(0xffffffffu, open)) {
      double nrm = 0.0;
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (g.i < N && g.col(r) < N) nrm += sqrt(an[r].x * an[r].x + an[r].y * an[r].y);
#pragma unroll
      for (int off = S::G / 2; off > 0; off >>= 1) nrm += __shfl_xor_sync(0xffffffffu, nrm, off);
      if (open) done = nrm <= o.tol;
    }
    if (run) {
      it = itc;
      if (sing) st |= PT_SINGULAR;
      if (done) {
        conv = true;
        run = false;
      }
    }
  }
  if (!conv) st |= PT_NOT_CONVERGED;

  // GLL, GRR, GB (:127-134) and their sums, as fp64_finals
  double sums[9];
#pragma unroll
  for (int c = 0; c < 9; ++c) sums[c] = 0.0;
  const int m0 = N - o.nw, l = (threadIdx.x & 31) - g.base;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const Mat& X = k == 0 ? ES : k == 1 ? ET : E;
    // surfstat's spin sums read GRR's leading block as well (src/surfstat.f90:178-192)
    int blk = m0 <= 0 || k == 2 ? 0 : k == 0 ? 1 : (o.spin[0] && !o.spin_right_bottom) ? 0 : 2;
    Mat m;
    unsigned cols = 0;
    bool full = blk == 0;
    if (!full) {
      g.load(X, w, blk == 1, m);
      full = !g.schur(m, o.nw, cols);
    }
    if (__any_sync(0xffffffffu, full)) {
      Mat q;
      unsigned cq;
      g.load(X, w, false, q);
      const bool sing = g.gj(q, 0, N, cq);
      if (full) {
        if (sing) st |= PT_SINGULAR;
        cols = cq;
        blk = 0;
#pragma unroll
        for (int r = 0; r < R; ++r) m[r] = q[r];
      }
    }
    auto ginv = [&](int a, int b) {                 // any lane, any entry (block entries if blk)
      if (blk) {
        a = blk == 1 ? o.nw - 1 - a : a - m0;
        b = blk == 1 ? o.nw - 1 - b : b - m0;
      }
      const int off = blk ? m0 : 0;
      a = min(max(a, 0), N - 1 - off);
      b = min(max(b, 0), N - 1 - off);
      return g.at(m, off + a, off + ((cols >> (4 * b)) & 15));
    };
    auto scaled = [&](double v) { return o.divide_by_pi ? v / PI_REF : v; };
    const int n = k == 0 ? o.ntop : k == 1 ? o.nbot : N;
    for (int q0 = 0; q0 < n; q0 += S::G) {          // terms in parallel, subtracted in order
      const int q = min(q0 + l, n - 1);
      const int io = k == 0 ? o.top[q] - 1 : k == 1 ? m0 + o.bot[q] - 1 : q;
      const double v = scaled(ginv(io, io).y);
      for (int x = 0; x < min(S::G, n - q0); ++x)
        sums[k] = sums[k] - __shfl_sync(0xffffffffu, v, g.base + x);
    }
    if (k < 2 && o.spin[0]) {
      const bool top = k == 0 || !o.spin_right_bottom;
      const int off = top ? 0 : m0, ns = top ? o.ntop : o.nbot, nwh = o.nw / 2;
      for (int q0 = 0; q0 < ns; q0 += S::G) {
        const int q = min(q0 + l, ns - 1);
        const int io = off + (top ? o.top[q] : o.bot[q]) - 1, jo = io % o.nw;
        const bool has = jo < 2 * nwh;
        const int partner = !has ? io : jo < nwh ? io + nwh : io - nwh;
        const double sgn = jo < nwh ? 1.0 : -1.0;
        const double2 gp = ginv(io, partner), gd = ginv(io, io);
        double v[3] = {has ? gp.y : 0.0, has ? sgn * gp.x : 0.0, has ? sgn * gd.y : 0.0};
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          v[c] = scaled(v[c]);
          for (int x = 0; x < min(S::G, ns - q0); ++x)
            sums[3 + 3 * k + c] = sums[3 + 3 * k + c] - __shfl_sync(0xffffffffu, v[c], g.base + x);
        }
      }
    }
  }
  if (valid && l == 0) {
    if (!isfinite(sums[0]) || !isfinite(sums[1]) || !isfinite(sums[2])) st |= PT_NONFINITE;
    emit(sums[0], sums[1], sums[2], sums + 3, it, st);
  }
  __syncwarp();
}

// one point whose H00 and H01 sit in workspace matrices 0 and 3 (a batch kernel's
// first warp)
template <class O, class Emit>
__device__ __forceinline__ void small_point(int N, double2 w, const O& o, const double2* W, Emit emit) {
  const bool first = N > 4 || threadIdx.x < 16;
  if (N <= 4) small_solve<4>(N, w, o, W, W + 3 * N * N, first, emit);
  else small_solve<8>(N, w, o, W, W + 3 * N * N, first, emit);
}
