// fa_solve.cu -- device-side trust-region solver (FP64). Built with -fmad=false: every product and
// sum is rounded separately, in the same order as the CPU statement of the algorithm, so that given
// identical f, g and H the device takes bit-identical steps.
//
// Algorithm (the reference calls dlib::find_min_trust_region at FrameAligner/FrameWarpAligner.cpp:
// 205-209 with objective_delta_stop_strategy(1e-8) and radius 40; dlib's source is not part of the
// reference tree, so this is the project's own statement of the method):
//   outer loop: Nocedal & Wright, Numerical Optimization (2nd ed.), Algorithm 4.1 with eta = 0,
//     Delta_max = 1000; rho < 1/4 shrinks Delta by 4, rho > 3/4 on the boundary doubles it; a
//     rejected step leaves f unchanged, so the |delta f| < 1e-8 rule ends the solve.
//   subproblem: More & Sorensen (1983) Newton iteration on 1/|p(lambda)| - 1/Delta with a
//     safeguarded bracket, eps = 0.1, at most 20 factorisations, using a block-tridiagonal
//     Cholesky of H + lambda I (H = J^T J has n_dim x n_dim blocks, |i - j| <= 1).
#include <float.h>

#include "fa_device.cuh"

namespace fa {

namespace {

constexpr double kDblEps = 2.220446049250313080847e-16;
constexpr double kMinDelta = 1e-8;
constexpr double kRadius0 = 40.0;
constexpr double kRadiusMax = 1000.0;

template <int ND>
struct Band {
  static constexpr int nd = ND;
  const double* Hd;
  const double* Hl;
  int nD, P;
  double hinf, mindiag;  // band_bounds of H
  // band_chol(lambda = 0) computed once per reference (RefDev::L0), or null
  const double* L0 = nullptr;
  const double* inv0 = nullptr;
  int chol0_ok = 0;
};

// Band factor storage: row i of block b holds 2*n_dim entries, the columns of block b-1 then those of
// block b.

// Cholesky of H + lambda I by block rows, fully unrolled over the n_dim x n_dim blocks. Each entry
// L_ij accumulates A_ij (+ lambda) minus L_ik L_jk over ascending k -- the previous block's columns
// first, then the earlier columns of its own block -- which is the dense algorithm's order (its
// other terms are exact zeros). inv[i] = 1 / L_ii; off-diagonal entries multiply by it.
//
// One thread runs this and the two substitutions below: each is a chain of dependent FP64 operations
// whose order is fixed. What one block needs of the previous one stays in registers, and the next
// block's matrix entries are loaded while the current block computes, so that the chain waits for
// arithmetic only, not for a store and a load per row.
template <int ND>
__device__ __forceinline__ int band_chol(const Band<ND>& B, double lambda, double* __restrict__ L,
                                         double* __restrict__ inv) {
  constexpr int NN = ND * ND;
  double Dp[ND][ND];  // previous block's own-column L (rows of block b-1), lower triangle
  double ip[ND];      // and its reciprocal diagonal
  double hd[NN], hl[NN];
#pragma unroll
  for (int i = 0; i < NN; i++) {
    hd[i] = B.Hd[i];
    hl[i] = 0.0;
    Dp[i / ND][i % ND] = 0.0;
  }
#pragma unroll
  for (int r = 0; r < ND; r++) ip[r] = 0.0;
  for (int b = 0; b < B.nD; b++) {
    double hdn[NN], hln[NN];
    if (b + 1 < B.nD) {
#pragma unroll
      for (int i = 0; i < NN; i++) {
        hdn[i] = B.Hd[(b + 1) * NN + i];
        hln[i] = B.Hl[(b + 1) * NN + i];
      }
    }
    const int i0 = b * ND;
    double C[ND][ND];   // L rows of block b, columns of block b-1
    double Dg[ND][ND];  // L rows of block b, its own columns (lower triangle)
    double ic[ND];
#pragma unroll
    for (int r = 0; r < ND; r++)
#pragma unroll
      for (int c = 0; c < ND; c++) {
        double s = hl[r * ND + c];
#pragma unroll
        for (int k = 0; k < c; k++) s -= C[r][k] * Dp[c][k];
        C[r][c] = b > 0 ? s * ip[c] : 0.0;
      }
#pragma unroll
    for (int r = 0; r < ND; r++) {
#pragma unroll
      for (int c = 0; c <= r; c++) {
        double s = hd[r * ND + c] + (r == c ? lambda : 0.0);
        if (b > 0) {
#pragma unroll
          for (int k = 0; k < ND; k++) s -= C[r][k] * C[c][k];
        }
#pragma unroll
        for (int k = 0; k < c; k++) s -= Dg[r][k] * Dg[c][k];
        if (r == c) {
          if (!(s > 0.0)) return -1;
          const double d = sqrt(s);
          Dg[r][r] = d;
          ic[r] = 1.0 / d;
          inv[i0 + r] = ic[r];
        } else {
          Dg[r][c] = s * ic[c];
        }
      }
    }
    // store row i0 + r as [block b-1 columns | block b columns] (2 * ND entries)
#pragma unroll
    for (int r = 0; r < ND; r++) {
      double* row = L + (i0 + r) * 2 * ND;
#pragma unroll
      for (int c = 0; c < ND; c++) {
        row[c] = C[r][c];
        row[ND + c] = c <= r ? Dg[r][c] : 0.0;
        Dp[r][c] = c <= r ? Dg[r][c] : 0.0;
      }
      ip[r] = ic[r];
    }
#pragma unroll
    for (int i = 0; i < NN; i++) {
      hd[i] = hdn[i];
      hl[i] = hln[i];
    }
  }
  return 0;
}

// One block's rows of the factor, their reciprocal diagonal and right-hand side.
template <int ND>
struct FwdBlock {
  double c[ND][ND], d[ND][ND], inv[ND], b[ND];
  __device__ __forceinline__ void load(const double* __restrict__ L, const double* __restrict__ iv,
                                       const double* __restrict__ rhs, int blk) {
#pragma unroll
    for (int r = 0; r < ND; r++) {
      const double* row = L + (blk * ND + r) * 2 * ND;
#pragma unroll
      for (int k = 0; k < ND; k++) c[r][k] = row[k];
#pragma unroll
      for (int k = 0; k < r; k++) d[r][k] = row[ND + k];
      inv[r] = iv[blk * ND + r];
      b[r] = rhs[blk * ND + r];
    }
  }
};

// L y = b by block rows (ascending k per entry, as the dense forward substitution). y may be b.
template <int ND>
__device__ __forceinline__ void band_forward(const Band<ND>& B, const double* __restrict__ L,
                                             const double* __restrict__ inv, const double* b, double* y) {
  double yp[ND];
  FwdBlock<ND> A, N;
  auto step = [&](const FwdBlock<ND>& f, int blk) {
    double yc[ND];
#pragma unroll
    for (int r = 0; r < ND; r++) {
      double s = f.b[r];
      if (blk > 0) {
#pragma unroll
        for (int k = 0; k < ND; k++) s -= f.c[r][k] * yp[k];
      }
#pragma unroll
      for (int k = 0; k < r; k++) s -= f.d[r][k] * yc[k];
      yc[r] = s * f.inv[r];
    }
#pragma unroll
    for (int r = 0; r < ND; r++) {
      y[blk * ND + r] = yc[r];
      yp[r] = yc[r];
    }
  };
#pragma unroll
  for (int r = 0; r < ND; r++) yp[r] = 0.0;
  A.load(L, inv, b, 0);
  for (int blk = 0; blk < B.nD; blk += 2) {
    if (blk + 1 < B.nD) N.load(L, inv, b, blk + 1);
    step(A, blk);
    if (blk + 1 < B.nD) {
      if (blk + 2 < B.nD) A.load(L, inv, b, blk + 2);
      step(N, blk + 1);
    }
  }
}

// One block of the back substitution: its own columns below the diagonal, the next block's rows of
// this block's columns, reciprocal diagonal and right-hand side.
template <int ND>
struct BwdBlock {
  double c[ND][ND], d[ND][ND], inv[ND], b[ND];  // c[k][r] = L(next block row k, column r), d[k][r] = L(row k, r)
  __device__ __forceinline__ void load(const double* __restrict__ L, const double* __restrict__ iv,
                                       const double* __restrict__ y, int blk, bool next) {
#pragma unroll
    for (int k = 0; k < ND; k++) {
      const double* row = L + (blk * ND + k) * 2 * ND;
#pragma unroll
      for (int r = 0; r < k; r++) d[k][r] = row[ND + r];
      if (next) {
#pragma unroll
        for (int r = 0; r < ND; r++) c[k][r] = row[ND * 2 * ND + r];
      }
      inv[k] = iv[blk * ND + k];
      b[k] = y[blk * ND + k];
    }
  }
};

// L^T x = y by block rows from the end (ascending k per entry, as the dense back substitution). x may
// be y.
template <int ND>
__device__ __forceinline__ void band_backward(const Band<ND>& B, const double* __restrict__ L,
                                              const double* __restrict__ inv, const double* y, double* x) {
  double xn[ND];
  BwdBlock<ND> A, N;
  const int last = B.nD - 1;
  auto step = [&](const BwdBlock<ND>& f, int blk) {
    double xc[ND];
#pragma unroll
    for (int r = ND - 1; r >= 0; r--) {
      double s = f.b[r];
#pragma unroll
      for (int k = r + 1; k < ND; k++) s -= f.d[k][r] * xc[k];
      if (blk < last) {
#pragma unroll
        for (int k = 0; k < ND; k++) s -= f.c[k][r] * xn[k];
      }
      xc[r] = s * f.inv[r];
    }
#pragma unroll
    for (int r = 0; r < ND; r++) {
      x[blk * ND + r] = xc[r];
      xn[r] = xc[r];
    }
  };
#pragma unroll
  for (int r = 0; r < ND; r++) xn[r] = 0.0;
  A.load(L, inv, y, last, false);
  for (int blk = last; blk >= 0; blk -= 2) {
    if (blk >= 1) N.load(L, inv, y, blk - 1, true);
    step(A, blk);
    if (blk >= 1) {
      if (blk >= 2) A.load(L, inv, y, blk - 2, true);
      step(N, blk - 1);
    }
  }
}

__device__ double norm2(int n, const double* v) {
  double s = 0;
  for (int i = 0; i < n; i++) s += v[i] * v[i];
  return sqrt(s);
}

template <int ND>
__device__ int subproblem(const Band<ND>& B, const double* g, double radius, double eps, int max_iter, double* p,
                          double* work) {
  const int P = B.P;
  double* L = work;
  double* inv = work + P * 2 * B.nd;
  double* y = inv + P;
  double* rhs = y + P;
  const double gnorm = norm2(P, g);
  if (gnorm == 0.0) {
    for (int i = 0; i < P; i++) p[i] = 0.0;
    return 0;
  }
  const double hinf = B.hinf, mindiag = B.mindiag;
  double lam_hi = gnorm / radius + hinf;
  double lam_lo = gnorm / radius - hinf;
  if (-mindiag > lam_lo) lam_lo = -mindiag;
  if (lam_lo < 0) lam_lo = 0;
  int have_p = 0, boundary = 1;
  double lambda = 0.0;
  for (int i = 0; i < P; i++) rhs[i] = -g[i];
  for (int it = 0; it < max_iter; it++) {
    // H + 0 I is the same matrix for every frame and step of the reference: its factor is computed
    // once (by this same band_chol, so the values are identical) and reused
    const double* Lc = L;
    const double* ic = inv;
    bool ok;
    if (lambda == 0.0 && B.L0 != nullptr) {
      ok = B.chol0_ok != 0;
      Lc = B.L0;
      ic = B.inv0;
    } else {
      ok = band_chol(B, lambda, L, inv) == 0;
    }
    if (!ok) {
      if (lambda > lam_lo) lam_lo = lambda;
      const double a = sqrt(lam_lo * lam_hi), b = lam_lo + 0.001 * (lam_hi - lam_lo);
      lambda = a > b ? a : b;
      continue;
    }
    band_forward(B, Lc, ic, rhs, y);
    band_backward(B, Lc, ic, y, p);
    have_p = 1;
    const double pn = norm2(P, p);
    if (lambda == 0.0 && pn <= radius) {
      boundary = 0;
      break;
    }
    if (fabs(pn - radius) <= eps * radius) break;
    if (pn < radius) {
      if (lambda < lam_hi) lam_hi = lambda;
    } else {
      if (lambda > lam_lo) lam_lo = lambda;
    }
    band_forward(B, Lc, ic, p, y);
    const double qn = norm2(P, y);
    const double r = pn / qn;
    double next = lambda + r * r * (pn - radius) / radius;
    if (!(next > lam_lo && next < lam_hi)) {
      const double a = sqrt(lam_lo * lam_hi), b = lam_lo + 0.001 * (lam_hi - lam_lo);
      next = a > b ? a : b;
    }
    lambda = next;
  }
  if (!have_p) {
    for (int i = 0; i < P; i++) p[i] = -g[i] * (radius / gnorm);
  } else if (boundary) {
    const double pn = norm2(P, p);
    if (pn > radius) {
      const double s = radius / pn;
      for (int i = 0; i < P; i++) p[i] *= s;
    }
  }
  return boundary;
}

// Predicted reduction -(g.p + 0.5 p.H.p) with the dense algorithm's summation order: row i of H p
// sums over ascending j within the band (blocks b-1, b, b+1 of row block b).
template <int ND>
__device__ double predicted(const Band<ND>& B, const double* g, const double* p) {
  constexpr int NN = ND * ND;
  double gp = 0, pHp = 0;
  for (int b = 0; b < B.nD; b++) {
    const double* hl0 = B.Hl + b * NN;        // block (b, b-1)
    const double* hd = B.Hd + b * NN;         // block (b, b)
    const double* hl1 = B.Hl + (b + 1) * NN;  // block (b+1, b), read transposed
#pragma unroll
    for (int a = 0; a < ND; a++) {
      const int i = b * ND + a;
      double s = 0;
      if (b > 0) {
#pragma unroll
        for (int c = 0; c < ND; c++) s += hl0[a * ND + c] * p[(b - 1) * ND + c];
      }
#pragma unroll
      for (int c = 0; c < ND; c++) s += hd[a * ND + c] * p[b * ND + c];
      if (b + 1 < B.nD) {
#pragma unroll
        for (int c = 0; c < ND; c++) s += hl1[c * ND + a] * p[(b + 1) * ND + c];
      }
      gp += g[i] * p[i];
      pHp += p[i] * s;
    }
  }
  return -(gp + 0.5 * pHp);
}

// ------------------------------------------------------------------ the whole block ---------------
//
// What a step needs one thread for is the chain of the two substitutions (3 and up to 7 dependent FP64
// operations a row); everything else is per parameter. The sums whose rounding the algorithm fixes (the
// norms and the predicted reduction) only feed comparisons: they are formed in parallel with an error
// bound, and the ordered sum is taken by one thread only when the bound does not decide the
// comparison. The steps taken are those of the ordered sums, bit for bit.

// How far a sum over P parameters may lie from the ordered one, relative to the sum of magnitudes
// (each order is within P * 2^-53 of the exact sum).
__device__ __forceinline__ double sum_tol(int P) { return 1e-12 + P * 1e-15; }

// Sums of up to three values over the block; every thread gets them. red: 3 doubles per warp, shared.
template <int N>
__device__ __forceinline__ void block_sums(double (&v)[N], double* red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int i = 0; i < N; i++)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
  __syncthreads();  // earlier readers of red are done; the callers' shared stores are visible after the next
  if (lane == 0)
#pragma unroll
    for (int i = 0; i < N; i++) red[w * 3 + i] = v[i];
  __syncthreads();
#pragma unroll
  for (int i = 0; i < N; i++) {
    double a = 0.0;
    for (int k = 0; k < nw; k++) a += red[k * 3 + i];
    v[i] = a;
  }
}

// subproblem by the whole block (g visible to every thread; p visible to every thread on return). An
// interior step -- the first factorisation's (lambda = 0) step inside the radius -- takes the two
// substitutions with the reference's cached factor; anything else goes to subproblem on one thread.
// flag: one int, shared.
template <int ND>
__device__ __forceinline__ int subproblem_block(const Band<ND>& B, const double* g, double radius, double eps,
                                                int max_iter, double* p, double* work, double* red, int* flag) {
  const int P = B.P;
  double* y = work + P * 2 * ND + P;
  double* rhs = y + P;
  double gg[1] = {0.0};
  for (int i = threadIdx.x; i < P; i += blockDim.x) {
    rhs[i] = -g[i];
    gg[0] += g[i] * g[i];
  }
  block_sums(gg, red);
  if (gg[0] == 0.0) {  // squares are not negative: the ordered norm is zero exactly when this sum is
    for (int i = threadIdx.x; i < P; i += blockDim.x) p[i] = 0.0;
    __syncthreads();
    return 0;
  }
  if (B.L0 != nullptr && B.chol0_ok != 0 && max_iter > 0) {
    if (threadIdx.x == 0) {
      band_forward<ND>(B, B.L0, B.inv0, rhs, y);
      band_backward<ND>(B, B.L0, B.inv0, y, p);
    }
    __syncthreads();
    double pp[1] = {0.0};
    for (int i = threadIdx.x; i < P; i += blockDim.x) pp[0] += p[i] * p[i];
    block_sums(pp, red);
    if (pp[0] < radius * radius * (1.0 - 4.0 * sum_tol(P))) return 0;  // |p| <= radius for certain
  }
  if (threadIdx.x == 0) *flag = subproblem<ND>(B, g, radius, eps, max_iter, p, work);
  __syncthreads();
  const int r = *flag;
  __syncthreads();
  return r;
}

// The ratio test of a trial point: measured reduction meas over the predicted reduction, as the ordered
// sums decide it. Returns bits: 1 the solve ends, 2 rho < 1/4, 4 rho > 3/4, 8 rho > 0.
__device__ __forceinline__ int ratio_bits(double pred, double meas) {
  if (fabs(pred) <= fabs(meas) * kDblEps) return 1;
  const double rho = meas / fabs(pred);
  if (!isfinite(rho)) return 1;
  return (rho < 0.25 ? 2 : 0) | (rho > 0.75 ? 4 : 0) | (rho > 0 ? 8 : 0);
}

template <int ND>
__device__ __forceinline__ int ratio_block(const Band<ND>& B, const double* g, const double* p, double meas,
                                           double* red, int* flag) {
  constexpr int NN = ND * ND;
  double v[3] = {0.0, 0.0, 0.0};  // g.p, p.H.p, the sum of their terms' magnitudes
  for (int i = threadIdx.x; i < B.P; i += blockDim.x) {
    const int b = i / ND, a = i - b * ND;
    double s = 0, m = 0;
    auto term = [&](double h, double q) {
      s += h * q;
      m += fabs(h * q);
    };
    if (b > 0) {
#pragma unroll
      for (int c = 0; c < ND; c++) term(B.Hl[b * NN + a * ND + c], p[(b - 1) * ND + c]);
    }
#pragma unroll
    for (int c = 0; c < ND; c++) term(B.Hd[b * NN + a * ND + c], p[b * ND + c]);
    if (b + 1 < B.nD) {
#pragma unroll
      for (int c = 0; c < ND; c++) term(B.Hl[(b + 1) * NN + c * ND + a], p[(b + 1) * ND + c]);
    }
    v[0] += g[i] * p[i];
    v[1] += p[i] * s;
    v[2] += fabs(g[i] * p[i]) + 0.5 * fabs(p[i]) * m;
  }
  block_sums(v, red);
  const double pred = -(v[0] + 0.5 * v[1]), rel = sum_tol(B.P), tol = rel * v[2];
  const double lo = fabs(pred) - tol, hi = fabs(pred) + tol;
  if (lo > 0.0 && isfinite(hi) && isfinite(meas) && fabs(meas) > 1e-200 && fabs(meas) < 1e200 && hi < 1e200 &&
      lo > 1e-200 && lo > 2.0 * fabs(meas) * kDblEps) {
    // the ordered sum lies in [lo, hi]: decided when both ends give the same answer
    const int b0 = ratio_bits(lo * (1.0 - rel), meas), b1 = ratio_bits(hi * (1.0 + rel), meas);
    if (b0 == b1) return b0;
  }
  if (threadIdx.x == 0) *flag = ratio_bits(predicted<ND>(B, g, p), meas);
  __syncthreads();
  const int r = *flag;
  __syncthreads();
  return r;
}

// Doubles of shared memory one frame's solve uses when staged: Hessian blocks, g, p, x and the trial
// gradient, band factor, 1/L_ii and two work vectors, and a copy of the reference's cached factor of H
// and its 1/L_ii, which the chain of every interior step reads.
__host__ __device__ inline long long solve_smem_doubles(int nD, int nd) {
  const long long P = (long long)nD * nd;
  return 2LL * nD * nd * nd + 2 * (P * 2 * nd) + 8 * P;
}

// The trust-region state machine for one frame after a fused pass at its trial point, by the whole
// block. S (shared) is the frame's state; gt the gradient at the trial point, in p the rigid point's
// gradient in the paired start.
template <int ND>
__device__ __forceinline__ void state_step(FrameState& S, const Band<ND>& B, double* x, double* g, double* p,
                                           const double* gt, double* work, double ft, double ft2, double* red,
                                           int* flag) {
  const int P = B.P, t0 = threadIdx.x, nt = blockDim.x;
  const bool lead = threadIdx.x == 0;
  const int phase = S.phase;
  const bool warm = S.use_warm && S.warm != nullptr;
  bool go_top = false, done = false, top = false;
  int next = kPhaseTrial;
  const double f0 = S.f, f_start = S.f_start;
  double radius = S.radius, f = f0;
  int evaluations = S.evaluations + 1, accepted = S.accepted;
  double f_zero = f_start;
  __syncthreads();  // every thread has read the state
  switch (phase) {
    case kPhaseStartZero: {
      f_zero = ft;
      for (int i = t0; i < P; i += nt) g[i] = gt[i];
      bool rigid = false;
#pragma unroll
      for (int c = 0; c < ND; c++) rigid = rigid || (S.rigid[c] != 0.0);
      if (rigid) {
        for (int i = t0; i < P; i += nt) p[i] = S.rigid[i % ND];
        next = kPhaseStartRigid;
      } else {
        f = ft;
        if (warm)
          next = kPhaseWaitWarm;
        else
          go_top = true;
      }
      break;
    }
    case kPhaseStartPair: {
      // Both cold starting points from one pass: ft, gt at zero; ft2 and (in p) its gradient at the
      // rigid shift. The same choice as kPhaseStartZero followed by kPhaseStartRigid.
      evaluations++;
      f_zero = ft;
      if (ft2 < ft) {
        for (int i = t0; i < P; i += nt) {
          x[i] = S.rigid[i % ND];
          g[i] = p[i];
        }
        f = ft2;
      } else {
        for (int i = t0; i < P; i += nt) g[i] = gt[i];
        f = ft;
      }
      if (warm)
        next = kPhaseWaitWarm;
      else
        go_top = true;
      break;
    }
    case kPhaseStartRigid: {
      // Starting points {0, 0, rigid}: std::min_element keeps the first minimum
      // (FrameWarpAligner.cpp:194-198).
      if (ft < f_start) {
        for (int i = t0; i < P; i += nt) {
          x[i] = p[i];
          g[i] = gt[i];
        }
        f = ft;
      } else {
        f = f_start;
      }
      // a warm start waits (out of the passes) until the earlier frame's solution is written; the
      // CTA that builds the next list then sets p = warm - x and the trial point (compact_block)
      if (warm)
        next = kPhaseWaitWarm;
      else
        go_top = true;
      break;
    }
    case kPhaseStartLast: {
      // Warm start: the previous frame's solution as a fourth starting point after {0, 0, rigid};
      // only a strictly smaller value replaces the current start (first minimum kept). The trial
      // point was x + (warm - x), and that is the point taken.
      if (ft < f0) {
        for (int i = t0; i < P; i += nt) {
          x[i] = x[i] + p[i];
          g[i] = gt[i];
        }
        f = ft;
      }
      go_top = true;
      break;
    }
    case kPhaseTrial: {
      const int r = ratio_block<ND>(B, g, p, f0 - ft, red, flag);
      if (r & 1) {
        done = true;
        break;
      }
      if (r & 2) {
        radius *= 0.25;
        if (radius <= kRadius0 * kDblEps) {
          done = true;
          break;
        }
      } else if ((r & 4) && S.boundary) {
        radius = 2 * radius < kRadiusMax ? 2 * radius : kRadiusMax;
      }
      if (r & 8) {
        for (int i = t0; i < P; i += nt) {
          x[i] = x[i] + p[i];
          g[i] = gt[i];
        }
        f = ft;
        accepted++;
      }
      top = true;
      break;
    }
    default:
      done = true;
  }
  __syncthreads();  // x, g, p as this phase leaves them
  int iter = S.iter, have_prev = S.have_prev, hit_max = S.hit_max, boundary = S.boundary;
  double f_prev = S.f_prev;
  if (go_top) {
    radius = kRadius0;
    iter = 0;
    have_prev = 0;
    for (int i = t0; i < P; i += nt) p[i] = 0.0;
    __syncthreads();
  }
  if (go_top || top) {
    // a new trust-region iteration, if the stop rules allow it
    if (S.max_iter > 0 && iter >= S.max_iter) {
      hit_max = 1;
      done = true;
    } else if (have_prev && fabs(f - f_prev) < kMinDelta) {
      done = true;
    } else {
      have_prev = 1;
      f_prev = f;
      iter++;
      boundary = subproblem_block<ND>(B, g, radius, 0.1, 20, p, work, red, flag);
    }
  }
  __syncthreads();  // every thread is done with the old state
  if (lead) {
    S.f = f;
    S.f_start = f_zero;
    S.f_prev = f_prev;
    S.radius = radius;
    S.iter = iter;
    S.accepted = accepted;
    S.evaluations = evaluations;
    S.have_prev = have_prev;
    S.boundary = boundary;
    S.hit_max = hit_max;
    S.phase = done ? kPhaseDone : next;
  }
  __syncthreads();
}

static_assert(sizeof(Job) % 8 == 0 && sizeof(FrameState) % 8 == 0, "copied by words");
template <typename T>
__device__ __forceinline__ void copy_words(T* dst, const T* src) {
  for (int i = threadIdx.x; i < (int)(sizeof(T) / 8); i += blockDim.x)
    reinterpret_cast<unsigned long long*>(dst)[i] = __ldcg(reinterpret_cast<const unsigned long long*>(src) + i);
}

// One trust-region step of one frame per CTA; returns the frame's items in the next fused pass (0: done or
// waiting). The step is latency: a few rounds of dependent loads
// (job, then reference and state, then everything they point at, brought into shared memory when it
// fits), the tile reduction, and the chain of two substitutions; a pass over the frame takes
// longer only for volumes. The chain was the whole step before it ran from registers with its loads
// ahead of it and without the ordered norms (mean over the steps of a solve, before -> after: 22.9 ->
// 9.2 us for a 512 x 512 plane with nD = 32, 58 -> 21 us for 512 x 512 x 16 with nD = 32, 261 -> 90 us
// for 1024 x 1024 x 64 with nD = 64).
template <int ND, bool STAGED>
__device__ __forceinline__ int solve_step(const Job* job_src, double* s_dyn) {
  __shared__ Job job;
  __shared__ FrameState S;
  __shared__ double s_f, s_f2, s_red[3 * (kSolveThreads / 32)];
  __shared__ int s_flag;
  copy_words(&job, job_src);
  __syncthreads();
  copy_words(&S, job.state);
  __syncthreads();
  const RefDev& R = job.R;
  if (S.phase == kPhaseDone || S.phase == kPhaseWaitWarm) return 0;
  const bool pair = S.phase == kPhaseStartPair;
  const int nD = R.nD, P = R.P, nn = ND * ND;
  const bool cached = R.L0 != nullptr;
  Band<ND> B{R.Hd, R.Hl, nD, P, R.h_inf, R.h_mindiag, R.L0, R.inv0, R.chol0_ok};
  double *x = job.x, *g = job.g, *p = job.p, *gt = job.gt, *work = job.work;
  if constexpr (STAGED) {
    double* sHd = s_dyn;
    double* sHl = sHd + nD * nn;
    x = sHl + nD * nn;
    g = x + P;
    p = g + P;
    gt = p + P;
    work = gt + P;
    double* sL0 = work + P * 2 * ND + 3 * P;
    double* sinv0 = sL0 + P * 2 * ND;
    for (int i = threadIdx.x; i < nD * nn; i += blockDim.x) {
      sHd[i] = R.Hd[i];
      sHl[i] = R.Hl[i];
    }
    for (int i = threadIdx.x; i < P; i += blockDim.x) {
      x[i] = job.x[i];
      g[i] = job.g[i];
      p[i] = job.p[i];
    }
    B.Hd = sHd;
    B.Hl = sHl;
    if (cached) {
      for (int i = threadIdx.x; i < P * 2 * ND; i += blockDim.x) sL0[i] = R.L0[i];
      for (int i = threadIdx.x; i < P; i += blockDim.x) sinv0[i] = R.inv0[i];
      B.L0 = sL0;
      B.inv0 = sinv0;
    }
    if (pair) __syncthreads();  // p is loaded before the rigid point's gradient replaces it
  }
  cudaGridDependencySynchronize();  // the fused pass's partial sums (everything above is older)
  cudaTriggerProgrammaticLaunchCompletion();  // the next pass may come in and wait for this launch's end
  if (R.n_tiles > kWideTiles) {  // reduced by the launch before this one (p, too, in the paired start)
    if (threadIdx.x == 0) {
      s_f = job.work[0];
      s_f2 = job.work[1];
    }
    if constexpr (STAGED)
      for (int i = threadIdx.x; i < P; i += blockDim.x) gt[i] = job.gt[i];
    __syncthreads();
  } else {
    reduce_partials(R, job.partials, &s_f, gt);
    // paired start: the rigid point's sums, its gradient into p (free until the first step)
    if (pair) reduce_partials(R, job.partials2, &s_f2, p);
  }
  state_step<ND>(S, B, x, g, p, gt, work, s_f, pair ? s_f2 : 0.0, s_red, &s_flag);
  if constexpr (STAGED) {
    for (int i = threadIdx.x; i < P; i += blockDim.x) {
      job.x[i] = x[i];
      job.g[i] = g[i];
      job.p[i] = p[i];
    }
  }
  for (int i = threadIdx.x; i < (int)(sizeof(FrameState) / 8); i += blockDim.x)
    reinterpret_cast<unsigned long long*>(job.state)[i] = reinterpret_cast<const unsigned long long*>(&S)[i];
  if (S.phase == kPhaseDone) {
    // Finished in this step: report the state and parameters, and keep them as the warm start.
    if (job.report != nullptr) {
      if (threadIdx.x == 0) *static_cast<FrameState*>(job.report) = S;
      double* xr = reinterpret_cast<double*>(static_cast<char*>(job.report) + kReportHeaderBytes);
      for (int i = threadIdx.x; i < P; i += blockDim.x) xr[i] = x[i];
    }
    if (S.warm != nullptr) {
      for (int i = threadIdx.x; i < P; i += blockDim.x) S.warm[i] = x[i];
      // Read by the last CTA of this launch (compact_block) and by later launches: the fence and the count in
      // solve_kernel put the warm start before it for the first.
      if (threadIdx.x == 0 && S.warm_seq != nullptr) *S.warm_seq = S.seq;
    }
    return 0;
  }
  if (S.phase == kPhaseWaitWarm) return 0;
  // Next trial point D = x + p, as the fused pass's control-point parameters.
  write_trial_dparams(job.dparams, x, p, nD, ND, threadIdx.x, blockDim.x);
  return R.n_tiles;
}

// The CTA that finishes last builds the next active list: one launch per iteration fewer than a
// compaction of its own (3.6 us and a launch gap; 6.8 us on a 256-entry table with a frame to resume).
template <int ND, bool STAGED>
__global__ void __launch_bounds__(kSolveThreads, 1) solve_kernel(const Job* __restrict__ jobs,
                                                                 const int* __restrict__ active,
                                                                 const int* __restrict__ n_active, ActiveOut next,
                                                                 unsigned* finished, int end_of_round) {
  extern __shared__ double s_dyn[];
  __shared__ bool s_last;
  // Started early, everything read before the step's wait is older than the pass: the pass waited for the
  // launch before it, and lets this one start only then.
  int na = 1, mine = blockIdx.x;
  if (active != nullptr) {
    na = *n_active;
    mine = active[blockIdx.x];  // within the list's room, whatever its length
    // with no frame active one CTA still ends the round
    if ((int)blockIdx.x >= (finished != nullptr ? max(na, 1) : na)) return;
  }
  const int items = na > 0 ? solve_step<ND, STAGED>(jobs + mine, s_dyn) : 0;
  cudaGridDependencySynchronize();  // (a CTA without a step: the launch never ends before the pass)
  if (finished == nullptr) return;
  if (na > 1 || next.busy != nullptr) {
    __syncthreads();
    if (threadIdx.x == 0) {
      if (next.items != nullptr) next.items[blockIdx.x] = items;
      __threadfence();  // the step's writes before the count
      s_last = atomicAdd(finished, 1u) == (unsigned)max(na, 1) - 1u;
      if (s_last) *finished = 0u;
      __threadfence();
    }
    __syncthreads();
    if (!s_last) return;
    if (next.busy != nullptr)
      compact_block(jobs, next);
    else  // frames only leave a list without busy flags
      list_block(
          na, next, [&](int i) { return ListEntry{active[i], __ldcg(next.items + i), false}; }, [] {});
  } else if (threadIdx.x == 0) {  // the list of one frame, or none
    *next.n_active = items > 0 ? 1 : 0;
    next.active[0] = mine;
    next.prefix[0] = 0;
    next.prefix[1] = items;
  }
  if (end_of_round && threadIdx.x == 0) {
    const int r = *next.rounds + 1;
    *next.rounds = r;
    *next.rounds_host = r;
    cudaGraphSetConditional(next.loop, *next.n_active > 0 && r < next.max_rounds ? 1u : 0u);
  }
}

}  // namespace

namespace {
template <int ND>
cudaError_t launch_solve_nd(const Job* jobs_dev, int n_jobs, int max_nD, cudaStream_t s, const int* active,
                            const int* n_active, const ActiveOut& next, unsigned* finished, int end_of_round,
                            bool overlap) {
  // 328 control points in 3-D, 640 in 2-D. Beyond, a solve is slower (128 x 128 x 16, nD 328 / 329: 1.75 / 2.00 ms).
  constexpr long long kCapBytes = 200 * 1024;
  const long long need = solve_smem_doubles(max_nD, ND) * (long long)sizeof(double);
  if (need > kCapBytes)  // every frame of the launch works in global memory
    return launch_overlapped(solve_kernel<ND, false>, dim3(n_jobs), dim3(kSolveThreads), 0, s, overlap, jobs_dev, active,
                             n_active, next, finished, end_of_round);
  const cudaError_t e = allow_smem<solve_kernel<ND, true>>((size_t)need, (size_t)kCapBytes, 40 * 1024);  // (8 KB are static)
  if (e != cudaSuccess) return e;
  return launch_overlapped(solve_kernel<ND, true>, dim3(n_jobs), dim3(kSolveThreads), (size_t)need, s, overlap, jobs_dev,
                           active, n_active, next, finished, end_of_round);
}
}  // namespace

cudaError_t launch_solve(const Job* jobs_dev, int n_jobs, int max_nD, int n_dim, cudaStream_t s, const int* active,
                         const int* n_active, const ActiveOut* next, unsigned* finished, bool end_of_round, bool overlap) {
  const ActiveOut out = next ? *next : ActiveOut{};
  unsigned* count = next ? finished : nullptr;
  const int end = end_of_round ? 1 : 0;
  return n_dim == 3 ? launch_solve_nd<3>(jobs_dev, n_jobs, max_nD, s, active, n_active, out, count, end, overlap)
                    : launch_solve_nd<2>(jobs_dev, n_jobs, max_nD, s, active, n_active, out, count, end, overlap);
}

// The factor of H itself, once per reference: one block brings the blocks of H into shared memory (when
// they fit) for the chain that one thread runs.
template <int ND>
__global__ void __launch_bounds__(128) chol0_kernel(const double* Hd, const double* Hl, int nD, double* L0, double* inv0,
                                                    int* ok, int staged) {
  extern __shared__ double s_dyn[];
  constexpr int NN = ND * ND;
  Band<ND> B{Hd, Hl, nD, nD * ND, 0.0, 0.0};
  if (staged) {
    for (int i = threadIdx.x; i < nD * NN; i += blockDim.x) {
      s_dyn[i] = Hd[i];
      s_dyn[nD * NN + i] = Hl[i];
    }
    __syncthreads();
    B.Hd = s_dyn;
    B.Hl = s_dyn + nD * NN;
  }
  if (threadIdx.x == 0) *ok = band_chol<ND>(B, 0.0, L0, inv0) == 0;
}

cudaError_t launch_chol0(const double* Hd, const double* Hl, int nD, int nd, double* L0, double* inv0, int* ok,
                         cudaStream_t s) {
  const size_t bytes = (size_t)2 * nD * nd * nd * sizeof(double);
  const int staged = bytes <= 48 * 1024;
  if (nd == 3)
    chol0_kernel<3><<<1, 128, staged ? bytes : 0, s>>>(Hd, Hl, nD, L0, inv0, ok, staged);
  else
    chol0_kernel<2><<<1, 128, staged ? bytes : 0, s>>>(Hd, Hl, nD, L0, inv0, ok, staged);
  return cudaGetLastError();
}

// The subproblem of one frame on given H, g and radius, with the cached factor as the solver has it.
// work: P * (2 * nd) + 3 * P doubles, then the cached factor and its reciprocal diagonal, P * (2 * nd)
// + P doubles.
template <int ND>
__global__ void __launch_bounds__(kSolveThreads) test_subproblem_kernel(const double* Hd, const double* Hl, int nD,
                                                                        double hinf, double mindiag, const double* g,
                                                                        double radius, double* p, int* boundary,
                                                                        double* work) {
  __shared__ double s_red[3 * (kSolveThreads / 32)];
  __shared__ int s_flag, s_ok;
  const int P = nD * ND;
  double* L0 = work + P * 2 * ND + 3 * P;
  double* inv0 = L0 + P * 2 * ND;
  Band<ND> B{Hd, Hl, nD, P, hinf, mindiag};
  if (threadIdx.x == 0) s_ok = band_chol<ND>(B, 0.0, L0, inv0) == 0;
  __syncthreads();
  B.L0 = L0;
  B.inv0 = inv0;
  B.chol0_ok = s_ok;
  const int b = subproblem_block<ND>(B, g, radius, 0.1, 20, p, work, s_red, &s_flag);
  if (threadIdx.x == 0) *boundary = b;
}

cudaError_t launch_test_subproblem(const double* Hd, const double* Hl, int nD, int nd, double hinf, double mindiag,
                                   const double* g, double radius, double* p_out, int* boundary_out, double* work,
                                   cudaStream_t s) {
  if (nd == 3)
    test_subproblem_kernel<3><<<1, kSolveThreads, 0, s>>>(Hd, Hl, nD, hinf, mindiag, g, radius, p_out, boundary_out, work);
  else
    test_subproblem_kernel<2><<<1, kSolveThreads, 0, s>>>(Hd, Hl, nD, hinf, mindiag, g, radius, p_out, boundary_out, work);
  return cudaGetLastError();
}

// The ratio test on given H, g and p for n measured reductions: as the solver takes it, and as the ordered
// sum alone decides it. pred: the ordered predicted reduction.
template <int ND>
__global__ void __launch_bounds__(kSolveThreads) test_ratio_kernel(const double* Hd, const double* Hl, int nD, const double* g,
                                                                   const double* p, const double* meas, int n, double* pred,
                                                                   int* taken, int* ordered) {
  __shared__ double s_red[3 * (kSolveThreads / 32)];
  __shared__ int s_flag;
  const Band<ND> B{Hd, Hl, nD, nD * ND, 0.0, 0.0};
  for (int i = 0; i < n; i++) {
    const int r = ratio_block<ND>(B, g, p, meas[i], s_red, &s_flag);
    if (threadIdx.x == 0) {
      taken[i] = r;
      *pred = predicted<ND>(B, g, p);
      ordered[i] = ratio_bits(*pred, meas[i]);
    }
  }
}

cudaError_t launch_test_ratio(const double* Hd, const double* Hl, int nD, int nd, const double* g, const double* p,
                              const double* meas, int n, double* pred, int* taken, int* ordered, cudaStream_t s) {
  if (nd == 3)
    test_ratio_kernel<3><<<1, kSolveThreads, 0, s>>>(Hd, Hl, nD, g, p, meas, n, pred, taken, ordered);
  else
    test_ratio_kernel<2><<<1, kSolveThreads, 0, s>>>(Hd, Hl, nD, g, p, meas, n, pred, taken, ordered);
  return cudaGetLastError();
}

}  // namespace fa
