// Per-thread operations of the square-root filter/smoother (one time step,
// one element combine), on thread-private arrays.
//
// Notation: D state dimension, DY observation (ODE) dimension, all matrices
// row-major.  Filter elements are (A, b, U, eta, Z) as in
// pof/parallel_filtsmooth/filter.py:50-81; smoother elements (g, E, Dm) as in
// pof/parallel_filtsmooth/smoother.py:37-50.
#pragma once

#include "pof_linalg.cuh"

namespace pof {

template <typename T>
struct Log2Pi {
  static constexpr T half = T(0.91893853320467274178032973640562);  // log(2 pi) / 2
};

// Running log of a product of |x| (the observation factor's diagonal over a
// chunk's steps): mantissas multiplied, exponents added, one logarithm at the
// end instead of one per step (about 25 FP64 instructions each).
struct LogProd {
  double p = 1.0, extra = 0.0;
  long long e = 0;
  __device__ __forceinline__ void mul(double x) {
    const long long b = __double_as_longlong(x) & 0x7fffffffffffffffLL;
    const int ex = (int)(b >> 52);
    if (ex == 0 || ex == 0x7ff) {
      extra += log(fabs(x));  // zero, subnormal, infinite, NaN
      return;
    }
    p *= __longlong_as_double((b & 0xfffffffffffffLL) | (1023LL << 52));  // p in [1, 4)
    const long long pb = __double_as_longlong(p);
    e += (ex - 1023) + ((int)(pb >> 52) - 1023);
    p = __longlong_as_double((pb & 0xfffffffffffffLL) | (1023LL << 52));
  }
  __device__ __forceinline__ void mul(float x) { extra += (double)logf(fabsf(x)); }
  __device__ __forceinline__ double value() const {
    return log(p) + (double)e * 0.69314718055994530941723212145818 + extra;
  }
};

// E = Phi21 Phi11^{-1} row by row (X: Phi11, lower triangular) and
// g = m - E mp.
template <typename T, int D, int LDX, int LDY>
__device__ __forceinline__ void gain(const T* X, const T* Y, const T* m, const T* mp, T* g, T* E) {
  T rd[D];
#pragma unroll
  for (int i = 0; i < D; ++i) rd[i] = rcp(X[i * LDX + i]);
#pragma unroll
  for (int j = 0; j < D; ++j) {
    T gj = m[j];
#pragma unroll
    for (int i = D - 1; i >= 0; --i) {
      T s = Y[j * LDY + i];
#pragma unroll
      for (int k = i + 1; k < D; ++k) s = fma(-X[k * LDX + i], E[j * D + k], s);
      E[j * D + i] = s * rd[i];
    }
#pragma unroll
    for (int i = 0; i < D; ++i) gj = fma(-E[j * D + i], mp[i], gj);
    g[j] = gj;
  }
}

// The update's small solves: r = H mp + c, wv = -Psi11^{-1} r, the terms
// ||Psi11^{-T} r||^2 (whiten quirk, pof/utils.py:110-112), ||Psi11^{-1} r||^2
// and |Psi11_ii| of sigma^2 and the NLL; m <- mp + Psi21 wv.
template <typename T, int D, int DY, int LDPS>
__device__ __forceinline__ void update_mean(const T* P, const T* H, int h1, const T* c, const T* mp, T* m,
                                            double& ssq, double& yy, LogProd& lp) {
  T r[DY], rd[DY], wv[DY], wq[DY];
#pragma unroll
  for (int i = 0; i < DY; ++i) {
    T s = c[i];
#pragma unroll
    for (int k = 0; k < D; ++k)
      if (k < h1) s = fma(H[i * D + k], mp[k], s);
    r[i] = s;
    rd[i] = rcp(P[i * LDPS + i]);
  }
#pragma unroll
  for (int i = 0; i < DY; ++i) {
    T v = -r[i];
#pragma unroll
    for (int k = 0; k < i; ++k) v = fma(-P[i * LDPS + k], wv[k], v);
    wv[i] = v * rd[i];
  }
  T s2 = T(0), y2 = T(0);
#pragma unroll
  for (int i = DY - 1; i >= 0; --i) {
    T v = r[i];
#pragma unroll
    for (int k = i + 1; k < DY; ++k) v = fma(-P[k * LDPS + i], wq[k], v);
    wq[i] = v * rd[i];
    s2 = fma(wq[i], wq[i], s2);
    y2 = fma(wv[i], wv[i], y2);
    lp.mul(P[i * LDPS + i]);
  }
  ssq += (double)s2;
  yy += (double)y2;
#pragma unroll
  for (int i = 0; i < D; ++i) {
    T acc = mp[i];
#pragma unroll
    for (int k = 0; k < DY; ++k) acc = fma(P[(DY + i) * LDPS + k], wv[k], acc);
    m[i] = acc;
  }
}

// ---------------------------------------------------------------------------
// One square-root Kalman filter step (predict with (F, QL), update with
// (H, c, R)) from the filtered state (m, L) at grid point s, fused with the
// smoother element of grid point s.
//
// Phi = tria([[F L, QL], [L, 0]]) (pof/parallel_filtsmooth/smoother.py:42-46);
// its top block is the predicted chol Lp (sequential_filtsmooth/filter.py:
// 59-66), its bottom right one enters only triangularizations, which take any
// square root, so Dm is that block as the reflectors leave it (not
// triangular).  Psi = tria([[H Lp, R], [Lp, 0]]) (filter.py:69-92).
// Outputs: m, L <- filtered state at s+1; the sums of update_mean; smoother
// element (g, E, Dm) of s when SMOOTH.  Any F, QL, H, R and any square root L.
// ---------------------------------------------------------------------------
template <typename T, int D, int DY, bool SMOOTH>
__device__ __forceinline__ void kf_step(const T* __restrict__ F, const T* __restrict__ QL,
                                        const T* __restrict__ H, const T* __restrict__ c,
                                        const T* __restrict__ R, T* m, T* L, double& ssq, double& yy, LogProd& lp,
                                        T* g, T* E, T* Dm) {
  constexpr int D2 = 2 * D;
  constexpr int DP = D + DY;
  constexpr int MX = SMOOTH ? D2 : D;
  T X[MX * D2];  // [F L, QL] over [L, 0]
  mm<T, D, D, D, D, D, D2>(F, L, X);
  copy<T, D, D, D, D2>(QL, X + D);
  if constexpr (SMOOTH) {
    copy<T, D, D, D, D2>(L, X + D * D2);
    zero<T, D, D, D2>(X + D * D2 + D);
  }
  lq_rows<T, D, MX, D2, D2>(X);
  T mp[D];
  mv<T, D, D, D>(F, m, mp);
  if constexpr (SMOOTH) {
    gain<T, D, D2, D2>(X, X + D * D2, m, mp, g, E);
    copy<T, D, D, D2, D>(X + D * D2 + D, Dm);
  }
  T P[DP * DP];
#pragma unroll
  for (int i = 0; i < DY; ++i) {
#pragma unroll
    for (int j = 0; j < D; ++j) {
      T s = T(0);
#pragma unroll
      for (int k = j; k < D; ++k) s = fma(H[i * D + k], X[k * D2 + j], s);
      P[i * DP + j] = s;
    }
#pragma unroll
    for (int j = 0; j < DY; ++j) P[i * DP + D + j] = R ? R[i * DY + j] : T(0);
  }
#pragma unroll
  for (int i = 0; i < D; ++i)
#pragma unroll
    for (int j = 0; j < DP; ++j) P[(DY + i) * DP + j] = j <= i ? X[i * D2 + j] : T(0);
  lq_rows<T, DP, DP, DP, DP>(P);
  update_mean<T, D, DY, DP>(P, H, D, c, mp, m, ssq, yy, lp);
#pragma unroll
  for (int i = 0; i < D; ++i)
#pragma unroll
    for (int k = 0; k < D; ++k) L[i * D + k] = k <= i ? P[(DY + i) * DP + DY + k] : T(0);
}

// The structure of the solver's model (the IWP prior with exact
// observations), found by the level-0 kernels at run time, for which a step
// leaves out what is zero (the thread form of pof_team.cuh's level 0):
// F block-diagonal with upper-triangular Q x Q blocks, Q = D / DY; QL lower
// triangular; no noise; H reaching the first two columns of the last block at
// most; L lower triangular with NL nonzero columns (D - DY after such a step).
// Level 0 of the small shapes is FP64-pipe bound: a D = 4, d = 1 step has
// 4 + 1 reflectors with tails of 3 and 1 entries, against 4 + 4 + 4 with tails
// of up to 7.
template <int D, int DY>
struct PriorDims {
  static constexpr bool ok = D % DY == 0 && D / DY >= 2;
  static constexpr int Q = ok ? D / DY : D;
  static constexpr int H1 = ok ? (DY - 1) * Q + 2 : D;  // columns of H
};

template <typename T, int D, int DY>
__device__ __forceinline__ bool is_prior(const T* __restrict__ F, const T* __restrict__ QL) {
  if (!PriorDims<D, DY>::ok) return false;
  constexpr int Q = PriorDims<D, DY>::Q;
  bool ok = true;
#pragma unroll
  for (int i = 0; i < D; ++i)
#pragma unroll
    for (int j = 0; j < D; ++j) {
      if (j > i) ok = ok && is_zero(QL[i * D + j]);
      if (j < i || j >= (i / Q + 1) * Q) ok = ok && is_zero(F[i * D + j]);
    }
  return ok;
}

// no noise, and nothing of H beyond the prior's observation columns
template <typename T, int D, int DY>
__device__ __forceinline__ bool is_exact_obs(const T* __restrict__ H, const T* __restrict__ R) {
  bool ok = true;
#pragma unroll
  for (int i = 0; i < DY; ++i)
#pragma unroll
    for (int k = PriorDims<D, DY>::H1; k < D; ++k) ok = ok && is_zero(H[i * D + k]);
  if (R) {
#pragma unroll
    for (int i = 0; i < DY * DY; ++i) ok = ok && is_zero(R[i]);
  }
  return ok;
}

// Predict and observation block of such a step: X <- Phi11 (lower), [Yp | Yw]
// <- the reflected [0 | L] when SMOOTH, P <- Psi (columns 0 .. H1 - 1 of its
// rows; Psi22's columns D - DY).
template <typename T, int D, int DY, int NL, bool SMOOTH>
__device__ __forceinline__ void predict_prior(const T* __restrict__ F, const T* __restrict__ QL,
                                              const T* __restrict__ H, const T* L, T* X, T* Yp, T* Yw, T* P) {
  constexpr int Q = PriorDims<D, DY>::Q, H1 = PriorDims<D, DY>::H1;
  constexpr int NLX = NL > 0 ? NL : 1;
  T W[D * NLX];
#pragma unroll
  for (int i = 0; i < D; ++i) {
#pragma unroll
    for (int j = 0; j < D; ++j) X[i * D + j] = j <= i ? QL[i * D + j] : T(0);
#pragma unroll
    for (int j = 0; j < NL; ++j) {
      T s = T(0);
#pragma unroll
      for (int k = 0; k < D; ++k)
        if (k >= i && k >= j && k < (i / Q + 1) * Q) s = fma(F[i * D + k], L[k * D + j], s);
      W[i * NLX + j] = s;
    }
  }
  if constexpr (SMOOTH) {
#pragma unroll
    for (int i = 0; i < D; ++i) {
#pragma unroll
      for (int j = 0; j < D; ++j) Yp[i * D + j] = T(0);
#pragma unroll
      for (int j = 0; j < NL; ++j) Yw[i * D + j] = L[i * D + j];
    }
    lq_pivot<T, D, NL, D, Q, D, NLX, D, D>(X, W, Yp, Yw);
  } else if constexpr (NL > 0) {
    lq_pivot<T, D, NL, 0, Q, D, NLX, D, D>(X, W, nullptr, nullptr);
  }
#pragma unroll
  for (int i = 0; i < DY; ++i)
#pragma unroll
    for (int j = 0; j < D; ++j) {
      T s = T(0);
#pragma unroll
      for (int k = j; k < H1; ++k) s = fma(H[i * D + k], X[k * D + j], s);
      P[i * D + j] = s;
    }
#pragma unroll
  for (int i = 0; i < D; ++i)
#pragma unroll
    for (int j = 0; j < D; ++j) P[(DY + i) * D + j] = X[i * D + j];
  lq_rows<T, H1 - 1, D + DY, H1, D>(P);
}

// L <- Psi22 of such a step
template <typename T, int D, int DY>
__device__ __forceinline__ void psi22_prior(const T* P, T* L) {
#pragma unroll
  for (int i = 0; i < D; ++i)
#pragma unroll
    for (int k = 0; k < D; ++k) L[i * D + k] = (k <= i && k < D - DY) ? P[(DY + i) * D + (DY + k < D ? DY + k : 0)] : T(0);
}

template <typename T, int D, int DY>
__device__ __forceinline__ void mv_prior(const T* __restrict__ F, const T* x, T* y) {
  constexpr int Q = PriorDims<D, DY>::Q;
#pragma unroll
  for (int i = 0; i < D; ++i) {
    T s = T(0);
#pragma unroll
    for (int k = 0; k < D; ++k)
      if (k >= i && k < (i / Q + 1) * Q) s = fma(F[i * D + k], x[k], s);
    y[i] = s;
  }
}

template <typename T, int D, int DY, int NL, bool SMOOTH>
__device__ __forceinline__ void kf_step_prior(const T* __restrict__ F, const T* __restrict__ QL,
                                              const T* __restrict__ H, const T* __restrict__ c, T* m, T* L,
                                              double& ssq, double& yy, LogProd& lp, T* g, T* E, T* Dm) {
  T X[D * D], P[(D + DY) * D], mp[D];
  if constexpr (SMOOTH) {
    T Yp[D * D];
    predict_prior<T, D, DY, NL, true>(F, QL, H, L, X, Yp, Dm, P);
    mv_prior<T, D, DY>(F, m, mp);
    gain<T, D, D, D>(X, Yp, m, mp, g, E);
#pragma unroll
    for (int i = 0; i < D; ++i)
#pragma unroll
      for (int j = NL; j < D; ++j) Dm[i * D + j] = T(0);
  } else {
    predict_prior<T, D, DY, NL, false>(F, QL, H, L, X, nullptr, nullptr, P);
    mv_prior<T, D, DY>(F, m, mp);
  }
  update_mean<T, D, DY, D>(P, H, PriorDims<D, DY>::H1, c, mp, m, ssq, yy, lp);
  psi22_prior<T, D, DY>(P, L);
}

// One step of the conditional fold that turns the elements of a chunk into
// their combined element (A, b, U, eta, Z): a Kalman filter conditioned on
// the state x at the chunk start, whose mean is affine in x (A x + b) and
// whose observations carry the information (eta, Z Z^T) about x.  Same
// element as folding pof/parallel_filtsmooth/filter.py:50-81 elements with
// the operator of filter.py:117-142.  Start values: A = I, b = 0, L = 0,
// eta = 0, Z = 0 (lower triangular).  fold_finish: everything after the
// step's Psi (in P, leading dimension LDPS), with FA = F A, Fb = F b.
template <typename T, int D, int DY, int LDPS>
__device__ __forceinline__ void fold_finish(const T* P, const T* H, int h1, const T* c, const T* FA, const T* Fb,
                                            T* A, T* b, T* eta, T* Z) {
  T rd[DY], w[DY], W[D * DY];  // w = Psi11^{-1} (H Fb + c), W^T = Psi11^{-1} H FA
#pragma unroll
  for (int i = 0; i < DY; ++i) rd[i] = rcp(P[i * LDPS + i]);
#pragma unroll
  for (int i = 0; i < DY; ++i) {
    T s = c[i];
#pragma unroll
    for (int k = 0; k < D; ++k)
      if (k < h1) s = fma(H[i * D + k], Fb[k], s);
#pragma unroll
    for (int k = 0; k < i; ++k) s = fma(-P[i * LDPS + k], w[k], s);
    w[i] = s * rd[i];
  }
#pragma unroll
  for (int j = 0; j < D; ++j)
#pragma unroll
    for (int i = 0; i < DY; ++i) {
      T s = T(0);
#pragma unroll
      for (int k = 0; k < D; ++k)
        if (k < h1) s = fma(H[i * D + k], FA[k * D + j], s);
#pragma unroll
      for (int k = 0; k < i; ++k) s = fma(-P[i * LDPS + k], W[j * DY + k], s);
      W[j * DY + i] = s * rd[i];
    }
#pragma unroll
  for (int i = 0; i < D; ++i) {
#pragma unroll
    for (int j = 0; j < D; ++j) {
      T acc = FA[i * D + j];
#pragma unroll
      for (int k = 0; k < DY; ++k) acc = fma(-P[(DY + i) * LDPS + k], W[j * DY + k], acc);
      A[i * D + j] = acc;
    }
    T acc = Fb[i], e = eta[i];
#pragma unroll
    for (int k = 0; k < DY; ++k) {
      acc = fma(-P[(DY + i) * LDPS + k], w[k], acc);
      e = fma(-W[i * DY + k], w[k], e);
    }
    b[i] = acc;
    eta[i] = e;
  }
  lq_pivot<T, D, DY, 0, 0, D, DY, D, DY>(Z, W, nullptr, nullptr);  // Z <- tria([Z, W^T])
}

template <typename T, int D, int DY>
__device__ __forceinline__ void cond_fold_step(const T* __restrict__ F, const T* __restrict__ QL,
                                               const T* __restrict__ H, const T* __restrict__ c,
                                               const T* __restrict__ R, T* A, T* b, T* L, T* eta, T* Z) {
  constexpr int D2 = 2 * D;
  constexpr int DP = D + DY;
  T P[DP * DP];
  {
    T X[D * D2];
    mm<T, D, D, D, D, D, D2>(F, L, X);
    copy<T, D, D, D, D2>(QL, X + D);
    lq_rows<T, D, D, D2, D2>(X);
#pragma unroll
    for (int i = 0; i < DY; ++i) {
#pragma unroll
      for (int j = 0; j < D; ++j) {
        T s = T(0);
#pragma unroll
        for (int k = j; k < D; ++k) s = fma(H[i * D + k], X[k * D2 + j], s);
        P[i * DP + j] = s;
      }
#pragma unroll
      for (int j = 0; j < DY; ++j) P[i * DP + D + j] = R ? R[i * DY + j] : T(0);
    }
#pragma unroll
    for (int i = 0; i < D; ++i)
#pragma unroll
      for (int j = 0; j < DP; ++j) P[(DY + i) * DP + j] = j <= i ? X[i * D2 + j] : T(0);
  }
  lq_rows<T, DP, DP, DP, DP>(P);
  T FA[D * D], Fb[D];
  mm<T, D, D, D, D, D, D>(F, A, FA);
  mv<T, D, D, D>(F, b, Fb);
  fold_finish<T, D, DY, DP>(P, H, D, c, FA, Fb, A, b, eta, Z);
#pragma unroll
  for (int i = 0; i < D; ++i)
#pragma unroll
    for (int k = 0; k < D; ++k) L[i * D + k] = k <= i ? P[(DY + i) * DP + DY + k] : T(0);
}

template <typename T, int D, int DY, int NL>
__device__ __forceinline__ void cond_fold_prior(const T* __restrict__ F, const T* __restrict__ QL,
                                                const T* __restrict__ H, const T* __restrict__ c, T* A, T* b, T* L,
                                                T* eta, T* Z) {
  constexpr int Q = PriorDims<D, DY>::Q;
  T P[(D + DY) * D];
  {
    T X[D * D];
    predict_prior<T, D, DY, NL, false>(F, QL, H, L, X, nullptr, nullptr, P);
  }
  T FA[D * D], Fb[D];
#pragma unroll
  for (int i = 0; i < D; ++i)
#pragma unroll
    for (int j = 0; j < D; ++j) {
      T s = T(0);
#pragma unroll
      for (int k = 0; k < D; ++k)
        if (k >= i && k < (i / Q + 1) * Q) s = fma(F[i * D + k], A[k * D + j], s);
      FA[i * D + j] = s;
    }
  mv_prior<T, D, DY>(F, b, Fb);
  fold_finish<T, D, DY, D>(P, H, PriorDims<D, DY>::H1, c, FA, Fb, A, b, eta, Z);
  psi22_prior<T, D, DY>(P, L);
}

// Smoother composite accumulation, pof/parallel_filtsmooth/smoother.py:53-63
// with elem1 = (g1, E1, D1) later in time and elem2 = the running composite
// (g2, E2, D2) earlier in time.  In place on the composite:
// g2 <- E2 g1 + g2, E2 <- E2 E1, D2 <- tria([E2 D1, D2]).  D1 is raw with N1
// nonzero columns; `first`: so is D2 (its own columns), else D2 is triangular.
template <typename T, int D, int N1, bool FIRST>
__device__ __forceinline__ void smooth_combine(const T* __restrict__ g1, const T* __restrict__ E1,
                                               const T* __restrict__ D1, T* g2, T* E2, T* D2m) {
  T gn[D], En[D * D];
  mv<T, D, D, D>(E2, g1, gn);
  constexpr int ND = FIRST ? D : 0;
  constexpr int NX = N1 + ND;  // first: [E2 D1 | D2] without a pivot block
  T X[D * NX];
#pragma unroll
  for (int i = 0; i < D; ++i) {
#pragma unroll
    for (int j = 0; j < N1; ++j) {
      T s = T(0);
#pragma unroll
      for (int k = 0; k < D; ++k) s = fma(E2[i * D + k], D1[k * D + j], s);
      X[i * NX + ND + j] = s;
    }
    if constexpr (FIRST) {
#pragma unroll
      for (int j = 0; j < D; ++j) X[i * NX + j] = D2m[i * D + j];
    }
  }
  if constexpr (FIRST) {
    lq_rows<T, D, D, NX, NX>(X);
#pragma unroll
    for (int i = 0; i < D; ++i)
#pragma unroll
      for (int j = 0; j < D; ++j) D2m[i * D + j] = j <= i ? X[i * NX + j] : T(0);
  } else {
    lq_pivot<T, D, N1, 0, 0, D, NX, D, NX>(D2m, X, nullptr, nullptr);
  }
  mm<T, D, D, D, D, D, D>(E2, E1, En);
#pragma unroll
  for (int i = 0; i < D; ++i) g2[i] += gn[i];
  copy<T, D, D, D, D>(En, E2);
}

// Apply a smoother element, its factor raw with ND nonzero columns, to the
// smoothed state after it: m <- E m + g, L <- tria([E L, Dm]); LOWER: L is
// lower triangular (else any square root).
template <typename T, int D, int ND, bool LOWER>
__device__ __forceinline__ void smooth_apply(const T* __restrict__ g, const T* __restrict__ E,
                                             const T* __restrict__ Dm, T* m, T* L) {
  constexpr int NX = D + ND;
  T mn[D], X[D * NX];
  mv<T, D, D, D>(E, m, mn);
#pragma unroll
  for (int i = 0; i < D; ++i)
#pragma unroll
    for (int j = 0; j < D; ++j) {
      T s = T(0);
#pragma unroll
      for (int k = LOWER ? j : 0; k < D; ++k) s = fma(E[i * D + k], L[k * D + j], s);
      X[i * NX + j] = s;
    }
#pragma unroll
  for (int i = 0; i < D; ++i)
#pragma unroll
    for (int j = 0; j < ND; ++j) X[i * NX + D + j] = Dm[i * D + j];
  lq_rows<T, D, D, NX, NX>(X);
#pragma unroll
  for (int i = 0; i < D; ++i) {
    m[i] = mn[i] + g[i];
#pragma unroll
    for (int j = 0; j < D; ++j) L[i * D + j] = j <= i ? X[i * NX + j] : T(0);
  }
}

// Whether the last N columns of a D x D matrix are zero
template <typename T, int D, int N>
__device__ __forceinline__ bool last_cols_zero(const T* A) {
  bool z = true;
#pragma unroll
  for (int i = 0; i < D; ++i)
#pragma unroll
    for (int j = D - N; j < D; ++j)
      if (j >= 0) z = z && is_zero(A[i * D + j]);
  return z;
}

// Objective term of pof/utils.py:97-101 with the reference's swapped
// arguments: || QL^{-1} (m_k - F m_{k+1}) ||^2.
template <typename T, int D>
__device__ __forceinline__ T objective_term(const T* __restrict__ F, const T* __restrict__ QL,
                                            const T* __restrict__ mk, const T* __restrict__ mk1) {
  T r[D];
  mv<T, D, D, D>(F, mk1, r);
#pragma unroll
  for (int i = 0; i < D; ++i) r[i] = mk[i] - r[i];
  trsv_l<T, D, D>(QL, r);
  T s = T(0);
#pragma unroll
  for (int i = 0; i < D; ++i) s = fma(r[i], r[i], s);
  return s;
}

}  // namespace pof
