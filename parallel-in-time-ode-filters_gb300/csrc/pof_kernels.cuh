// Kernels of the chunked three-phase square-root filter and smoother.
//
// Time steps s = 0..n-1 (step s maps grid point s to s+1).  Level-0 chunks
// hold C0 consecutive steps; chunk totals form level 1; levels l >= 1 fold C
// consecutive elements into level l+1 until at most a few remain (the top).
// These level-0 kernels assign one thread to one chunk (small D); the team
// kernels (pof_team_kernels.cuh) take larger D and every level above.
//
// Internal buffers of the small shapes (D < 6, one thread per chunk) are
// structure-of-arrays: field f of element e of a level with n elements lives
// at base[f * n + e], so a warp touching 32 consecutive elements issues one
// coalesced access per field.  From D = 6 on a team works on one element, and
// an element's fields are contiguous (base[e * fields + f]): a team then reads
// whole lines, where a field of its own per 32-byte sector cost four times the
// L2 traffic (the sectors' other elements are read steps later, and shared
// memory leaves L1 too small to keep them).  element_index is the rule.
//
// Caller-facing arrays (x0, F, QL, H, c, R, means, chols) keep the
// reference's row-major layouts: H (n, DY, D), c (n, DY), means (n+1, D),
// chols (n+1, D, D).
#pragma once

#include <stdint.h>

#include "pof_fields.cuh"
#include "pof_ops.cuh"

namespace pof {

struct StepModel {
  const void* F;      // (D, D) or (n, D, D)
  const void* QL;     // (D, D) or (n, D, D)
  int64_t ft_stride;  // elements between consecutive steps' F/QL (0: constant)
  const void* H;      // (n, DY, D)
  const void* c;      // (n, DY)
  const void* R;      // (n, DY, DY), (DY, DY) or nullptr (zero)
  int64_t r_stride;   // elements between consecutive steps' R (0: constant)
};

template <int D>
struct FiltLayout {
  static constexpr int A = 0, B = D * D, U = D * D + D, ETA = 2 * D * D + D, Z = 2 * D * D + 2 * D;
  static constexpr int NF = 3 * D * D + 2 * D;
};
template <int D>
struct SmoLayout {
  static constexpr int G = 0, E = D, DM = D + D * D;
  static constexpr int NG = D + 2 * D * D;
};
template <int D>
struct StateLayout {
  static constexpr int M = 0, L = D;
  static constexpr int NS = D + D * D;
};

template <int D, int FIELDS>
__host__ __device__ __forceinline__ int64_t element_index(int f, int64_t e, int64_t n) {
  return D >= 6 ? e * FIELDS + f : f * n + e;
}

// per-chunk partial sums (double accumulators for every T)
enum Partial : int { P_SSQ = 0, P_NLL = 1, P_FOBJ = 2, P_SOBJ = 3, P_NOTCLOSE = 4, P_COUNT = 5 };

template <typename T, int K>
__device__ __forceinline__ void ld_soa(const T* __restrict__ base, int64_t n, int64_t e, T* dst) {
#pragma unroll
  for (int f = 0; f < K; ++f) dst[f] = base[f * n + e];
}
template <typename T, int K>
__device__ __forceinline__ void st_soa(T* __restrict__ base, int64_t n, int64_t e, const T* src) {
#pragma unroll
  for (int f = 0; f < K; ++f) base[f * n + e] = src[f];
}
template <typename T, int K>
__device__ __forceinline__ void ld(const T* __restrict__ src, T* dst) {
#pragma unroll
  for (int f = 0; f < K; ++f) dst[f] = src[f];
}
template <typename T, int K>
__device__ __forceinline__ void st(T* __restrict__ dst, const T* src) {
#pragma unroll
  for (int f = 0; f < K; ++f) dst[f] = src[f];
}

template <typename T, int D, int DY>
struct StepView {
  const T* F;
  const T* QL;
  const T* H;
  const T* c;
  const T* R;
  __device__ __forceinline__ StepView(const StepModel& sm, int64_t s) {
    F = static_cast<const T*>(sm.F) + s * sm.ft_stride;
    QL = static_cast<const T*>(sm.QL) + s * sm.ft_stride;
    H = static_cast<const T*>(sm.H) + s * (DY * D);
    c = static_cast<const T*>(sm.c) + s * DY;
    R = sm.R ? static_cast<const T*>(sm.R) + s * sm.r_stride : nullptr;
  }
};

// ---------------------------------------------------------------------------
// EK1 linearization of a built-in field at means[s+1], s = 0..n-1
// (pof/step.py:12-22 with pof/observations.py:35-40): H = E1 - J(E0 m) E0,
// c = (E1 m - f(E0 m)) - H m, with E0/E1 the Nordsieck-scaled projections
// (pof/convenience.py:26-28): E0 m = p0 * m[i(q+1)], E1 m = p1 * m[i(q+1)+1].
// ---------------------------------------------------------------------------
template <typename T, int D, int DY>
__global__ void k_linearize(int64_t n, int field, const T* __restrict__ params, T p0, T p1,
                            const T* __restrict__ means, T* __restrict__ H, T* __restrict__ c) {
  constexpr int Q1 = D / DY;  // q + 1
  const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (s >= n) return;
  const T* m = means + (s + 1) * D;
  T y[DY], f[DY], J[DY * DY];
#pragma unroll
  for (int i = 0; i < DY; ++i) y[i] = p0 * m[i * Q1];
  field_eval<T, DY>(field, params, y, f, J);
  T h[DY * D];
#pragma unroll
  for (int i = 0; i < DY; ++i) {
#pragma unroll
    for (int k = 0; k < D; ++k) h[i * D + k] = T(0);
#pragma unroll
    for (int j = 0; j < DY; ++j) h[i * D + j * Q1] = -(J[i * DY + j] * p0);
    h[i * D + i * Q1 + 1] += p1;
  }
#pragma unroll
  for (int i = 0; i < DY; ++i) {
    T res = p1 * m[i * Q1 + 1] - f[i];
    T hm = T(0);
#pragma unroll
    for (int k = 0; k < D; ++k) hm = fma(h[i * D + k], m[k], hm);
    c[s * DY + i] = res - hm;
  }
#pragma unroll
  for (int k = 0; k < DY * D; ++k) H[s * DY * D + k] = h[k];
}

// ---------------------------------------------------------------------------
// Level 0 with one thread per chunk (small D: the state fits registers).  A
// step with the prior's structure (is_prior, is_exact_obs) takes the forms that
// leave out its zeros; the transition model is tested once, per step only when
// it varies.
// ---------------------------------------------------------------------------
template <typename T, int D, int DY>
struct ChunkModel {
  const StepModel& sm;
  bool prior;
  __device__ __forceinline__ explicit ChunkModel(const StepModel& sm_) : sm(sm_) {
    prior = sm.ft_stride == 0 && is_prior<T, D, DY>(static_cast<const T*>(sm.F), static_cast<const T*>(sm.QL));
  }
  // whether step v takes the prior's form
  __device__ __forceinline__ bool exact(const StepView<T, D, DY>& v) const {
    const bool p = sm.ft_stride == 0 ? prior : is_prior<T, D, DY>(v.F, v.QL);
    return p && is_exact_obs<T, D, DY>(v.H, v.R);
  }
};

// kf_step in the form that fits; `thin`: the last DY columns of L are zero,
// `lower`: L is lower triangular.
template <typename T, int D, int DY, bool SMOOTH>
__device__ __forceinline__ void kf_step_any(const StepView<T, D, DY>& v, bool exact, bool& thin, bool& lower, T* m,
                                            T* L, double& ssq, double& yy, LogProd& lp, T* g, T* E, T* Dm) {
  if constexpr (PriorDims<D, DY>::ok) {
    if (exact && lower) {
      if (thin)
        kf_step_prior<T, D, DY, D - DY, SMOOTH>(v.F, v.QL, v.H, v.c, m, L, ssq, yy, lp, g, E, Dm);
      else
        kf_step_prior<T, D, DY, D, SMOOTH>(v.F, v.QL, v.H, v.c, m, L, ssq, yy, lp, g, E, Dm);
      thin = true;
      return;
    }
  }
  kf_step<T, D, DY, SMOOTH>(v.F, v.QL, v.H, v.c, v.R, m, L, ssq, yy, lp, g, E, Dm);
  thin = false;
  lower = true;
}

// Filter, phase 1 (level 0): chunk totals.  Chunk 0 runs the filter from x0
// and stores the filtering state as an element with A = 0, eta = 0, Z = 0
// (the operator of filter.py:117-142 reads only b and U of a left operand
// that holds x0); it has a block of its own, so no warp runs both kinds of
// step.  Other chunks run the conditional fold.
template <typename T, int D, int DY>
__global__ void __launch_bounds__(64) k_filt_l0_reduce(int64_t n, int C0, StepModel sm, const T* __restrict__ x0m,
                                                       const T* __restrict__ x0L, T* __restrict__ out, int64_t n1) {
  using FL = FiltLayout<D>;
  const int64_t t = blockIdx.x == 0 ? (threadIdx.x == 0 ? 0 : n1)
                                    : 1 + (blockIdx.x - 1) * (int64_t)blockDim.x + threadIdx.x;
  if (t >= n1) return;
  const int64_t s0 = t * C0;
  const int64_t s1 = (s0 + C0 < n) ? s0 + C0 : n;
  const ChunkModel<T, D, DY> cm(sm);
  T e[FL::NF];
#pragma unroll
  for (int i = 0; i < FL::NF; ++i) e[i] = T(0);
  if (t == 0) {
    T m[D], L[D * D];
    ld<T, D>(x0m, m);
    ld<T, D * D>(x0L, L);
    double ssq = 0.0, yy = 0.0;
    LogProd lp;
    bool thin = false, lower = false;
    for (int64_t s = 0; s < s1; ++s) {
      if (!POF_IN(s, n)) break;
      StepView<T, D, DY> v(sm, s);
      kf_step_any<T, D, DY, false>(v, cm.exact(v), thin, lower, m, L, ssq, yy, lp, nullptr, nullptr, nullptr);
    }
    st<T, D>(e + FL::B, m);
    st<T, D * D>(e + FL::U, L);
  } else {
    T* A = e + FL::A;
    T* b = e + FL::B;
    T* U = e + FL::U;
    T* eta = e + FL::ETA;
    T* Z = e + FL::Z;
#pragma unroll
    for (int i = 0; i < D; ++i) A[i * D + i] = T(1);
    int nl = 0;  // columns of U: none at the start, D - DY after a step of the prior's form
    for (int64_t s = s0; s < s1; ++s) {
      if (!POF_IN(s, n)) break;
      StepView<T, D, DY> v(sm, s);
      bool done = false;
      if constexpr (PriorDims<D, DY>::ok) {
        if (cm.exact(v)) {
          if (nl == 0)
            cond_fold_prior<T, D, DY, 0>(v.F, v.QL, v.H, v.c, A, b, U, eta, Z);
          else if (nl == 1)
            cond_fold_prior<T, D, DY, D - DY>(v.F, v.QL, v.H, v.c, A, b, U, eta, Z);
          else
            cond_fold_prior<T, D, DY, D>(v.F, v.QL, v.H, v.c, A, b, U, eta, Z);
          nl = 1;
          done = true;
        }
      }
      if (!done) {
        cond_fold_step<T, D, DY>(v.F, v.QL, v.H, v.c, v.R, A, b, U, eta, Z);
        nl = 2;
      }
    }
  }
  st_soa<T, FL::NF>(out, n1, t, e);
}

// Filter, phase 3 (level 0): the square-root KF inside chunk t from the state
// at its start; writes the filtered states (grid s0+1..s1, and grid 0 for
// chunk 0), the smoother elements of grid points s0..s1-1 and the chunk's
// partial sums (sigma^2, NLL, filter objective).
template <typename T, int D, int DY>
__global__ void __launch_bounds__(64) k_filt_l0_down(int64_t n, int C0, StepModel sm, const T* __restrict__ states1,
                                                     int64_t n1, T* __restrict__ means, T* __restrict__ chols,
                                                     T* __restrict__ selems, double* __restrict__ partials,
                                                     bool want_fobj) {
  using SL = StateLayout<D>;
  using GL = SmoLayout<D>;
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= n1) return;
  const int64_t s0 = t * C0;
  const int64_t s1 = (s0 + C0 < n) ? s0 + C0 : n;
  const ChunkModel<T, D, DY> cm(sm);
  T st_[SL::NS];
  ld_soa<T, SL::NS>(states1, n1, t, st_);
  T* m = st_ + SL::M;
  T* L = st_ + SL::L;
  if (t == 0) {
    st<T, D>(means, m);
    st<T, D * D>(chols, L);
  }
  double ssq = 0.0, yy = 0.0, fobj = 0.0;
  LogProd lp;
  bool thin = false, lower = t != 0;  // chunk 0 starts from x0, whose chol may be any square root
  T ge[GL::NG];
  for (int64_t s = s0; s < s1; ++s) {
    if (!POF_IN(s, n)) break;
    StepView<T, D, DY> v(sm, s);
    T mold[D];
    ld<T, D>(m, mold);
    kf_step_any<T, D, DY, true>(v, cm.exact(v), thin, lower, m, L, ssq, yy, lp, ge + GL::G, ge + GL::E, ge + GL::DM);
    if (want_fobj) fobj += (double)objective_term<T, D>(v.F, v.QL, mold, m);
    st_soa<T, GL::NG>(selems, n, s, ge);
    st<T, D>(means + (s + 1) * D, m);
    st<T, D * D>(chols + (s + 1) * D * D, L);
  }
  partials[P_SSQ * n1 + t] = ssq;
  partials[P_NLL * n1 + t] = 0.5 * yy + lp.value() + (double)((s1 - s0) * DY) * Log2Pi<double>::half;
  partials[P_FOBJ * n1 + t] = fobj;
}

// ---------------------------------------------------------------------------
// Smoother.  Element k (grid point k = 0..n-1) maps the smoothed state at
// k+1 to the one at k; composites of a range [k0, k1) map the state at k1 to
// the state at k0.  The elements' factors are raw square roots, D - DY columns
// after a step of the prior's form; the composites' are triangular.
// ---------------------------------------------------------------------------
template <typename T, int D, int DY>
__global__ void __launch_bounds__(64) k_smo_l0_reduce(const T* __restrict__ in, int64_t nin, int C,
                                                      T* __restrict__ out, int64_t nout) {
  using GL = SmoLayout<D>;
  constexpr int NT = DY < D ? D - DY : D;
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= nout) return;
  const int64_t i0 = t * C;
  const int64_t i1 = (i0 + C < nin) ? i0 + C : nin;
  T a[GL::NG], b[GL::NG];
  ld_soa<T, GL::NG>(in, nin, i0, a);
  for (int64_t i = i0 + 1; i < i1; ++i) {
    ld_soa<T, GL::NG>(in, nin, i, b);
    const bool thin = NT < D && last_cols_zero<T, D, D - NT>(b + GL::DM);
    if (i == i0 + 1) {
      if (thin)
        smooth_combine<T, D, NT, true>(b + GL::G, b + GL::E, b + GL::DM, a + GL::G, a + GL::E, a + GL::DM);
      else
        smooth_combine<T, D, D, true>(b + GL::G, b + GL::E, b + GL::DM, a + GL::G, a + GL::E, a + GL::DM);
    } else {
      if (thin)
        smooth_combine<T, D, NT, false>(b + GL::G, b + GL::E, b + GL::DM, a + GL::G, a + GL::E, a + GL::DM);
      else
        smooth_combine<T, D, D, false>(b + GL::G, b + GL::E, b + GL::DM, a + GL::G, a + GL::E, a + GL::DM);
    }
  }
  if (i1 - i0 == 1) {
    T* X = a + GL::DM;
    lq_rows<T, D, D, D, D>(X);
#pragma unroll
    for (int i = 0; i < D; ++i)
#pragma unroll
      for (int j = i + 1; j < D; ++j) X[i * D + j] = T(0);
  }
  st_soa<T, GL::NG>(out, nout, t, a);
}

// Smoother, phase 3 (level 0): backward recursion inside chunk t from the
// smoothed state at its end.  Writes smoothed means and chols (chols scaled
// by *scale when scale != nullptr), and partial sums of the smoother
// objective and of the convergence test against means_old.
template <typename T, int D, int DY>
__global__ void __launch_bounds__(64) k_smo_l0_down(int64_t n, int C0, const T* __restrict__ F,
                                                    const T* __restrict__ QL, int64_t ft_stride,
                                                    const T* __restrict__ selems, const T* __restrict__ ends1,
                                                    int64_t n1, T* __restrict__ means, T* __restrict__ chols,
                                                    const T* __restrict__ scale, const T* __restrict__ means_old,
                                                    double c_mrtol, double c_matol, double* __restrict__ partials) {
  using SL = StateLayout<D>;
  using GL = SmoLayout<D>;
  constexpr int NT = DY < D ? D - DY : D;
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= n1) return;
  const int64_t s0 = t * C0;
  const int64_t s1 = (s0 + C0 < n) ? s0 + C0 : n;
  const T sc = scale ? *scale : T(1);
  T st_[SL::NS];
  ld_soa<T, SL::NS>(ends1, n1, t, st_);
  T* m = st_ + SL::M;
  T* L = st_ + SL::L;
  double sobj = 0.0;
  int notclose = 0;
  auto close_count = [&](int64_t k, const T* mk) {
    if (!means_old) return;
#pragma unroll
    for (int i = 0; i < D; ++i) {
      const double a = (double)means_old[k * D + i], b = (double)mk[i];
      bool ok;
      if (isfinite(a) && isfinite(b))
        ok = fabs(a - b) <= c_matol + c_mrtol * fabs(b);
      else
        ok = (a == b);
      notclose += ok ? 0 : 1;
    }
  };
  if (s1 == n) {  // the terminal grid point n belongs to the last chunk
    close_count(n, m);
    if (scale) {
#pragma unroll
      for (int i = 0; i < D * D; ++i) chols[n * D * D + i] = L[i] * sc;
    }
  }
  T ge[GL::NG];
  bool lower = s1 != n;  // the terminal state may be the caller's, with any square root
  for (int64_t k = s1 - 1; k >= s0; --k) {
    if (!POF_IN(k, n)) break;
    T mnext[D];
    ld<T, D>(m, mnext);
    ld_soa<T, GL::NG>(selems, n, k, ge);
    if (lower && NT < D && last_cols_zero<T, D, D - NT>(ge + GL::DM))
      smooth_apply<T, D, NT, true>(ge + GL::G, ge + GL::E, ge + GL::DM, m, L);
    else
      smooth_apply<T, D, D, false>(ge + GL::G, ge + GL::E, ge + GL::DM, m, L);
    lower = true;
    sobj += (double)objective_term<T, D>(F + k * ft_stride, QL + k * ft_stride, m, mnext);
    close_count(k, m);
    st<T, D>(means + k * D, m);
    if (scale) {
#pragma unroll
      for (int i = 0; i < D * D; ++i) chols[k * D * D + i] = L[i] * sc;
    } else {
      st<T, D * D>(chols + k * D * D, L);
    }
  }
  partials[P_SOBJ * n1 + t] = sobj;
  partials[P_NOTCLOSE * n1 + t] = (double)notclose;
}

// Fixed-order sum of per-chunk partials (deterministic: the same sums in the
// same order on every run).  One block of 256 threads: thread j sums chunks
// j, j+256, ... in order, then a fixed pairwise tree.
template <int NT>
__device__ __forceinline__ double block_sum_fixed(const double* __restrict__ v, int64_t n) {
  __shared__ double red[NT];
  double s = 0.0;
  for (int64_t i = threadIdx.x; i < n; i += NT) s += v[i];
  red[threadIdx.x] = s;
  __syncthreads();
#pragma unroll
  for (int w = NT / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  const double r = red[0];
  __syncthreads();
  return r;
}

}  // namespace pof
