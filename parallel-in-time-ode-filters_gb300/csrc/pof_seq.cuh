// Sequential square-root filter and smoother (the reference's sequential
// twin, pof/sequential_filtsmooth/*): the whole trajectory of one problem,
// step after step.  Used for solve(sequential=True)'s linear twin and
// sequential_eks_solve (EKF + RTS).
//
// One block of two warps.  A step is a chain of dependent FP64 instructions
// (64 cycles each on its sub-partition's pipe), so the work of a step is spread
// over a team of 32 lanes with the level-0 operations of pof_team.cuh, zeros
// left out.  Forward, warp 0 runs the filter.  Backward, the smoother element
// (Phi, gain) of step k - 1 depends on the filtered state alone: warp 1 builds
// it, on another sub-partition, while warp 0 applies the element of step k
// (double-buffered, one barrier per step).  One thread per trajectory took
// 125 us per step both ways at D = 6, d = 2.
#pragma once

#include "pof_team_kernels.cuh"

namespace pof {

template <typename T, int D>
struct SeqElem {
  T g[D], E[D * Ld<D>::v], Dm[D * Ld<D>::v];
};

template <typename T, int D, int DY>
struct SeqWs {
  FQ<T, D> fq[2];               // transition model of each warp
  StepKFWs<T, D, DY> kf[2];     // warp 0: filter; warp 1: smoother elements
  SmoTeamWs<T, D> sm;           // warp 0: smoother state
  SeqElem<T, D> el[2];
  T mnext[D], r[D];
};

// EK1 model of a built-in field at the predicted mean F m
// (pof/sequential_filtsmooth/filter.py:9-30, observations.py:35-40).
template <typename T, int TS, int D, int DY>
__device__ __forceinline__ StepObs t_ek1_step(const Team<TS>& tm, StepKFWs<T, D, DY>& w, const T* F, int wf, int field,
                                              const T* __restrict__ params, T p0, T p1) {
  constexpr int Q1 = D / DY, L1 = Ld<D>::v;
  for (int i = tm.r; i < D; i += TS) {
    const int k0 = wf ? i : 0, k1 = wf ? (i / wf + 1) * wf : D;
    T s = T(0);
    for (int k = k0; k < k1; ++k) s = fma(F[i * L1 + k], w.m[k], s);
    w.mp[i] = s;
  }
  tm.sync();
  T y[DY], f[DY], J[DY * DY];
#pragma unroll
  for (int i = 0; i < DY; ++i) y[i] = p0 * w.mp[i * Q1];
  field_eval<T, DY>(field, params, y, f, J);
  if (tm.r == 0) {
#pragma unroll
    for (int i = 0; i < DY * DY; ++i) w.R[i] = J[i];  // (no noise here: R's place is free)
#pragma unroll
    for (int i = 0; i < DY; ++i) w.g[i] = f[i];
  }
  tm.sync();
  int h1 = 0;
  for (int e = tm.r; e < DY * D; e += TS) {
    const int i = e / D, k = e % D;
    T v = k % Q1 == 0 ? -(w.R[i * DY + k / Q1] * p0) : T(0);
    if (k == i * Q1 + 1) v += p1;
    w.H[i * L1 + k] = v;
    if (!is_zero(v)) h1 = max(h1, k + 1);
  }
  h1 = (int)__reduce_max_sync(tm.mask, (unsigned)h1);
  tm.sync();
  for (int i = tm.r; i < DY; i += TS) {
    T hm = T(0);
    for (int k = 0; k < h1; ++k) hm = fma(w.H[i * L1 + k], w.mp[k], hm);
    w.c[i] = (p1 * w.mp[i * Q1 + 1] - w.g[i]) - hm;
  }
  tm.sync();
  return StepObs{h1, true};
}

// The whole sequential filter (+ smoother when `smooth`) of one trajectory.
// FIELD >= 1: EKF; FIELD == 0: the linear filter with the caller's (H, c, R)
// (filter.py:33-56).  scalars[S_NLL] gets +sum log-lik (the sequential twin's
// sign, sequential_filtsmooth/filter.py:23-30), S_SSQ, S_OBJ (smoother).
template <typename T, int D, int DY>
__global__ void __launch_bounds__(64) k_seq_filtsmooth(int64_t n, StepModel sm, int field,
                                                       const T* __restrict__ params, T p0, T p1,
                                                       const T* __restrict__ x0m, const T* __restrict__ x0L,
                                                       int smooth, T* means, T* chols,
                                                       double* __restrict__ scalars) {
  constexpr int TS = 32, L1 = Ld<D>::v, L2 = Ld<2 * D>::v, Q1 = StepDims<T, D, DY>::Q1;
  extern __shared__ __align__(16) unsigned char smem_raw_[];
  SeqWs<T, D, DY>& ws = *reinterpret_cast<SeqWs<T, D, DY>*>(smem_raw_);
  const Team<TS> tm;
  const int warp = threadIdx.x / 32;
  FQ<T, D>& fq = ws.fq[warp];
  StepKFWs<T, D, DY>& w = ws.kf[warp];
  auto load_model = [&](int64_t s, bool objective) {
    t_load_FQ<T, TS, D>(tm, fq, sm, s, Q1);
    tm.sync();
    if (objective) t_inv_lower<T, TS, D>(tm, fq.QL, fq.QLi);
  };
  auto store_state = [&](int64_t g, const T* m, const T* L) {
    for (int f = tm.r; f < D + D * D; f += TS) {
      if (f < D)
        means[g * D + f] = m[f];
      else
        chols[g * D * D + f - D] = L[((f - D) / D) * L1 + (f - D) % D];
    }
  };
  load_model(0, warp == 0);
  if (warp == 0) {
    t_load_state_plain<T, TS, D>(tm, x0m, x0L, w.m, w.L);
    tm.sync();
    store_state(0, w.m, w.L);
    bool lower;
    int nl = t_ncols<T, TS, D, D, L1>(tm, w.L, &lower);
    double ssq = 0.0, yy = 0.0;
    LogProd lp;
    for (int64_t s = 0; s < n; ++s) {
      if (sm.ft_stride && s > 0) load_model(s, false);
      StepObs ob;
      bool ek1 = false;
      if constexpr (Q1 >= 2) {
        if (field != 0) {
          ob = t_ek1_step<T, TS, D, DY>(tm, w, fq.F, fq.wf, field, params, p0, p1);
          ek1 = true;
        }
      }
      if (!ek1) {
        StepView<T, D, DY> v(sm, s);
        ob = t_load_step<T, TS, D, DY>(tm, w, v.H, v.c, v.R);
        tm.sync();
      }
      nl = t_kf_step<T, TS, D, DY, false>(tm, w, fq.F, fq.QL, StepStruct{fq.wq != 0, fq.wf}, ob, nl, lower, ssq, yy,
                                          lp);
      lower = true;
      store_state(s + 1, w.m, w.L);
      tm.sync();
    }
    const double ld = tm.sum(tm.r < DY ? lp.value() : 0.0);
    if (tm.r == 0) {
      scalars[0] = -(0.5 * yy + ld + (double)(n * DY) * Log2Pi<double>::half);
      scalars[1] = 0.0;
      scalars[2] = ssq / (double)n / (double)DY;
    }
    if (smooth) {  // the smoother starts from the terminal state
      t_copy<T, TS, D, D, L1, L1>(tm, w.L, ws.sm.D1);
      for (int i = tm.r; i < D; i += TS) ws.sm.g1[i] = w.m[i];
      if (sm.ft_stride) load_model(n - 1, true);
    }
  }
  if (!smooth) return;
  // backward pass (pof/sequential_filtsmooth/smoother.py:8-48)
  __syncthreads();
  double obj = 0.0;
  bool lower = false;
  for (int64_t k = n; k >= 0; --k) {
    if (warp == 1 && k > 0) {  // element of step k - 1 from its filtered state
      const int64_t e = k - 1;
      if (sm.ft_stride) load_model(e, false);
      t_load_state_plain<T, TS, D>(tm, means + e * D, chols + e * D * D, w.m, w.L);
      tm.sync();
      bool low;
      const int nl = t_ncols<T, TS, D, D, L1>(tm, w.L, &low);
      t_predict_gain<T, TS, D, DY, true>(tm, w, fq.F, fq.QL, StepStruct{fq.wq != 0, fq.wf}, nl, low);
      tm.sync();
      SeqElem<T, D>& el = ws.el[e & 1];
      for (int i = tm.r; i < D; i += TS) el.g[i] = w.g[i];
      for (int f = tm.r; f < D * D; f += TS) {
        const int i = f / D, j = f % D;
        el.E[i * L1 + j] = w.E[i * L1 + j];
        el.Dm[i * L1 + j] = j < nl ? w.Y[i * L2 + D + j] : T(0);
      }
    }
    if (warp == 0 && k < n) {  // apply the element of step k
      SmoTeamWs<T, D>& u = ws.sm;
      const SeqElem<T, D>& el = ws.el[k & 1];
      if (sm.ft_stride && k < n - 1) load_model(k, true);
      for (int i = tm.r; i < D; i += TS) {
        ws.mnext[i] = u.g1[i];
        u.g2[i] = el.g[i];
      }
      t_copy<T, TS, D, D, L1, L1>(tm, el.E, u.E2);
      t_copy<T, TS, D, D, L1, L1>(tm, el.Dm, u.D2m);
      tm.sync();
      t_smooth_apply_raw<T, TS, D>(tm, u, lower);
      lower = true;
      obj += (double)t_objective<T, TS, D>(tm, fq.F, fq.QLi, u.g1, ws.mnext, ws.r, fq.wf);
      store_state(k, u.g1, u.D1);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) scalars[1] = obj;
}

}  // namespace pof
