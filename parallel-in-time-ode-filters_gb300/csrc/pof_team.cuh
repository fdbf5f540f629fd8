// Team-cooperative small-matrix operations: a team of TS lanes of one warp
// (TS = 8, 16 or 32) works on one element combine, matrices in shared
// memory, one matrix row per lane where rows are independent.
//
// Used where there are too few independent combines to give every lane its
// own (the levels >= 1 of the chunked scan, and the single-team top): on a
// GB300 SM a warp instruction occupies the FP64 pipe for ~64 cycles however
// few lanes are active, so a combine spread over TS lanes finishes up to TS
// times sooner than one run by a single lane.
//
// Independent operations of the same shape inside a combine (the two
// triangularizations U and Z, the two triangular solves M and Mu of the
// filter operator) run side by side on the two halves of the team: one
// instruction stream, different operands, half the FP64 instructions.
//
// Layout: row-major with an odd leading dimension (LD = cols + 1 for even
// cols) so the lanes of a team reading one column hit distinct banks.
#pragma once

#include "pof_ops.cuh"

namespace pof {

template <int TS>
struct Team {
  unsigned mask;
  int r;  // lane index inside the team
  __device__ __forceinline__ Team() {
    const int lane = threadIdx.x & 31;
    r = lane % TS;
    if constexpr (TS == 32)
      mask = 0xffffffffu;
    else
      mask = ((1u << TS) - 1u) << (lane / TS * TS);
  }
  __device__ __forceinline__ void sync() const { __syncwarp(mask); }
  template <typename T>
  __device__ __forceinline__ T sum(T v) const {
#pragma unroll
    for (int o = TS / 2; o > 0; o >>= 1) v += __shfl_xor_sync(mask, v, o, TS);
    return v;
  }
};

// odd leading dimension for a row of `cols` doubles
template <int COLS>
struct Ld {
  static constexpr int v = (COLS % 2 == 0) ? COLS + 1 : COLS;
};

// C(MxN) = op(A) op(B): lanes split the M*N outputs.
// TA: A is stored transposed (K x M, leading dim LDA); TB: B stored as (N x K).
template <typename T, int TS, int M, int K, int N, int LDA, int LDB, int LDC, bool TA = false, bool TB = false>
__device__ __forceinline__ void t_mm(const Team<TS>& tm, const T* A, const T* B, T* C) {
  for (int idx = tm.r; idx < M * N; idx += TS) {
    const int i = idx / N, j = idx % N;
    Acc<T> s(T(0));
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const T a = TA ? A[k * LDA + i] : A[i * LDA + k];
      const T b = TB ? B[j * LDB + k] : B[k * LDB + j];
      s.mul_add(a, b);
    }
    C[i * LDC + j] = s.value();
  }
}

// ---------------------------------------------------------------------------
// LQ with a triangular pivot block.  Rows [P | W] (M rows, pivot entry (j, j)
// of row j in column j, tail columns [kb(j), ke(j)) given by `tail`) and MB
// more rows Y in the same columns below: reflector j combines pivot column j
// with row j's tail, so that afterwards the pivot block is L (lower
// triangular, L L^T = P P^T + W W^T) and the rows Y have been multiplied by
// the same orthogonal matrix.  The tails of the M rows (zero in exact
// arithmetic) are not cleared and must not be read.
//
// This is every triangularization of the filter and smoother: tria([X, L])
// with a lower-triangular L is [P | W] = [L | X] (TailFixed), a general
// matrix is P = W with the tail right of the diagonal (TailUpper).
//
// GB300 issues one FP64 instruction per warp and 64 cycles on each of the
// SM's sub-partitions, whatever its lanes do and whether it depends on the
// one before (measured: 64.4 cycles dependent or independent, 1 or 32 lanes,
// and 76 once all four sub-partitions issue), so the cost of a reflector is
// its count of FP64 instructions plus what does not overlap with them.  The
// row's own squared norm is therefore one more of the dot products (entry 0),
// the scalars are computed by every lane instead of on one and broadcast (the
// same instructions), the tail is not rescaled, and one team barrier per
// reflector is left where a row belongs to one lane.  An exactly zero tail
// (LAPACK's tau = 0) skips the reflector.
//
// Entries (the reflector's row and the rows below) are spread over RS row
// slots; a team with more lanes than entries gives each row G = TS / RS
// lanes, which take every G-th tail column.  All of them need the row's pivot
// entry and the first writes it, so a second barrier separates the two.
// ---------------------------------------------------------------------------
template <int R>
struct Pow2Ceil {
  static constexpr int v = R <= 1 ? 1 : (R <= 2 ? 2 : (R <= 4 ? 4 : (R <= 8 ? 8 : (R <= 16 ? 16 : 32))));
};

template <int KB, int KE>
struct TailFixed {  // the same columns for every reflector
  static constexpr int count = KE - KB;
  __device__ __forceinline__ void operator()(int, int& b, int& e) const { b = KB, e = KE; }
};
struct TailRange {  // the same columns for every reflector, found at run time
  static constexpr int count = 0;  // not a constant
  int kb, ke;
  __device__ __forceinline__ void operator()(int, int& b, int& e) const { b = kb, e = ke; }
};
// [L | F S] with a block-diagonal F (blocks of Q) and a lower-triangular S of
// `n` nonzero columns: row j of F S, in block j / Q, has no entry beyond
// column (j / Q + 1) Q - 1, and the reflectors before j fill no further.
// Q = 0: no such structure.
template <int Q>
struct TailBlocks {
  static constexpr int count = 0;
  int kb, n;
  __device__ __forceinline__ void operator()(int j, int& b, int& e) const {
    int w = n;
    if constexpr (Q > 0) w = min((j / Q + 1) * Q, n);
    b = kb, e = kb + w;
  }
};
struct TailUpper {  // the columns right of the diagonal, up to `n`
  static constexpr int count = 0;  // not a constant
  int n;
  __device__ __forceinline__ void operator()(int j, int& b, int& e) const { b = j + 1, e = n; }
};

template <typename T, int TS, int M, int MB, int LD, int LDY, typename Tail>
__device__ __forceinline__ void t_lq(const Team<TS>& tm, T* X, T* Y, const Tail& tail, int mlim = M) {
  constexpr int NE = M + MB;
  constexpr int RS = Pow2Ceil<NE>::v < TS ? Pow2Ceil<NE>::v : TS;
  constexpr int G = TS / RS;
  constexpr int NP = (NE + RS - 1) / RS;
  const int src = (threadIdx.x & 31) / TS * TS;  // lane 0 of this team within the warp
  const int slot = tm.r % RS, ph = tm.r / RS;
  T pend = T(0);  // diagonal of the reflector before, written once every lane has read it
  int pj = -1;
#pragma unroll 1
  for (int j = 0; j < mlim; ++j) {
    int kb, ke;
    tail(j, kb, ke);
    if (kb >= ke) continue;
    tm.sync();
    if (pj >= 0 && tm.r == 0) X[pj * LD + pj] = pend;
    T* xj = X + j * LD;
    const T alpha = xj[j];
    const int ne = M - j + MB;  // entries of this reflector; pass p has one if p RS < ne
    T* row[NP];
    T piv[NP];
    Acc<T> dot[NP];
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      const int e = slot + p * RS;
      row[p] = e >= ne ? X + j * LD : (e < M - j ? X + (j + e) * LD : Y + (e - (M - j)) * LDY);
      piv[p] = row[p][j];
      dot[p] = Acc<T>(T(0));
    }
    if constexpr (Tail::count > 0 && Tail::count % G == 0) {
#pragma unroll
      for (int t = 0; t < Tail::count; t += G) {
        const T x = xj[kb + ph + t];
#pragma unroll
        for (int p = 0; p < NP; ++p)
          if (p == 0 || p * RS < ne) dot[p].mul_add(row[p][kb + ph + t], x);
      }
    } else {
#pragma unroll 2
      for (int k = kb + ph; k < ke; k += G) {
        const T x = xj[k];
#pragma unroll
        for (int p = 0; p < NP; ++p)
          if (p == 0 || p * RS < ne) dot[p].mul_add(row[p][k], x);
      }
    }
#pragma unroll
    for (int o = RS; o < TS; o <<= 1)
#pragma unroll
      for (int p = 0; p < NP; ++p) dot[p].join(tm.mask, o, TS);
    const T xn2 = __shfl_sync(tm.mask, dot[0].value(), src);
    pj = -1;
    if (is_zero(xn2)) continue;
    // a row's G lanes have read its pivot entry before the first of them writes it
    if constexpr (G > 1) tm.sync();
    Reflector<T> h;
    h.set(alpha, xn2, [&](T s) {  // (every lane has the same xn2)
#pragma unroll
      for (int p = 0; p < NP; ++p) dot[p].scale(s);
      tm.sync();
      for (int k = kb + tm.r; k < ke; k += TS) xj[k] *= s;
      tm.sync();
    });
    pend = h.beta;
    pj = j;
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      const int e = slot + p * RS;
      if (e == 0 || e >= ne) continue;
      T* xi = row[p];
      T ws;
      const T a = h.row(piv[p], dot[p].value(), ws);
      if (ph == 0) xi[j] = a;
      if constexpr (Tail::count > 0 && Tail::count % G == 0) {
#pragma unroll
        for (int t = 0; t < Tail::count; t += G) xi[kb + ph + t] = fma(-ws, xj[kb + ph + t], xi[kb + ph + t]);
      } else {
#pragma unroll 2
        for (int k = kb + ph; k < ke; k += G) xi[k] = fma(-ws, xj[k], xi[k]);
      }
    }
  }
  tm.sync();
  if (pj >= 0 && tm.r == 0) X[pj * LD + pj] = pend;
  tm.sync();
}

// The sum (op(A) x)(i) for row i = lane's row slot, A given by its row and
// column strides; G = TS / slots lanes share a row's terms, every lane of a
// slot gets the sum (slots beyond M: row 0's).
template <typename T, int TS, int M, int K>
__device__ __forceinline__ Acc<T> t_dotrow(const Team<TS>& tm, const T* A, int rs, int cs, const T* x) {
  constexpr int RS = Pow2Ceil<M>::v < TS ? Pow2Ceil<M>::v : TS;
  constexpr int G = TS / RS;
  static_assert(M <= RS, "one row per lane");
  const int i = tm.r % RS < M ? tm.r % RS : 0;
  Acc<T> s(T(0));
#pragma unroll
  for (int k0 = 0; k0 < K; k0 += G) {
    const int k = k0 + tm.r / RS;
    if (K % G == 0 || k < K) s.mul_add(A[i * rs + k * cs], x[k]);
  }
#pragma unroll
  for (int o = RS; o < TS; o <<= 1) s.join(tm.mask, o, TS);
  return s;
}

// C(M x N) = A(M x N) B with B (N x N) lower triangular: column group t of
// the outputs starts its sum at the group's first column (terms above B's
// diagonal are exact zeros), one row per lane slot.
template <typename T, int TS, int M, int N, int LDA, int LDB, int LDC>
__device__ __forceinline__ void t_mm_lowB(const Team<TS>& tm, const T* A, const T* B, T* C) {
  constexpr int RS = Pow2Ceil<M>::v < TS ? Pow2Ceil<M>::v : TS;
  constexpr int CG = TS / RS;
#pragma unroll
  for (int i0 = 0; i0 < M; i0 += RS) {
    const int i = i0 + tm.r % RS;
    if (M % RS != 0 && i >= M) continue;
#pragma unroll
    for (int t = 0; t < N; t += CG) {
      const int j = t + tm.r / RS;
      if (N % CG != 0 && j >= N) continue;
      Acc<T> s(T(0));
#pragma unroll
      for (int k = t; k < N; ++k) s.mul_add(A[i * LDA + k], B[k * LDB + j]);
      C[i * LDC + j] = s.value();
    }
  }
}

// 1 / L_ii for i = 0..M-1, computed in parallel (lane i) and read by every
// lane through a shuffle: each division is done once per team, not once per
// right-hand side.
template <typename T, int TS, int M, int LDL>
__device__ __forceinline__ T t_recip_diag(const Team<TS>& tm, const T* L) {
  static_assert(M <= TS, "t_recip_diag needs M <= TS");
  return (tm.r < M) ? rcp(L[tm.r * LDL + tm.r]) : T(0);
}

// B(M x NR) <- L^{-1} B (lower L): one right-hand-side column per lane.
template <typename T, int TS, int M, int NR, int LDL, int LDB>
__device__ __forceinline__ void t_trsm_l(const Team<TS>& tm, const T* L, T* B) {
  if constexpr (M <= TS) {
    const int src = (threadIdx.x & 31) / TS * TS;
    const T rd = t_recip_diag<T, TS, M, LDL>(tm, L);
    T rdi[M];
#pragma unroll
    for (int i = 0; i < M; ++i) rdi[i] = __shfl_sync(tm.mask, rd, src + i);
    for (int j = tm.r; j < NR; j += TS) {
#pragma unroll
      for (int i = 0; i < M; ++i) {
        Acc<T> s(B[i * LDB + j]);
#pragma unroll
        for (int k = 0; k < i; ++k) s.mul_add(-L[i * LDL + k], B[k * LDB + j]);
        B[i * LDB + j] = s.value() * rdi[i];
      }
    }
  } else {
    for (int j = tm.r; j < NR; j += TS) {
#pragma unroll
      for (int i = 0; i < M; ++i) {
        Acc<T> s(B[i * LDB + j]);
#pragma unroll
        for (int k = 0; k < i; ++k) s.mul_add(-L[i * LDL + k], B[k * LDB + j]);
        B[i * LDB + j] = s.value() * rcp(L[i * LDL + i]);
      }
    }
  }
}

template <typename T, int TS, int M, int N, int LDS, int LDD, bool TR = false>
__device__ __forceinline__ void t_copy(const Team<TS>& tm, const T* S, T* Dst) {
  for (int idx = tm.r; idx < M * N; idx += TS) {
    const int i = idx / N, j = idx % N;
    Dst[i * LDD + j] = TR ? S[j * LDS + i] : S[i * LDS + j];
  }
}

template <typename T, int TS, int M, int N, int LDD>
__device__ __forceinline__ void t_fill(const Team<TS>& tm, T* Dst, T v, T diag) {
  for (int idx = tm.r; idx < M * N; idx += TS) {
    const int i = idx / N, j = idx % N;
    Dst[i * LDD + j] = (i == j) ? diag : v;
  }
}

// ---------------------------------------------------------------------------
// Element operations (same formulas as pof_ops.cuh, team-parallel)
// ---------------------------------------------------------------------------

// Shared-memory workspace of one team for the filter operations.
template <typename T, int D>
struct FiltTeamWs {
  static constexpr int D2 = 2 * D;
  static constexpr int LD2 = Ld<D2>::v;
  static constexpr int LD1 = Ld<D>::v;
  // element 1 (running) and element 2 (incoming): A, U, Z (D x LD1), b, eta (D)
  T A1[D * LD1], U1[D * LD1], Z1[D * LD1], b1[D], e1[D];
  T A2[D * LD1], U2[D * LD1], Z2[D * LD1], b2[D], e2[D];
  T Xt[D * LD2], Xb[D * LD2];  // [U1^T Z2, I] and [Z2, 0] -> Xi
  T M[D * LD1], Mu[D * LD1], W[D * LD1];
  T UX[D * LD2];
  T v1[D], v2[D], v3[D], v4[D];
};

// Xi = tria([[U1^T Z2, I], [Z2, 0]]) as [P | W] = [I | U1^T Z2] over
// [0 | Z2]: Xi11 = Xt[:, :D], Xi21 = Xb[:, :D], and Xb[:, D:] is Xi22 before
// its own triangularization -- its only use is Z = tria([A1^T Xi22, Z1]),
// which takes any square root, so that triangularization (a third of the
// operator's reflectors) is not done.  M = Xi11^{-1} U1^T A2^T and
// Mu = Xi11^{-1} U1^T follow; both vector chains of the operator use Mu:
// m^T Xi21^T = Mu^T Xi21^T and e^T U1^T = Xi21 Mu (e = Xi11^{-T} Xi21^T).
template <typename T, int TS, int D>
__device__ __forceinline__ void t_filt_xi(const Team<TS>& tm, FiltTeamWs<T, D>& w) {
  using W = FiltTeamWs<T, D>;
  constexpr int L1 = W::LD1, L2 = W::LD2;
  t_mm<T, TS, D, D, D, L1, L1, L2, true, false>(tm, w.U1, w.Z2, w.Xt + D);
  t_fill<T, TS, D, D, L2>(tm, w.Xt, T(0), T(1));
  t_copy<T, TS, D, D, L1, L2>(tm, w.Z2, w.Xb + D);
  t_fill<T, TS, D, D, L2>(tm, w.Xb, T(0), T(0));
  t_lq<T, TS, D, D, L2, L2>(tm, w.Xt, w.Xb, TailFixed<D, 2 * D>{});
  t_mm<T, TS, D, D, D, L1, L1, L1, true, true>(tm, w.U1, w.A2, w.M);
  t_copy<T, TS, D, D, L1, L1, true>(tm, w.U1, w.Mu);
  tm.sync();
  {  // M and Mu side by side on the two halves of the team
    const Team<TS / 2> h;
    t_trsm_l<T, TS / 2, D, D, L2, L1>(h, w.Xt, tm.r >= TS / 2 ? w.Mu : w.M);
  }
  tm.sync();
}

// e1 <- e1 (x) e2 (pof/parallel_filtsmooth/filter.py:117-142)
//
// Latency-bound on the tree's upper levels (FP64 instructions of one warp,
// 64 cycles each).  Per combine on a 32-lane team at D = 8 about 530 FP64
// instructions, from about 1060 with Xi22 triangularized, the e solve and
// the vector chains one after the other.
template <typename T, int TS, int D>
__device__ __forceinline__ void t_filt_combine(const Team<TS>& tm, FiltTeamWs<T, D>& w) {
  using W = FiltTeamWs<T, D>;
  constexpr int L1 = W::LD1, L2 = W::LD2;
  const Team<TS / 2> h;
  const bool hi = tm.r >= TS / 2;  // the half that runs eta's chain (the other: b's)
  const bool put = h.r < D;
  static_assert(TS / 2 >= D || TS == 32, "a half-team holds one row per lane");
  // b: t2 = b1 + U1 U1^T eta2; eta: s2 = eta2 - Z2 Z2^T b1
  T* const va = hi ? w.v3 : w.v1;
  T* const vb = hi ? w.v4 : w.v2;
  const T* const S = hi ? w.Z2 : w.U1;
  Acc<T> x = t_dotrow<T, TS / 2, D, D>(h, S, 1, L1, hi ? w.b1 : w.e2);
  if (put) va[h.r] = x.value();
  tm.sync();
  x = t_dotrow<T, TS / 2, D, D>(h, S, L1, 1, va);
  if (put) vb[h.r] = hi ? x.from(w.e2[h.r]) : x.plus(w.b1[h.r]);  // read again after t_filt_xi's barriers
  t_filt_xi<T, TS, D>(tm, w);
  // b: t3 = Xi21^T t2, t2 -= Mu^T t3; eta: s3 = Mu s2, s2 -= Xi21 s3
  // (one instruction stream: the halves differ in pointers and strides)
  x = t_dotrow<T, TS / 2, D, D>(h, hi ? w.Mu : w.Xb, hi ? L1 : 1, hi ? 1 : L2, vb);
  if (put) va[h.r] = x.value();
  tm.sync();
  x = t_dotrow<T, TS / 2, D, D>(h, hi ? w.Xb : w.Mu, hi ? L2 : 1, hi ? 1 : L1, va);
  if (put) vb[h.r] = x.from(vb[h.r]);
  tm.sync();
  // b = A2 t2 + b2; eta = A1^T s2 + eta1
  x = t_dotrow<T, TS / 2, D, D>(h, hi ? w.A1 : w.A2, hi ? 1 : L1, hi ? L1 : 1, vb);
  if (put) {
    if (hi)
      w.e1[h.r] = x.plus(w.e1[h.r]);
    else
      w.b1[h.r] = x.plus(w.b2[h.r]);
  }
  // W = A2 - M^T Xi21^T
  for (int idx = tm.r; idx < D * D; idx += TS) {
    const int i = idx / D, j = idx % D;
    Acc<T> s(w.A2[i * L1 + j]);
#pragma unroll
    for (int k = 0; k < D; ++k) s.mul_add(-w.M[k * L1 + i], w.Xb[j * L2 + k]);
    w.W[i * L1 + j] = s.value();
  }
  // Z = tria([Z1 | A1^T Xi22]) (the rows of Xt reused), U = tria([U2 | M^T])
  t_mm<T, TS, D, D, D, L1, L2, L2, true, false>(tm, w.A1, w.Xb + D, w.Xt + D);
  t_copy<T, TS, D, D, L1, L2>(tm, w.Z1, w.Xt);
  t_copy<T, TS, D, D, L1, L2, true>(tm, w.M, w.UX + D);
  t_copy<T, TS, D, D, L1, L2>(tm, w.U2, w.UX);
  tm.sync();
  // A = W A1, kept in M until A1 is no longer read
  t_mm<T, TS, D, D, D, L1, L1, L1>(tm, w.W, w.A1, w.M);
  {  // U and Z side by side on the two halves of the team
    T* X = hi ? w.Xt : w.UX;
    t_lq<T, TS / 2, D, 0, L2, L2>(h, X, X, TailFixed<D, 2 * D>{});
  }
  tm.sync();
  t_copy<T, TS, D, D, L1, L1>(tm, w.M, w.A1);
  t_copy<T, TS, D, D, L2, L1>(tm, w.UX, w.U1);
  t_copy<T, TS, D, D, L2, L1>(tm, w.Xt, w.Z1);
  tm.sync();
}

// (m, L) <- state after element 2: (b, U) part of the combine with e1 = (m, L)
// held in (b1, U1).
template <typename T, int TS, int D>
__device__ __forceinline__ void t_filt_apply(const Team<TS>& tm, FiltTeamWs<T, D>& w) {
  using W = FiltTeamWs<T, D>;
  constexpr int L1 = W::LD1, L2 = W::LD2;
  const bool put = tm.r < D;
  Acc<T> x = t_dotrow<T, TS, D, D>(tm, w.U1, 1, L1, w.e2);
  if (put) w.v1[tm.r] = x.value();
  tm.sync();
  x = t_dotrow<T, TS, D, D>(tm, w.U1, L1, 1, w.v1);
  if (put) w.v2[tm.r] = x.plus(w.b1[tm.r]);
  t_filt_xi<T, TS, D>(tm, w);
  x = t_dotrow<T, TS, D, D>(tm, w.Xb, 1, L2, w.v2);
  if (put) w.v3[tm.r] = x.value();
  t_copy<T, TS, D, D, L1, L2, true>(tm, w.M, w.UX + D);
  t_copy<T, TS, D, D, L1, L2>(tm, w.U2, w.UX);
  tm.sync();
  x = t_dotrow<T, TS, D, D>(tm, w.Mu, 1, L1, w.v3);
  if (put) w.v1[tm.r] = x.from(w.v2[tm.r]);
  tm.sync();
  x = t_dotrow<T, TS, D, D>(tm, w.A2, L1, 1, w.v1);
  if (put) w.b1[tm.r] = x.plus(w.b2[tm.r]);
  t_lq<T, TS, D, 0, L2, L2>(tm, w.UX, w.UX, TailFixed<D, 2 * D>{});
  t_copy<T, TS, D, D, L2, L1>(tm, w.UX, w.U1);
  tm.sync();
}

// Smoother: shared-memory workspace of one team.
template <typename T, int D>
struct SmoTeamWs {
  static constexpr int D2 = 2 * D;
  static constexpr int LD2 = Ld<D2>::v;
  static constexpr int LD1 = Ld<D>::v;
  T E1[D * LD1], D1[D * LD1], g1[D];  // later element (or the state: D1 = L, g1 = m)
  T E2[D * LD1], D2m[D * LD1], g2[D];  // earlier element / running composite
  T X[D * LD2], En[D * LD1];
};

// composite (g2, E2, D2) <- (g2, E2, D2) o (g1, E1, D1)
// (pof/parallel_filtsmooth/smoother.py:53-63 with elem1 later, elem2 earlier)
template <typename T, int TS, int D>
__device__ __forceinline__ void t_smooth_combine(const Team<TS>& tm, SmoTeamWs<T, D>& w) {
  using W = SmoTeamWs<T, D>;
  constexpr int L1 = W::LD1, L2 = W::LD2;
  const Acc<T> x = t_dotrow<T, TS, D, D>(tm, w.E2, L1, 1, w.g1);
  t_mm_lowB<T, TS, D, D, L1, L1, L2>(tm, w.E2, w.D1, w.X + D);
  t_copy<T, TS, D, D, L1, L2>(tm, w.D2m, w.X);
  t_mm<T, TS, D, D, D, L1, L1, L1>(tm, w.E2, w.E1, w.En);
  t_lq<T, TS, D, 0, L2, L2>(tm, w.X, w.X, TailFixed<D, 2 * D>{});
  if (tm.r < D) w.g2[tm.r] = x.plus(w.g2[tm.r]);
  t_copy<T, TS, D, D, L1, L1>(tm, w.En, w.E2);
  t_copy<T, TS, D, D, L2, L1>(tm, w.X, w.D2m);
  tm.sync();
}

// state (g1 = m, D1 = L) <- element (g2, E2, D2) applied: m = E m + g, L = tria([E L, D])
// (L any square root: the terminal state may be the caller's)
template <typename T, int TS, int D>
__device__ __forceinline__ void t_smooth_apply(const Team<TS>& tm, SmoTeamWs<T, D>& w) {
  using W = SmoTeamWs<T, D>;
  constexpr int L1 = W::LD1, L2 = W::LD2;
  const Acc<T> x = t_dotrow<T, TS, D, D>(tm, w.E2, L1, 1, w.g1);
  t_mm<T, TS, D, D, D, L1, L1, L2>(tm, w.E2, w.D1, w.X + D);
  t_copy<T, TS, D, D, L1, L2>(tm, w.D2m, w.X);
  t_lq<T, TS, D, 0, L2, L2>(tm, w.X, w.X, TailFixed<D, 2 * D>{});
  if (tm.r < D) w.g1[tm.r] = x.plus(w.g2[tm.r]);
  t_copy<T, TS, D, D, L2, L1>(tm, w.X, w.D1);
  tm.sync();
}

// Number of columns of A (M x N, leading dimension LDA) up to the last one with
// a nonzero entry, and whether A is lower triangular (integer operations only).
template <typename T, int TS, int M, int N, int LDA>
__device__ __forceinline__ int t_ncols(const Team<TS>& tm, const T* A, bool* lower = nullptr) {
  int nc = 0;
  bool up = false;
  for (int idx = tm.r; idx < M * N; idx += TS) {
    const int i = idx / N, j = idx % N;
    if (!is_zero(A[i * LDA + j])) {
      nc = max(nc, j + 1);
      up |= j > i;
    }
  }
  if (lower) *lower = !__any_sync(tm.mask, up);
  return (int)__reduce_max_sync(tm.mask, (unsigned)nc);
}

// ---------------------------------------------------------------------------
// Level-0 smoother operations.  The elements' factors Dm are raw square roots
// (D x nk, not triangular: see t_kf_step), nk their column count.
// ---------------------------------------------------------------------------

// C(M x nc) = A(M x N) B, the first nc columns of B
template <typename T, int TS, int M, int N, int LDA, int LDB, int LDC>
__device__ __forceinline__ void t_mm_cols(const Team<TS>& tm, const T* A, const T* B, T* C, int nc) {
  constexpr int RS = Pow2Ceil<M>::v < TS ? Pow2Ceil<M>::v : TS;
  constexpr int CG = TS / RS;
#pragma unroll
  for (int i0 = 0; i0 < M; i0 += RS) {
    const int i = i0 + tm.r % RS;
    if (M % RS != 0 && i >= M) continue;
    T a[N];
#pragma unroll
    for (int k = 0; k < N; ++k) a[k] = A[i * LDA + k];
    for (int j = tm.r / RS; j < nc; j += CG) {
      Acc<T> s(T(0));
#pragma unroll
      for (int k = 0; k < N; ++k) s.mul_add(a[k], B[k * LDB + j]);
      C[i * LDC + j] = s.value();
    }
  }
}

// Dm <- its triangular form
template <typename T, int TS, int D>
__device__ __forceinline__ void t_smooth_tria(const Team<TS>& tm, SmoTeamWs<T, D>& w) {
  using W = SmoTeamWs<T, D>;
  constexpr int L1 = W::LD1;
  const int nk = t_ncols<T, TS, D, D, L1>(tm, w.D2m);
  t_lq<T, TS, D, 0, L1, L1>(tm, w.D2m, w.D2m, TailUpper{nk});
  for (int idx = tm.r; idx < D * D; idx += TS) {
    const int i = idx / D, k = idx % D;
    if (k > i) w.D2m[i * L1 + k] = T(0);
  }
  tm.sync();
}

// t_smooth_combine with a raw D1; `first`: the composite's D2 is raw too.
template <typename T, int TS, int D>
__device__ __forceinline__ void t_smooth_combine_raw(const Team<TS>& tm, SmoTeamWs<T, D>& w, bool first) {
  using W = SmoTeamWs<T, D>;
  constexpr int L1 = W::LD1, L2 = W::LD2;
  const int n1 = t_ncols<T, TS, D, D, L1>(tm, w.D1);
  const Acc<T> x = t_dotrow<T, TS, D, D>(tm, w.E2, L1, 1, w.g1);
  t_mm<T, TS, D, D, D, L1, L1, L1>(tm, w.E2, w.E1, w.En);
  if (first) {  // [E2 D1 | D2], both dense
    const int n2 = t_ncols<T, TS, D, D, L1>(tm, w.D2m);
    t_mm_cols<T, TS, D, D, L1, L1, L2>(tm, w.E2, w.D1, w.X, n1);
    for (int idx = tm.r; idx < D * D; idx += TS) {
      const int i = idx / D, k = idx % D;
      if (n1 + k < 2 * D) w.X[i * L2 + n1 + k] = w.D2m[i * L1 + k];  // zero from column n1 + n2 on
    }
    t_lq<T, TS, D, 0, L2, L2>(tm, w.X, w.X, TailUpper{n1 + n2});
  } else {  // [D2 | E2 D1]
    t_mm_cols<T, TS, D, D, L1, L1, L2>(tm, w.E2, w.D1, w.X + D, n1);
    t_copy<T, TS, D, D, L1, L2>(tm, w.D2m, w.X);
    t_lq<T, TS, D, 0, L2, L2>(tm, w.X, w.X, TailRange{D, D + n1});
  }
  if (tm.r < D) w.g2[tm.r] = x.plus(w.g2[tm.r]);
  t_copy<T, TS, D, D, L1, L1>(tm, w.En, w.E2);
  for (int idx = tm.r; idx < D * D; idx += TS) {
    const int i = idx / D, k = idx % D;
    w.D2m[i * L1 + k] = k <= i ? w.X[i * L2 + k] : T(0);
  }
  tm.sync();
}

// t_smooth_apply with a raw D2: L = tria([E L, D2]); `lower`: L is lower
// triangular (every state but a caller's terminal one).
template <typename T, int TS, int D>
__device__ __forceinline__ void t_smooth_apply_raw(const Team<TS>& tm, SmoTeamWs<T, D>& w, bool lower) {
  using W = SmoTeamWs<T, D>;
  constexpr int L1 = W::LD1, L2 = W::LD2;
  const int nk = t_ncols<T, TS, D, D, L1>(tm, w.D2m);
  const Acc<T> x = t_dotrow<T, TS, D, D>(tm, w.E2, L1, 1, w.g1);
  if (lower)
    t_mm_lowB<T, TS, D, D, L1, L1, L2>(tm, w.E2, w.D1, w.X);
  else
    t_mm<T, TS, D, D, D, L1, L1, L2>(tm, w.E2, w.D1, w.X);
  t_copy<T, TS, D, D, L1, L2>(tm, w.D2m, w.X + D);
  t_lq<T, TS, D, 0, L2, L2>(tm, w.X, w.X, TailUpper{D + nk});
  if (tm.r < D) w.g1[tm.r] = x.plus(w.g2[tm.r]);
  for (int idx = tm.r; idx < D * D; idx += TS) {
    const int i = idx / D, k = idx % D;
    w.D1[i * L1 + k] = k <= i ? w.X[i * L2 + k] : T(0);
  }
  tm.sync();
}

}  // namespace pof

namespace pof {

// ---------------------------------------------------------------------------
// Level-0 (per time step) operations, team-parallel.  Same quantities as
// kf_step / cond_fold_step of pof_ops.cuh.
//
// Level 0 is bound by the FP64 pipe (every FP64 instruction of a warp holds
// it for 64 cycles), so a step's triangularizations leave out what is zero:
//   [QL | F L]: L has nl nonzero columns -- D - d after a noiseless update,
//     none at the start of a conditional fold -- and with a block-diagonal F
//     (the IWP prior) row j of F L ends with its block (TailBlocks): tails of
//     4 and 6 columns at D = 8, d = 2 instead of 8;
//   Psi = [[H Lp, R], [Lp, 0]] without noise (no R, or a step whose R is
//     zero) ends with the last column h that H reaches (its E0 and E1
//     columns): D - q + 1 of D + d columns, and Psi22 has D - d columns;
//   Phi22, the smoother element's factor, is left as the D x nl matrix that
//     the reflectors of [QL | F L] leave below them: it enters only
//     triangularizations that take any square root;
//   [Z | W^T]: the tail is W^T's d columns.
// The structure is found when the model is loaded (integer operations: it is
// the caller's data and need not have any); sums over it leave out exact
// zeros.  D = 8, d = 2: 8 + 5 reflectors per Kalman step instead of 8 + 9 + 7.
// ---------------------------------------------------------------------------
template <typename T, int D, int DY>
struct StepDims {
  static constexpr int D2 = 2 * D;
  static constexpr int DP = D + DY;
  static constexpr int Q1 = D % DY == 0 ? D / DY : 0;  // block size of the IWP prior
  static constexpr int LD2 = Ld<D2>::v;
  static constexpr int LD1 = Ld<D>::v;
  static constexpr int LDP = Ld<DP>::v;
  static constexpr int LDZ = Ld<D + DY>::v;
};

// Shared-memory workspace of one team for the Kalman filter step fused with
// the smoother element (the transition model F, QL is passed separately:
// one copy per block).
template <typename T, int D, int DY>
struct StepKFWs : StepDims<T, D, DY> {
  using B = StepDims<T, D, DY>;
  T H[DY * B::LD1], c[DY], R[DY * DY];          // observation model of the step
  T m[D], L[D * B::LD1];                        // filtered state
  T X[D * B::LD2], Y[D * B::LD2];               // [QL | F L], [0 | L]
  T P[B::DP * B::LDP];                          // Psi
  T E[D * B::LD1], g[D], mp[D];                 // smoother element, predicted mean
};

// ... for the conditional fold (and the plain Kalman step of a first chunk).
template <typename T, int D, int DY>
struct StepFoldWs : StepDims<T, D, DY> {
  using B = StepDims<T, D, DY>;
  T H[DY * B::LD1], c[DY], R[DY * DY];
  T m[D], L[D * B::LD1];                        // mean (of x = 0 in the fold) and conditional L
  T X[D * B::LD2];                              // [QL | F L]
  T P[B::DP * B::LDP];
  T mp[D];
  T ZX[D * B::LDZ];                             // [Z | W^T]
};

// Zero structure of a step's transition model (D - by - D F and QL):
//   qlow: QL is lower triangular; wf: the block size Q when F is
//   block-diagonal with upper-triangular Q x Q blocks (the IWP prior), else 0.
struct StepStruct {
  bool qlow;
  int wf;
};

// What a step's observation model leaves out: h1 columns of H up to its last
// nonzero one, no noise.
struct StepObs {
  int h1;
  bool rzero;
};

template <typename T, int TS, int D, int DY, typename WS>
__device__ __forceinline__ StepObs t_load_step(const Team<TS>& tm, WS& w, const T* H, const T* c, const T* R) {
  constexpr int L1 = Ld<D>::v;
  int h1 = 0;
  bool noise = false;
  for (int f = tm.r; f < DY * D; f += TS) {
    const T v = H[f];
    w.H[(f / D) * L1 + f % D] = v;
    if (!is_zero(v)) h1 = max(h1, f % D + 1);
  }
  for (int f = tm.r; f < DY; f += TS) w.c[f] = c[f];
  if (R) {
    for (int f = tm.r; f < DY * DY; f += TS) {
      const T v = R[f];
      w.R[f] = v;
      noise |= !is_zero(v);
    }
    noise = __any_sync(tm.mask, noise);
  }
  return StepObs{(int)__reduce_max_sync(tm.mask, (unsigned)h1), !noise};
}

// [QL | F L] in w.X and, when SMOOTH, [0 | L] in w.Y; their reflectors.
template <typename T, int TS, int D, int DY, bool SMOOTH, typename WS>
__device__ __forceinline__ void t_predict(const Team<TS>& tm, WS& w, const T* F, const T* QL, StepStruct ss, int nl,
                                          bool lower) {
  using W = StepDims<T, D, DY>;
  constexpr int L1 = W::LD1, L2 = W::LD2;
  t_copy<T, TS, D, D, L1, L2>(tm, QL, w.X);
  for (int idx = tm.r; idx < D * D; idx += TS) {
    const int i = idx / D, j = idx % D;
    if (j >= nl) continue;
    const int k0 = ss.wf ? i : 0, k1 = ss.wf ? (i / ss.wf + 1) * ss.wf : D;
    Acc<T> s(T(0));
    for (int k = k0; k < k1; ++k) s.mul_add(F[i * L1 + k], w.L[k * L1 + j]);
    w.X[i * L2 + D + j] = s.value();
  }
  T* Y = w.X;
  if constexpr (SMOOTH) {
    Y = w.Y;
    t_fill<T, TS, D, D, L2>(tm, w.Y, T(0), T(0));
    t_copy<T, TS, D, D, L1, L2>(tm, w.L, w.Y + D);
  }
  constexpr int MB = SMOOTH ? D : 0;
  if (ss.qlow) {
    if (ss.wf && lower)
      t_lq<T, TS, D, MB, L2, L2>(tm, w.X, Y, TailBlocks<W::Q1>{D, nl});
    else
      t_lq<T, TS, D, MB, L2, L2>(tm, w.X, Y, TailBlocks<0>{D, nl});
  } else {  // a caller's QL that is not triangular: no pivot block
    t_lq<T, TS, D, MB, L2, L2>(tm, w.X, Y, TailUpper{D + nl});
    for (int idx = tm.r; idx < D * D; idx += TS) {
      const int i = idx / D, k = idx % D;
      if (k > i) w.X[i * L2 + k] = T(0);
    }
    tm.sync();
  }
}

// Psi = tria([[H Lp, R], [Lp, 0]]) with Lp = X[:, :D] in w.P.
template <typename T, int TS, int D, int DY, typename WS>
__device__ __forceinline__ void t_psi(const Team<TS>& tm, WS& w, StepObs ob) {
  using W = StepDims<T, D, DY>;
  constexpr int L1 = W::LD1, L2 = W::LD2, LP = W::LDP, DP = W::DP;
  for (int idx = tm.r; idx < DY * D; idx += TS) {
    const int i = idx / D, j = idx % D;
    Acc<T> s(T(0));
    for (int k = 0; k < ob.h1; ++k) s.mul_add(w.H[i * L1 + k], w.X[k * L2 + j]);
    w.P[i * LP + j] = s.value();
  }
  // (with more observations than states Psi11 reaches into these columns)
  if (!ob.rzero || DY > D)
    for (int idx = tm.r; idx < DY * DY; idx += TS) w.P[(idx / DY) * LP + D + idx % DY] = ob.rzero ? T(0) : w.R[idx];
  for (int idx = tm.r; idx < D * DP; idx += TS) {
    const int i = idx / DP, j = idx % DP;
    w.P[(DY + i) * LP + j] = (j <= i) ? w.X[i * L2 + j] : T(0);
  }
  const int nc = ob.rzero ? ob.h1 : DP;  // columns with entries right of the diagonal
  t_lq<T, TS, DP, 0, LP, LP>(tm, w.P, w.P, TailUpper{nc}, nc < DP ? nc : DP);
}

// L <- Psi22 (columns beyond Psi's are zero; right of the diagonal the
// reflected tails are left out)
template <typename T, int TS, int D, int DY, typename WS>
__device__ __forceinline__ void t_psi22(const Team<TS>& tm, WS& w, StepObs ob) {
  using W = StepDims<T, D, DY>;
  constexpr int L1 = W::LD1, LP = W::LDP, DP = W::DP;
  const int nc = ob.rzero ? D : DP;
  for (int idx = tm.r; idx < D * D; idx += TS) {
    const int i = idx / D, k = idx % D;
    w.L[i * L1 + k] = (k <= i && DY + k < nc) ? w.P[(DY + i) * LP + DY + k] : T(0);
  }
}

// wv = -Psi11^{-1} (H x + c) (every lane has all of it), the lane's share
// being one row; rdv[i] = 1 / Psi11_ii, r the residual.
template <typename T, int TS, int D, int DY, typename WS>
__device__ __forceinline__ void t_innovation(const Team<TS>& tm, WS& w, const T* x, int h1, T (&r)[DY], T (&rdv)[DY],
                                             T (&wv)[DY]) {
  using W = StepDims<T, D, DY>;
  constexpr int L1 = W::LD1, LP = W::LDP;
  const int src = (threadIdx.x & 31) / TS * TS;
  const int i = tm.r % DY;
  Acc<T> sa(w.c[i]);
  for (int k = 0; k < h1; ++k) sa.mul_add(w.H[i * L1 + k], x[k]);
  const T s = sa.value();
  const T rd = rcp(w.P[i * LP + i]);
#pragma unroll
  for (int a = 0; a < DY; ++a) {
    r[a] = __shfl_sync(tm.mask, s, src + a);
    rdv[a] = __shfl_sync(tm.mask, rd, src + a);
  }
#pragma unroll
  for (int a = 0; a < DY; ++a) {
    T v = -r[a];
#pragma unroll
    for (int k = 0; k < a; ++k) v = fma(-w.P[a * LP + k], wv[k], v);
    wv[a] = v * rdv[a];
  }
}

// Predicted mean and factor from the state (m, L), L with nl nonzero columns,
// and the smoother element of that state when SMOOTH: g, E, and its factor in
// Y[:, D : D + nl] (a D x nl square root of Phi22 Phi22^T, not triangular).
template <typename T, int TS, int D, int DY, bool SMOOTH, typename WS>
__device__ __forceinline__ void t_predict_gain(const Team<TS>& tm, WS& w, const T* F, const T* QL, StepStruct ss,
                                               int nl, bool lower) {
  using W = StepDims<T, D, DY>;
  constexpr int L1 = W::LD1, L2 = W::LD2;
  static_assert(D <= TS && DY <= TS, "one row of the state per lane");
  for (int i = tm.r; i < D; i += TS) {
    const int k0 = ss.wf ? i : 0, k1 = ss.wf ? (i / ss.wf + 1) * ss.wf : D;
    Acc<T> s(T(0));
    for (int k = k0; k < k1; ++k) s.mul_add(F[i * L1 + k], w.m[k]);
    w.mp[i] = s.value();
  }
  t_predict<T, TS, D, DY, SMOOTH>(tm, w, F, QL, ss, nl, lower);  // Phi11 = X[:, :D], Phi21 = Y[:, :D]
  if constexpr (SMOOTH) {
    // E = Phi21 Phi11^{-1}, lane j solves for row j; g = m - E mp
    const int src = (threadIdx.x & 31) / TS * TS;
    const T rd = t_recip_diag<T, TS, D, L2>(tm, w.X);
    const int j = tm.r < D ? tm.r : 0;
    T x[D];
#pragma unroll
    for (int i = D - 1; i >= 0; --i) {
      Acc<T> s(w.Y[j * L2 + i]);
#pragma unroll
      for (int k = i + 1; k < D; ++k) s.mul_add(-w.X[k * L2 + i], x[k]);
      x[i] = s.value() * __shfl_sync(tm.mask, rd, src + i);
    }
    Acc<T> gj(w.m[j]);
#pragma unroll
    for (int i = 0; i < D; ++i) gj.mul_add(-x[i], w.mp[i]);
    if (tm.r < D) {
      w.g[j] = gj.value();
#pragma unroll
      for (int i = 0; i < D; ++i) w.E[j * L1 + i] = x[i];
    }
  }
}

// One square-root KF step from the filtered state (m, L) at grid s
// (t_predict_gain, then the update).  Adds ||Psi11^{-T} r||^2 to ssq (whiten
// quirk, pof/utils.py:110-112), ||Psi11^{-1} r||^2 to yy and |Psi11_ii| to
// lane i's lp; returns the column count of the new L.
template <typename T, int TS, int D, int DY, bool SMOOTH, typename WS>
__device__ __forceinline__ int t_kf_step(const Team<TS>& tm, WS& w, const T* F, const T* QL, StepStruct ss,
                                         StepObs ob, int nl, bool lower, double& ssq, double& yy, LogProd& lp) {
  using W = StepDims<T, D, DY>;
  constexpr int LP = W::LDP;
  t_predict_gain<T, TS, D, DY, SMOOTH>(tm, w, F, QL, ss, nl, lower);
  t_psi<T, TS, D, DY>(tm, w, ob);
  T r[DY], rdv[DY], wv[DY], wq[DY];
  t_innovation<T, TS, D, DY>(tm, w, w.mp, ob.h1, r, rdv, wv);
  T s2 = T(0), y2 = T(0);
#pragma unroll
  for (int i = DY - 1; i >= 0; --i) {
    T v = r[i];
#pragma unroll
    for (int k = i + 1; k < DY; ++k) v = fma(-w.P[k * LP + i], wq[k], v);
    wq[i] = v * rdv[i];
    s2 = fma(wq[i], wq[i], s2);
    y2 = fma(wv[i], wv[i], y2);
  }
  ssq += (double)s2;
  yy += (double)y2;
  if (tm.r < DY) lp.mul(w.P[tm.r * LP + tm.r]);
  for (int i = tm.r; i < D; i += TS) {
    Acc<T> acc(w.mp[i]);
#pragma unroll
    for (int k = 0; k < DY; ++k) acc.mul_add(w.P[(DY + i) * LP + k], wv[k]);
    w.m[i] = acc.value();
  }
  t_psi22<T, TS, D, DY>(tm, w, ob);
  tm.sync();
  return ob.rzero && DY < D ? D - DY : D;
}

// Conditional fold of a chunk (cond_fold_step of pof_ops.cuh): lane j holds
// column j of A and entry j of eta; b is w.m, U is w.L, Z is w.ZX[:, :D].
template <typename T, int D>
struct FoldRegs {
  T a[D], eta;
};

template <typename T, int TS, int D, int DY>
__device__ __forceinline__ void t_fold_start(const Team<TS>& tm, StepFoldWs<T, D, DY>& w, FoldRegs<T, D>& fr) {
  using W = StepDims<T, D, DY>;
#pragma unroll
  for (int i = 0; i < D; ++i) fr.a[i] = T(i == tm.r ? 1 : 0);
  fr.eta = T(0);
  t_fill<T, TS, D, D, W::LD1>(tm, w.L, T(0), T(0));
  t_fill<T, TS, D, D, W::LDZ>(tm, w.ZX, T(0), T(0));
  for (int i = tm.r; i < D; i += TS) w.m[i] = T(0);
}

template <typename T, int TS, int D, int DY>
__device__ __forceinline__ int t_cond_fold_step(const Team<TS>& tm, StepFoldWs<T, D, DY>& w, FoldRegs<T, D>& fr,
                                                const T* F, const T* QL, StepStruct ss, StepObs ob, int nl) {
  using W = StepDims<T, D, DY>;
  constexpr int L1 = W::LD1, LP = W::LDP, LZ = W::LDZ, Q1 = W::Q1;
  static_assert(D <= TS && DY <= TS, "one column of A per lane");
  t_predict<T, TS, D, DY, false>(tm, w, F, QL, ss, nl, true);
  t_psi<T, TS, D, DY>(tm, w, ob);
  // FA (lane's column) and Fb
  T fa[D];
  if (Q1 > 0 && ss.wf) {
#pragma unroll
    for (int i = 0; i < D; ++i) {
      Acc<T> s(T(0));
#pragma unroll
      for (int k = i; k < (i / (Q1 > 0 ? Q1 : 1) + 1) * Q1; ++k) s.mul_add(F[i * L1 + k], fr.a[k]);
      fa[i] = s.value();
    }
  } else {
#pragma unroll
    for (int i = 0; i < D; ++i) {
      Acc<T> s(T(0));
#pragma unroll
      for (int k = 0; k < D; ++k) s.mul_add(F[i * L1 + k], fr.a[k]);
      fa[i] = s.value();
    }
  }
  for (int i = tm.r; i < D; i += TS) {
    const int k0 = ss.wf ? i : 0, k1 = ss.wf ? (i / ss.wf + 1) * ss.wf : D;
    Acc<T> s(T(0));
    for (int k = k0; k < k1; ++k) s.mul_add(F[i * L1 + k], w.m[k]);
    w.mp[i] = s.value();
  }
  tm.sync();
  // w = Psi11^{-1} (H Fb + c) = -wv, W = Psi11^{-1} H FA (lane's column)
  T r[DY], rdv[DY], wv[DY], wc[DY];
  t_innovation<T, TS, D, DY>(tm, w, w.mp, ob.h1, r, rdv, wv);
#pragma unroll
  for (int i = 0; i < DY; ++i) {
    Acc<T> s(T(0));
#pragma unroll
    for (int k = 0; k < D; ++k)
      if (k < ob.h1) s.mul_add(w.H[i * L1 + k], fa[k]);
#pragma unroll
    for (int k = 0; k < i; ++k) s.mul_add(-w.P[i * LP + k], wc[k]);
    wc[i] = s.value() * rdv[i];
  }
  // A = FA - Psi21 W; b = Fb - Psi21 w; eta -= W^T w; [Z | W^T]
#pragma unroll
  for (int i = 0; i < D; ++i) {
    T acc = fa[i];
#pragma unroll
    for (int k = 0; k < DY; ++k) acc = fma(-w.P[(DY + i) * LP + k], wc[k], acc);
    fr.a[i] = acc;
  }
#pragma unroll
  for (int k = 0; k < DY; ++k) fr.eta = fma(wc[k], wv[k], fr.eta);
  if (tm.r < D) {
#pragma unroll
    for (int k = 0; k < DY; ++k) w.ZX[tm.r * LZ + D + k] = wc[k];
  }
  for (int i = tm.r; i < D; i += TS) {
    Acc<T> acc(w.mp[i]);
#pragma unroll
    for (int k = 0; k < DY; ++k) acc.mul_add(w.P[(DY + i) * LP + k], wv[k]);
    w.m[i] = acc.value();
  }
  t_psi22<T, TS, D, DY>(tm, w, ob);
  t_lq<T, TS, D, 0, LZ, LZ>(tm, w.ZX, w.ZX, TailFixed<D, D + DY>{});
  return ob.rzero && DY < D ? D - DY : D;
}

}  // namespace pof
