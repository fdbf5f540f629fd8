// Per-thread dense linear algebra on small row-major matrices.
//
// Every routine works on one thread's private data with compile-time sizes,
// so loops unroll and index arithmetic folds into immediate offsets.  The
// state dimension D of the solver is small (2..16); at these sizes the FP64
// pipe of a GB300 SM (2 FMA/clk/SM) is the bound, and one thread per chunk of
// time steps keeps every lane of every issued FP64 instruction useful (a
// warp-cooperative Householder leaves most lanes idle on triangular shapes).
//
// Leading dimensions are template parameters so sub-blocks of larger
// matrices (e.g. the two halves of [F L, QL]) are addressed in place.
#pragma once

#include <cuda_runtime.h>
#include <math.h>

#include <type_traits>

namespace pof {

// ---------------------------------------------------------------------------
// Runtime bounds checks (the sanitizer substitute): compiled in with
// -DPOF_CHECKS (a build with relocatable device code, so every translation
// unit shares one device word), they test the global-memory indices the
// kernels derive from sizes and plan tables -- element, step and problem
// indices -- before the access.  A failing check skips its access and
// records the source line of the first failure in pof_check_line
// (pof_checks_read).  In the normal build every check is the constant true.
// ---------------------------------------------------------------------------
#ifdef POF_CHECKS
extern __device__ unsigned long long pof_check_line;
__device__ __forceinline__ bool pof_check_fail(int line) {
  atomicCAS(&pof_check_line, 0ull, (unsigned long long)line);
  return false;
}
#define POF_IN(i, n) (((i) >= 0 && (i) < (n)) ? true : ::pof::pof_check_fail(__LINE__))
#else
#define POF_IN(i, n) true
#endif

// ---------------------------------------------------------------------------
// Reciprocal and reciprocal square root of a double, for the scalars of the
// Householder reflectors and the diagonal solves.
//
// GB300 runs FP64 at 1/64 of the FP32 rate: an FP64 instruction of a warp
// holds its SM sub-partition's FP64 pipe for 64 cycles, whatever its lanes
// do, so the instruction sequences of IEEE double division and square root
// -- computed once per reflector -- are a large share of a small
// factorization's time.  These take a single-precision hardware
// approximation of the argument's leading 21 significand bits as the seed
// (the float operand and the widened result are built with 32-bit integer
// operations, so no FP64 conversion is issued), then ONE third-order
// correction in double precision (Householder's iteration of order 3;
// Halley's method for the square root):
//   1/a:       r = 1 - a y,     y <- y (1 + r + r^2)
//   1/sqrt(a): r = 1 - a y^2,   y <- y (1 + r/2 + 3 r^2/8)
// which cubes the seed's relative error (below ~1.2e-6: truncation of the
// argument plus the approximation) to below 2e-18, so the result is within a
// few units in the last place of the correctly rounded value: 3 and 5 FP64
// instructions.  Arguments whose binary exponent is beyond +-1000 (zero,
// subnormals, infinities, NaN included) take the IEEE operations.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float approx_rcp(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float approx_rsqrt(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// high word of a double whose binary exponent is within +-1000
__device__ __forceinline__ bool exp_in_range(int hi) {
  return (unsigned)(((hi >> 20) & 0x7ff) - 23) <= 2000u;
}
// the leading significand bits of the double with high word hi, times 2^p
__device__ __forceinline__ float lead_float(int hi, int p) {
  return __int_as_float((((hi << 3) & 0x007ffff8) | 0x3f800000) + (p << 23));
}
// the float f > 0 times 2^e as a double (exact; no FP64 instruction)
__device__ __forceinline__ double widen_with_exp(float f, int e) {
  const int b = __float_as_int(f);
  return __hiloint2double((b >> 3) + ((896 + e) << 20), b << 29);
}

__device__ __forceinline__ double rcp_nr(double a) {
  const int hi = __double2hiint(a);
  if (!exp_in_range(hi)) return 1.0 / a;
  const double ym = widen_with_exp(approx_rcp(lead_float(hi, 0)), 1023 - ((hi >> 20) & 0x7ff));
  const double y = __hiloint2double(__double2hiint(ym) | (hi & 0x80000000), __double2loint(ym));
  const double r = fma(-a, y, 1.0);
  return fma(y, fma(r, r, r), y);
}

__device__ __forceinline__ double rsqrt_nr(double a) {
  const int hi = __double2hiint(a);
  if (!exp_in_range(hi) || hi < 0) return 1.0 / sqrt(a);
  const int t = hi - 0x3ff00000, k = t >> 21;  // a = m 4^k with m in [1, 4)
  const double y = widen_with_exp(approx_rsqrt(lead_float(hi, (t >> 20) & 1)), -k);
  const double r = fma(-(a * y), y, 1.0);
  return fma(y, r * fma(r, 0.375, 0.5), y);
}

template <typename T>
__device__ __forceinline__ T rcp(T a) {
  if constexpr (std::is_same<T, double>::value)
    return rcp_nr(a);
  else
    return T(1) / a;
}

// v / l with r = quotient_rcp(l): the product v r and one correction with its
// exact residual, rounded as the division is (Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", IBM J. Res.
// Dev. 1990).  Divisors whose reciprocal the type may not hold have r = 0 and
// are divided by.
__device__ __forceinline__ double quotient_rcp(double l) {
  return exp_in_range(__double2hiint(l)) ? rcp(l) : 0.0;
}
__device__ __forceinline__ float quotient_rcp(float l) {
  return (unsigned)(((__float_as_int(l) >> 23) & 0xff) - 27) <= 200u ? rcp(l) : 0.f;
}
__device__ __forceinline__ bool is_finite(double x) { return (__double2hiint(x) & 0x7ff00000) != 0x7ff00000; }
__device__ __forceinline__ bool is_finite(float x) { return (__float_as_int(x) & 0x7f800000) != 0x7f800000; }
template <typename T>
__device__ __forceinline__ T quotient(T v, T l, T r) {
  if (r == T(0)) return v / l;
  const T q = v * r;
  return is_finite(q) ? fma(fma(-q, l, v), r, q) : q;
}

// Scalars of the Householder reflector that maps (alpha, x), ||x||^2 = xn2,
// onto (beta, 0), with LAPACK dlarfg's conventions: beta = -sign(alpha)
// ||(alpha, x)|| (sign(0) = +1), tau = (beta - alpha) / beta, the tail
// scaled by scal = 1 / (alpha - beta); no reflection (beta = alpha,
// tau = scal = 0) when x is exactly zero.
template <typename T>
__device__ __forceinline__ void householder(T alpha, T xn2, T& beta, T& tau, T& scal) {
  const bool zero = (xn2 == T(0));
  if constexpr (std::is_same<T, double>::value) {
    const double a2 = fma(alpha, alpha, xn2);
    const double g = rsqrt_nr(a2);  // 1 / ||(alpha, x)||
    // sg = -sign(alpha) g = 1 / beta (sign flipped with an integer operation)
    const double sg = __longlong_as_double(__double_as_longlong(g) ^ (alpha >= 0.0 ? (1LL << 63) : 0LL));
    const double b = a2 * sg;  // beta = -sign(alpha) ||(alpha, x)||
    const double u = alpha - b;
    beta = zero ? alpha : b;
    tau = zero ? 0.0 : -u * sg;  // (beta - alpha) / beta
    scal = zero ? 0.0 : rcp_nr(u);
  } else {
    const T nrm = sqrt(fma(alpha, alpha, xn2));
    beta = zero ? alpha : (alpha >= T(0) ? -nrm : nrm);
    tau = zero ? T(0) : (beta - alpha) / beta;
    scal = zero ? T(0) : T(1) / (alpha - beta);
  }
}

// true when x is +0 or -0, tested on the bits (a floating-point compare of a
// double would go through the FP64 pipe)
__device__ __forceinline__ bool is_zero(double x) { return (__double_as_longlong(x) << 1) == 0; }
__device__ __forceinline__ bool is_zero(float x) { return (__float_as_uint(x) << 1) == 0; }

// The same reflector with the tail x left as it is, so the squared norm can be
// formed together with the dot products of the rows below and no pass scales
// x: a row (a, y) with dot = y . x becomes (a - w, y - ws x), where
//   double: H = I - kap v v^T, v = (u, x), u = alpha - beta, kap = -1 / (u beta):
//     ws = kap (u a + dot), w = u ws; ||(alpha, x)|| = h and
//     kap = 1 / (a2 + |alpha| h) from single-precision seeds and one
//     third-order correction each (as rsqrt_nr and rcp_nr), 11 FP64
//     instructions of scalars and 2 per row; measured alone on a warp
//     1399 cycles with 64-bit integer seeds one after the other.
//     Beyond 2^+-1000 the squared norm's reciprocal leaves double's range although
//     the reflector, which is that of s (alpha, x) but for beta, does not: there
//     s = 2^-k brings the norm near 1, and `scale(s)` puts s x in place of x and
//     of the dot products that were formed with it.  (As accurate as
//     householder: what the square loses to underflow is lost to both.)  The
//     rows that stay near 1 pay nothing for it; x left as it is, with a second u
//     for the pivot's own update, cost the sequential smoother 3 %, a test of its
//     own before the chain 6 %.
//   float: w = tau (a + scal dot), ws = w scal (kap would leave float's range
//     for tails below 1e-19).
// For xn2 != 0 only.
template <typename T>
struct Reflector;

template <>
struct Reflector<double> {
  double beta, u, kap;
  template <typename F>
  __device__ __forceinline__ void set(double alpha, double xn2, F&& scale) {
    const double a2 = fma(alpha, alpha, xn2);
    const int hi = __double2hiint(a2), ahi = __double2hiint(alpha) & 0x7fffffff;
    double h;
    if (exp_in_range(hi)) {
      const int t = hi - 0x3ff00000, k = t >> 21;  // a2 = m 4^k with m in [1, 4)
      const float mf = lead_float(hi, (t >> 20) & 1);
      const float yf = approx_rsqrt(mf);
      const double y = widen_with_exp(yf, -k);
      // the seed of 1 / (a2 + |alpha| h) from single precision too (|alpha| 2^-k
      // and m^(1/2)), while the square root's correction is in the FP64 pipe
      const int av = ahi - ((896 + k) << 20);
      const float af = __int_as_float(av > 0 ? av << 3 : 0);
      const double z = widen_with_exp(approx_rcp(fmaf(af, mf * yf, mf)), -2 * k);
      const double g = a2 * y;
      const double r = fma(-g, y, 1.0);
      h = fma(g, r * fma(r, 0.375, 0.5), g);
      const double s = fma(-fma(fabs(alpha), h, a2), z, 1.0);
      kap = fma(z, fma(s, s, s), z);
      finish(alpha, h);
    } else {
      const int e = (hi >> 20) & 0x7ff;
      const int k = e == 0 ? -524 : (e - 1023) >> 1;
      const double s = __hiloint2double((1023 - k) << 20, 0), back = __hiloint2double((1023 + k) << 20, 0);
      const double b2 = a2 * s * s;
      h = sqrt(b2);
      kap = 1.0 / fma(fabs(alpha * s), h, b2);
      finish(alpha * s, h);
      beta *= back;
      scale(s);
    }
  }
  __device__ __forceinline__ void finish(double alpha, double h) {
    // sign(0) = +, so alpha = -0 reflects like +0
    const bool neg = __double2hiint(alpha) < 0 && !is_zero(alpha);
    beta = neg ? h : __hiloint2double(__double2hiint(h) ^ 0x80000000, __double2loint(h));
    u = alpha - beta;
  }
  // new pivot entry; ws: the multiple of x taken off the row's tail
  __device__ __forceinline__ double row(double a, double dot, double& ws) const {
    ws = kap * fma(u, a, dot);
    return fma(-ws, u, a);
  }
};

template <>
struct Reflector<float> {
  float beta, tau, scal;
  template <typename F>
  __device__ __forceinline__ void set(float alpha, float xn2, F&&) {
    householder(alpha, xn2, beta, tau, scal);
  }
  __device__ __forceinline__ float row(float a, float dot, float& ws) const {
    const float w = tau * fmaf(scal, dot, a);
    ws = w * scal;
    return a - w;
  }
};

// A kernel launched while the one before it still runs (launch_next in
// pof_driver.cuh): grid_begin waits for that kernel's end and its writes, then
// lets the next launch come in.  Every thread passes it before it touches
// memory, and the pointers go through it, so that no load of a read-only
// parameter can be moved ahead of the wait.  In an ordinary launch both
// instructions do nothing that could be seen.
template <typename P>
__device__ __forceinline__ void grid_begin_ptr(P& p) {
  asm volatile("" : "+l"(p)::"memory");
}
template <typename... P>
__device__ __forceinline__ void grid_begin(P&... p) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  (grid_begin_ptr(p), ...);
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Accumulator of an inner product, v + sum a b.  double: fused multiply-adds.
// float: compensated (Ogita, Rump and Oishi, "Accurate sum and dot product",
// SISC 2005, Dot2), one rounding for the whole sum: the states carry integrals
// over the grid, along which the sums' rounding errors add up.  FP32
// instructions are not what bounds these kernels: on a float32 pass of 2000
// steps at D = 6 all team sums compensated cost 0.420 -> 0.460 ms and take the
// means' error against 64 bits from 2.0e-6 to 1.6e-6 (16 inputs), of 2900
// steps from 4.0e-6 to 2.8e-6.
template <typename T>
struct Acc;
template <>
struct Acc<double> {
  double h;
  Acc() = default;
  __device__ __forceinline__ explicit Acc(double v) : h(v) {}
  __device__ __forceinline__ void mul_add(double a, double b) { h = fma(a, b, h); }
  __device__ __forceinline__ void join(unsigned mask, int o, int width) {
    h += __shfl_xor_sync(mask, h, o, width);
  }
  __device__ __forceinline__ void scale(double s) { h *= s; }
  __device__ __forceinline__ double plus(double v) const { return v + h; }   // v + the sum
  __device__ __forceinline__ double from(double v) const { return v - h; }   // v - the sum
  __device__ __forceinline__ double value() const { return h; }
};
template <>
struct Acc<float> {
  float h, l;
  Acc() = default;
  __device__ __forceinline__ explicit Acc(float v) : h(v), l(0.f) {}
  __device__ __forceinline__ void add(float p) {  // h + p exactly as h + error
    const float s = __fadd_rn(h, p), t = __fsub_rn(s, h);
    l = __fadd_rn(l, __fadd_rn(__fsub_rn(h, __fsub_rn(s, t)), __fsub_rn(p, t)));
    h = s;
  }
  __device__ __forceinline__ void mul_add(float a, float b) {
    const float p = __fmul_rn(a, b);
    l = __fadd_rn(l, __fmaf_rn(a, b, -p));
    add(p);
  }
  __device__ __forceinline__ void join(unsigned mask, int o, int width) {
    const float h2 = __shfl_xor_sync(mask, h, o, width), l2 = __shfl_xor_sync(mask, l, o, width);
    add(h2);
    l = __fadd_rn(l, l2);
  }
  __device__ __forceinline__ void scale(float s) { h *= s, l *= s; }
  __device__ __forceinline__ float plus(float v) const {
    Acc<float> a = *this;
    a.add(v);
    return a.value();
  }
  __device__ __forceinline__ float from(float v) const {
    Acc<float> a(v);
    a.add(-h);
    a.l = __fsub_rn(a.l, l);
    return a.value();
  }
  // an overflowed or infinite sum has no error term (inf - inf): it is h, as in
  // the plain sum
  __device__ __forceinline__ float value() const {
    const float v = __fadd_rn(h, l);
    return v == v ? v : h;
  }
};

// C(MxN) = A(MxK) * B(KxN)
template <typename T, int M, int K, int N, int LDA, int LDB, int LDC>
__device__ __forceinline__ void mm(const T* __restrict__ A, const T* __restrict__ B, T* __restrict__ C) {
#pragma unroll
  for (int i = 0; i < M; ++i) {
#pragma unroll
    for (int j = 0; j < N; ++j) {
      T s = T(0);
#pragma unroll
      for (int k = 0; k < K; ++k) s = fma(A[i * LDA + k], B[k * LDB + j], s);
      C[i * LDC + j] = s;
    }
  }
}

// y(M) = A(MxN) x(N)
template <typename T, int M, int N, int LDA>
__device__ __forceinline__ void mv(const T* __restrict__ A, const T* __restrict__ x, T* __restrict__ y) {
#pragma unroll
  for (int i = 0; i < M; ++i) {
    T s = T(0);
#pragma unroll
    for (int k = 0; k < N; ++k) s = fma(A[i * LDA + k], x[k], s);
    y[i] = s;
  }
}

// The LQ factorisation by Householder reflectors of the first M of the MX
// rows of X (NC columns): afterwards X[:M, :M] holds L in its lower triangle
// (L L^T = the M rows' X X^T) and the rows below are multiplied by the same
// orthogonal matrix; what lies right of the diagonal in the M rows is left as
// it is and must not be read.
//
// LAPACK's dgeqr2 computes the R factor of X^T so: one reflector per row, in
// row order, with dlarfg's conventions -- beta = -sign(alpha) * ||(alpha, x)||,
// and no reflection (tau = 0, R_jj = alpha) when the tail x is exactly zero.
// The reference computes tria as qr(A^T, mode="r")^T (pof/utils.py:33-41).
template <typename T, int M, int MX, int NC, int LD>
__device__ __forceinline__ void lq_rows(T* X) {
#pragma unroll
  for (int j = 0; j < M; ++j) {
    T* xj = X + j * LD;
    T xn2 = T(0);
#pragma unroll
    for (int k = j + 1; k < NC; ++k) xn2 = fma(xj[k], xj[k], xn2);
    if (!is_zero(xn2)) {
      Reflector<T> h;
      h.set(xj[j], xn2, [&](T s) {
#pragma unroll
        for (int k = j + 1; k < NC; ++k) xj[k] *= s;
      });
      xj[j] = h.beta;
#pragma unroll
      for (int i = j + 1; i < MX; ++i) {
        T* xi = X + i * LD;
        T dot = T(0), ws;
#pragma unroll
        for (int k = j + 1; k < NC; ++k) dot = fma(xi[k], xj[k], dot);
        xi[j] = h.row(xi[j], dot, ws);
#pragma unroll
        for (int k = j + 1; k < NC; ++k) xi[k] = fma(-ws, xj[k], xi[k]);
      }
    }
  }
}

// LQ with a triangular pivot block (t_lq of pof_team.cuh, one thread): rows
// [P | W], P lower triangular M x M, W with NW columns, over MB rows [Yp | Yw]:
// P becomes L with L L^T = P P^T + W W^T, the rows below are multiplied by the
// same orthogonal matrix.  Q > 0: row j of W ends with column (j / Q + 1) Q - 1
// (W = F S, F block-diagonal, S lower triangular).  W must not be read after.
template <typename T, int M, int NW, int MB, int Q, int LDP, int LDW, int LDYP, int LDYW>
__device__ __forceinline__ void lq_pivot(T* P, T* W, T* Yp, T* Yw) {
#pragma unroll
  for (int j = 0; j < M; ++j) {
    const int nw = Q > 0 ? ((j / (Q > 0 ? Q : 1) + 1) * Q < NW ? (j / (Q > 0 ? Q : 1) + 1) * Q : NW) : NW;
    T* wj = W + j * LDW;
    T xn2 = T(0);
#pragma unroll
    for (int k = 0; k < NW; ++k)
      if (k < nw) xn2 = fma(wj[k], wj[k], xn2);
    if (!is_zero(xn2)) {
      Reflector<T> h;
      h.set(P[j * LDP + j], xn2, [&](T s) {
#pragma unroll
        for (int k = 0; k < NW; ++k)
          if (k < nw) wj[k] *= s;
      });
      P[j * LDP + j] = h.beta;
#pragma unroll
      for (int i = j + 1; i < M + MB; ++i) {
        T* y = i < M ? W + i * LDW : Yw + (i - M) * LDYW;
        T& a = i < M ? P[i * LDP + j] : Yp[(i - M) * LDYP + j];
        T dot = T(0), ws;
#pragma unroll
        for (int k = 0; k < NW; ++k)
          if (k < nw) dot = fma(y[k], wj[k], dot);
        a = h.row(a, dot, ws);
#pragma unroll
        for (int k = 0; k < NW; ++k)
          if (k < nw) y[k] = fma(-ws, wj[k], y[k]);
      }
    }
  }
}

// b <- L^{-1} b   (L lower-triangular M x M)
template <typename T, int M, int LDL>
__device__ __forceinline__ void trsv_l(const T* __restrict__ L, T* b) {
#pragma unroll
  for (int i = 0; i < M; ++i) {
    T s = b[i];
#pragma unroll
    for (int k = 0; k < i; ++k) s = fma(-L[i * LDL + k], b[k], s);
    b[i] = s * rcp(L[i * LDL + i]);
  }
}

template <typename T, int M, int N, int LDS, int LDD>
__device__ __forceinline__ void copy(const T* __restrict__ S, T* __restrict__ Dst) {
#pragma unroll
  for (int i = 0; i < M; ++i)
#pragma unroll
    for (int j = 0; j < N; ++j) Dst[i * LDD + j] = S[i * LDS + j];
}

template <typename T, int M, int N, int LDD>
__device__ __forceinline__ void zero(T* Dst) {
#pragma unroll
  for (int i = 0; i < M; ++i)
#pragma unroll
    for (int j = 0; j < N; ++j) Dst[i * LDD + j] = T(0);
}

}  // namespace pof
