// Taylor-mode initial values of the built-in fields on the host (declared in
// include/pof.h): the power series of the solution of y' = f(y) at the
// initial value, coefficient by coefficient in truncated series arithmetic
// (the recurrences of automatic differentiation in Taylor mode; Griewank and
// Walther, "Evaluating Derivatives", ch. 13).  The reference takes the same
// derivatives from jax.experimental.jet (pof/initialization.py:15-22).
//
// A solve spends 2 to 7 ms of host time on nested torch.func.jvp for them (q =
// 2 to 3), more than the device on a short grid; here it is microseconds.
#include <math.h>

#include <vector>

#include "../../include/pof.h"
#include "pof_fields.cuh"

namespace {

using Series = std::vector<double>;  // coefficients 0 .. q

Series cst(int n, double v) {
  Series s(n, 0.0);
  s[0] = v;
  return s;
}
Series operator+(Series a, const Series& b) {
  for (size_t i = 0; i < a.size(); ++i) a[i] += b[i];
  return a;
}
Series operator-(Series a, const Series& b) {
  for (size_t i = 0; i < a.size(); ++i) a[i] -= b[i];
  return a;
}
Series operator*(double s, Series a) {
  for (double& v : a) v *= s;
  return a;
}
Series operator*(const Series& a, const Series& b) {
  Series c(a.size(), 0.0);
  for (size_t i = 0; i < a.size(); ++i)
    for (size_t j = 0; j + i < a.size(); ++j) c[i + j] += a[i] * b[j];
  return c;
}
// s^e for s[0] > 0: k s_0 p_k = sum_{j=1..k} (e j - (k - j)) s_j p_{k-j}
Series power(const Series& s, double e) {
  Series p(s.size(), 0.0);
  p[0] = pow(s[0], e);
  for (size_t k = 1; k < s.size(); ++k) {
    double a = 0.0;
    for (size_t j = 1; j <= k; ++j) a += (e * (double)j - (double)(k - j)) * s[j] * p[k - j];
    p[k] = a / ((double)k * s[0]);
  }
  return p;
}

// f(y) as series (the expressions of pof/ivp.py)
std::vector<Series> field(int id, const double* p, const std::vector<Series>& y) {
  using namespace pof;
  const int n = (int)y[0].size();
  switch (id) {
    case FIELD_LOGISTIC: return {p[0] * (y[0] * (cst(n, 1.0) - y[0]))};
    case FIELD_LOTKAVOLTERRA:
      return {p[0] * y[0] - p[1] * (y[0] * y[1]), p[3] * (y[0] * y[1]) - p[2] * y[1]};
    case FIELD_VANDERPOL: return {y[1], p[0] * ((cst(n, 1.0) - y[0] * y[0]) * y[1] - y[0])};
    case FIELD_FITZHUGHNAGUMO:
      return {y[0] - (1.0 / 3.0) * (y[0] * y[0] * y[0]) - y[1] + cst(n, p[3]),
              p[2] * (y[0] + cst(n, p[0]) - p[1] * y[1])};
    case FIELD_FHN_CLASSIC:
      return {p[2] * (y[0] - (1.0 / 3.0) * (y[0] * y[0] * y[0]) + y[1]),
              (-1.0 / p[2]) * (y[0] - cst(n, p[0]) + p[1] * y[1])};
    case FIELD_ROBER: {
      const Series a = p[0] * y[0], b = p[2] * (y[1] * y[2]), c = p[1] * (y[1] * y[1]);
      return {b - a, a - c - b, c};
    }
    case FIELD_RIGID_BODY: return {p[0] * (y[1] * y[2]), p[1] * (y[0] * y[2]), p[2] * (y[0] * y[1])};
    case FIELD_SEIR: {
      const Series a = (p[1] / p[3]) * (y[0] * y[2]), b = p[0] * y[1], c = p[2] * y[2];
      return {-1.0 * a, a - b, b - c, c};
    }
    case FIELD_HENONHEILES:
      return {y[2], y[3], -1.0 * y[0] - (2.0 * p[0]) * (y[0] * y[1]),
              -1.0 * y[1] - p[0] * (y[0] * y[0] - y[1] * y[1])};
    case FIELD_THREEBODY: {
      const double mu = p[0], mp = 1.0 - p[0];
      const Series ax = y[0] + cst(n, mu), bx = y[0] - cst(n, mp), yy = y[1] * y[1];
      const Series d1 = mp * power(ax * ax + yy, -1.5), d2 = mu * power(bx * bx + yy, -1.5);
      return {y[2], y[3], y[0] + 2.0 * y[3] - ax * d1 - bx * d2, y[1] - 2.0 * y[2] - y[1] * (d1 + d2)};
    }
    default: {  // FIELD_FHN_RD
      const int m = (int)y.size() / 2;
      const double a = p[0], b = p[1], c = p[2], kv = p[3], kw = p[4];
      std::vector<Series> f(2 * m);
      for (int k = 0; k < m; ++k) {
        const int l = (k + m - 1) % m, r = (k + 1) % m;
        const Series &v = y[k], &w = y[m + k];
        f[k] = c * (v - (1.0 / 3.0) * (v * v * v) + w) + kv * (y[l] - 2.0 * v + y[r]);
        f[m + k] = (-1.0 / c) * (v - cst(n, a) + b * w) + kw * (y[m + l] - 2.0 * w + y[m + r]);
      }
      return f;
    }
  }
}

}  // namespace

extern "C" int pof_taylor(int32_t field_id, int32_t d, int32_t q, const double* params, const double* y0, double* out) {
  using namespace pof;
  if (field_id <= 0 || field_id >= FIELD_COUNT) return POF_ERR_FIELD;
  if (d < 1 || q < 0 || q > 64 || !params || !y0 || !out) return POF_ERR_ARG;
  const int fd = field_dim(field_id);
  if (fd > 0 ? fd != d : (d < 2 || d % 2 != 0)) return POF_ERR_FIELD;
  try {
    std::vector<Series> y(d, Series(q + 1, 0.0));
    for (int i = 0; i < d; ++i) y[i][0] = y0[i];
    for (int k = 0; k < q; ++k) {
      const std::vector<Series> f = field(field_id, params, y);
      for (int i = 0; i < d; ++i) y[i][k + 1] = f[i][k] / (double)(k + 1);
    }
    double fact = 1.0;
    for (int k = 0; k <= q; ++k) {
      if (k > 1) fact *= k;
      for (int i = 0; i < d; ++i) out[(int64_t)k * d + i] = y[i][k] * fact;
    }
  } catch (...) {
    return POF_ERR_ARG;  // out of host memory
  }
  return POF_OK;
}
