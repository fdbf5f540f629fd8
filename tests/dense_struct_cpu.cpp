// The dense schedule on the host with the structure that the GPU's context
// exploits (tria_rows, qlow of csrc/pof_dense.cu), which the plain context of
// dense_sched_cpu.cpp leaves out: the factorization of the leading rows, and
// W = [X | S] with S lower triangular, whose reflectors end with S's rows.  An
// entry beyond a row's declared end that is not zero is an error.
#include "dense_sched_cpu.cpp"

namespace {

struct StructCtx : CpuCtx {
  bool qlow = false;
  void tria_rows(int64_t batch, int mt, int m, int n, MV<double> W, int low) {
    op = "tria_rows";
    mt = std::min(mt, n);
    std::vector<double> v(n);
    for (int64_t b = 0; b < batch; ++b)
      for (int i = 0; i < mt; ++i) {
        const int ne = low > 0 ? std::min(n, low + i + 1) : n;
        for (int c = ne; c < n; ++c)
          if (get(W, b, i, c) != 0.0 && err.empty())
            err = "tria_rows: entry beyond the row's end (low = " + std::to_string(low) + ")";
        double s = 0.0;
        for (int c = i + 1; c < ne; ++c) s += get(W, b, i, c) * get(W, b, i, c);
        const double alpha = get(W, b, i, i);
        double beta = alpha, tau = 0.0;
        if (s != 0.0) {
          const double h = hypot(alpha, sqrt(s));
          beta = alpha >= 0.0 ? -h : h;
          tau = (beta - alpha) / beta;
          v[i] = 1.0;
          for (int c = i + 1; c < ne; ++c) v[c] = get(W, b, i, c) / (alpha - beta);
          for (int r = i + 1; r < m; ++r) {
            double dsum = 0.0;
            for (int c = i; c < ne; ++c) dsum += get(W, b, r, c) * v[c];
            for (int c = i; c < ne; ++c) put(W, b, r, c, get(W, b, r, c) - tau * dsum * v[c]);
          }
        }
        put(W, b, i, i, beta);
        for (int c = i + 1; c < n; ++c) put(W, b, i, c, 0.0);
      }
  }
  void tria(int64_t batch, int m, int n, MV<double> W) { tria_rows(batch, m, m, n, W, 0); }
};

}  // namespace

extern "C" int dense_struct_filtsmooth(int which, int64_t n, int D, int d, const double* x0m, const double* x0L,
                                       const double* F, const double* QL, int64_t fts, const double* H,
                                       const double* c, const double* R, int64_t rst, double* om, double* oL,
                                       double* osc, int chunks, char* msg, int msg_len) {
  Layout<double> sz = layout<double>(nullptr, which, n, D, d, chunks);
  std::vector<double> ws(sz.total / sizeof(double) + 64, std::numeric_limits<double>::quiet_NaN());
  char* base = reinterpret_cast<char*>(ws.data());
  char* al = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(base) + 255) & ~uintptr_t(255));
  std::vector<std::pair<size_t, size_t>> regions;
  Layout<double> L = layout<double>(al, which, n, D, d, chunks, &regions);
  StructCtx cx;
  cx.D = D;
  cx.qlow = fts == 0;  // as csrc/pof_dense.cu finds it: one QL for all steps, lower triangular
  for (int i = 0; i < D; ++i)
    for (int j = i + 1; j < D; ++j) cx.qlow = cx.qlow && QL[(int64_t)i * D + j] == 0.0;
  const int64_t DD = (int64_t)D * D, nft = fts ? n * DD : DD;
  for (const auto& r : regions)
    cx.ranges.push_back({"workspace", reinterpret_cast<const double*>(al + r.first),
                         (int64_t)(r.second / sizeof(double)), true});
  const int64_t ns = which == 2 ? n + 1 : 1;
  cx.ranges.push_back({"x0m", x0m, ns * D, false});
  cx.ranges.push_back({"x0L", x0L, ns * DD, false});
  if (which != 2) {
    cx.ranges.push_back({"H", H, n * d * D, false});
    cx.ranges.push_back({"c", c, n * d, false});
    if (R) cx.ranges.push_back({"R", R, rst ? n * d * d : (int64_t)d * d, false});
  }
  cx.ranges.push_back({"F", F, nft, false});
  cx.ranges.push_back({"QL", QL, nft, false});
  cx.ranges.push_back({"om", om, (n + 1) * D, true});
  cx.ranges.push_back({"oL", oL, (n + 1) * DD, true});
  cx.ranges.push_back({"osc", osc, 8, true});
  run_schedule<double>(cx, L, which, x0m, x0L, F, QL, fts, H, c, R, rst, om, oL, osc);
  if (!cx.err.empty()) {
    snprintf(msg, msg_len, "%s", cx.err.c_str());
    return -1;
  }
  return cx.qlow ? 1 : 0;
}
