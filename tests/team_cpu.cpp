// The team kernels of libpof on the host, one lane at a time: every thread of a
// block is a fiber that runs until it meets a warp or block barrier, a shuffle
// or a vote, and the order in which the fibers run between two of them is the
// caller's (tests/test_team_cpu.py).  A kernel whose lanes touch one word of
// shared memory from both sides of no barrier gives different results in
// different orders; one that reads shared memory nobody wrote gives different
// results for different contents of it.
//
// The headers are the library's, with the PTX statements and the shared-memory
// declarations replaced by the test before this file is compiled.
#include <math.h>
#include <stdint.h>
#include <string.h>
#include <ucontext.h>

#include <algorithm>
#include <vector>

#define __device__
#define __host__
#define __global__
#define __forceinline__ inline
#define __launch_bounds__(...)
#define __align__(x)

struct Dim {
  unsigned x = 0, y = 0, z = 0;
};
static Dim threadIdx, blockIdx, blockDim;
static unsigned char host_smem[256 * 1024] __attribute__((aligned(256)));

using std::max;
using std::min;
template <typename A, typename B>
static inline A bits(B b) {
  static_assert(sizeof(A) == sizeof(B), "");
  A a;
  memcpy(&a, &b, sizeof a);
  return a;
}
static inline long long __double_as_longlong(double x) { return bits<long long>(x); }
static inline double __longlong_as_double(long long x) { return bits<double>(x); }
static inline int __double2hiint(double x) { return (int)(bits<unsigned long long>(x) >> 32); }
static inline int __double2loint(double x) { return (int)bits<unsigned long long>(x); }
static inline double __hiloint2double(int hi, int lo) {
  return bits<double>(((unsigned long long)(unsigned)hi << 32) | (unsigned)lo);
}
static inline int __float_as_int(float x) { return bits<int>(x); }
static inline unsigned __float_as_uint(float x) { return bits<unsigned>(x); }
static inline float __int_as_float(int x) { return bits<float>(x); }
static inline float __uint_as_float(unsigned x) { return bits<float>(x); }
static inline float __fadd_rn(float a, float b) { return a + b; }
static inline float __fsub_rn(float a, float b) { return a - b; }
static inline float __fmul_rn(float a, float b) { return a * b; }
static inline float __fmaf_rn(float a, float b, float c) { return fmaf(a, b, c); }

// ---------------------------------------------------------------------------
// fibers
// ---------------------------------------------------------------------------
namespace emu {
constexpr int kMax = 128;
constexpr size_t kStack = 256 * 1024;
enum Wait { RUN, WARP, BLOCK, DONE };
struct Fiber {
  ucontext_t ctx;
  Wait wait;
  unsigned mask;                // WARP: lanes that meet
  unsigned long long post;      // this lane's word
  unsigned long long got[32];   // the words of all lanes of the mask (of the block: the or of all)
};
static Fiber fib[kMax];
static std::vector<char> stacks;
static ucontext_t sched;
static int nthr, cur;
static void (*body)(void*);
static void* arg;
static bool deadlock;

static void entry() {
  body(arg);
  fib[cur].wait = DONE;
  swapcontext(&fib[cur].ctx, &sched);
}
static void meet(Wait w, unsigned mask, unsigned long long post) {
  Fiber& f = fib[cur];
  f.wait = w, f.mask = mask, f.post = post;
  swapcontext(&f.ctx, &sched);
}
static bool release() {  // lanes whose partners have all arrived
  bool any = false;
  for (int i = 0; i < nthr; ++i) {
    if (fib[i].wait != WARP) continue;
    const int w0 = i / 32 * 32;
    bool all = true;
    for (int l = 0; l < 32; ++l)
      if (fib[i].mask >> l & 1) {
        const int j = w0 + l;
        all = all && j < nthr && fib[j].wait == WARP && fib[j].mask == fib[i].mask;
      }
    if (!all) continue;
    for (int l = 0; l < 32; ++l)
      if (fib[i].mask >> l & 1) {
        for (int k = 0; k < 32; ++k) fib[w0 + l].got[k] = (fib[i].mask >> k & 1) ? fib[w0 + k].post : 0;
      }
    const unsigned m = fib[i].mask;
    for (int l = 0; l < 32; ++l)
      if (m >> l & 1) fib[w0 + l].wait = RUN;
    any = true;
  }
  bool block = false, all = true;  // a block barrier waits for the threads that have not left
  unsigned long long orv = 0;
  for (int i = 0; i < nthr; ++i) {
    if (fib[i].wait == BLOCK) block = true, orv |= fib[i].post;
    else if (fib[i].wait != DONE) all = false;
  }
  if (block && all) {
    for (int i = 0; i < nthr; ++i)
      if (fib[i].wait == BLOCK) fib[i].got[0] = orv, fib[i].wait = RUN;
    any = true;
  }
  return any;
}
// order: 0 ascending, 1 descending, else a seed of random orders
static void run_block(int n, int order, void (*f)(void*), void* a) {
  nthr = n, body = f, arg = a;
  if (stacks.size() < (size_t)n * kStack) stacks.resize((size_t)n * kStack);
  for (int i = 0; i < n; ++i) {
    getcontext(&fib[i].ctx);
    fib[i].ctx.uc_stack.ss_sp = stacks.data() + i * kStack;
    fib[i].ctx.uc_stack.ss_size = kStack;
    fib[i].ctx.uc_link = nullptr;
    makecontext(&fib[i].ctx, entry, 0);
    fib[i].wait = RUN;
  }
  unsigned long long rng = 0x9e3779b97f4a7c15ull * (unsigned)(order + 1);
  std::vector<int> perm(n);
  for (int i = 0; i < n; ++i) perm[i] = order == 1 ? n - 1 - i : i;
  for (;;) {
    if (order > 1)
      for (int i = n - 1; i > 0; --i) {
        rng = rng * 6364136223846793005ull + 1442695040888963407ull;
        std::swap(perm[i], perm[(rng >> 33) % (i + 1)]);
      }
    for (int i : perm)
      if (fib[i].wait == RUN) {
        cur = i, threadIdx.x = i;
        swapcontext(&sched, &fib[i].ctx);
      }
    if (release()) continue;
    for (int i = 0; i < n; ++i) deadlock = deadlock || fib[i].wait != DONE;
    return;
  }
}
}  // namespace emu

static inline void __syncwarp(unsigned mask = 0xffffffffu) { emu::meet(emu::WARP, mask, 0); }
static inline void __syncthreads() { emu::meet(emu::BLOCK, 0, 0); }
static inline int __syncthreads_or(int v) {
  emu::meet(emu::BLOCK, 0, v != 0);
  return emu::fib[emu::cur].got[0] != 0;
}
template <typename T>
static inline T shfl_from(unsigned mask, T v, int lane) {
  unsigned long long w = 0;
  memcpy(&w, &v, sizeof v);
  emu::meet(emu::WARP, mask, w);
  T r;
  memcpy(&r, &emu::fib[emu::cur].got[lane], sizeof r);
  return r;
}
template <typename T>
static inline T __shfl_sync(unsigned mask, T v, int src, int width = 32) {
  const int lane = threadIdx.x & 31;
  return shfl_from(mask, v, lane / width * width + src % width);
}
template <typename T>
static inline T __shfl_xor_sync(unsigned mask, T v, int o, int width = 32) {
  const int lane = threadIdx.x & 31, to = lane ^ o;
  return shfl_from(mask, v, to / width == lane / width ? to : lane);
}
static inline unsigned warp_fold(unsigned mask, unsigned v, int op) {
  emu::meet(emu::WARP, mask, v);
  unsigned r = 0;
  for (int l = 0; l < 32; ++l)
    if (mask >> l & 1) {
      const unsigned w = (unsigned)emu::fib[emu::cur].got[l];
      r = op == 0 ? std::max(r, w) : (op == 1 ? r + w : (r | w));
    }
  return r;
}
static inline unsigned __reduce_max_sync(unsigned mask, unsigned v) { return warp_fold(mask, v, 0); }
static inline unsigned __reduce_add_sync(unsigned mask, unsigned v) { return warp_fold(mask, v, 1); }
static inline int __any_sync(unsigned mask, int v) { return warp_fold(mask, v != 0, 2) != 0; }

#include "pof_seq.cuh"  // and with it every team kernel
#include "pof_dense_views.h"
#include "trsm_diag.h"  // k_trsm_diag of pof_dense.cuh

using namespace pof;

template <typename F>
static void launch(unsigned grid, int threads, int order, int poison, F f) {
  blockDim.x = threads;
  for (unsigned b = 0; b < grid; ++b) {
    memset(host_smem, poison, sizeof host_smem);
    blockIdx.x = b;
    emu::run_block(threads, order, [](void* p) { (*static_cast<F*>(p))(); }, &f);
  }
}

// A whole filter and smoother pass in chunks of C0 with the tree in pairs, all
// levels by teams (the schedule of pof_driver.cuh, D >= 6).
template <typename T, int D, int DY, bool PS>
static void pass(int order, int poison, int64_t n, int C0, const StepModel& sm, const T* x0m, const T* x0L, T* means,
                 T* chols, T* sm_means, T* sm_chols, double* sums) {
  constexpr int TSW = 2 * D <= 8 ? 8 : (2 * D <= 16 ? 16 : 32), TSN = TSW / 2, TSX = TSW < 32 ? 2 * TSW : 32;
  using FL = FiltLayout<D>;
  using GL = SmoLayout<D>;
  const int64_t n1 = (n + C0 - 1) / C0;
  auto poisoned = [&](int64_t len) {
    std::vector<T> v(len);
    memset((void*)v.data(), poison, len * sizeof(T));
    return v;
  };
  std::vector<int64_t> cnt{n1};
  while (cnt.back() > 2) cnt.push_back((cnt.back() + 1) / 2);
  const int nl = (int)cnt.size();
  std::vector<std::vector<T>> fe, fs, ge, gs;
  for (int64_t c : cnt) {
    fe.push_back(poisoned(c * FL::NF));
    fs.push_back(poisoned(c * (D + D * D)));
    ge.push_back(poisoned(c * GL::NG));
    gs.push_back(poisoned(c * (D + D * D)));
  }
  std::vector<T> se = poisoned(n * GL::NG);
  std::vector<double> part(P_COUNT * n1);
  auto blocks = [](int64_t teams, int per) { return (unsigned)((teams + per - 1) / per); };
  {
    using B = TeamBlockH<L0FoldWs<T, D, DY, PS>, TSN, FQHeader<T, D, PS>::bytes>;
    launch(1 + blocks(n1 - 1, B::teams), B::threads, order, poison, [&] {
      k_filt_l0_reduce_team<T, D, DY, TSN, PS>(n, C0, sm, x0m, x0L, fe[0].data(), n1);
    });
  }
  using BF = TeamBlock<FiltTeamWs<T, D>, TSX>;
  using BS = TeamBlock<SmoTeamWs<T, D>, TSX>;
  for (int l = 0; l + 1 < nl; ++l)
    launch(blocks(cnt[l + 1], BF::teams), BF::threads, order, poison,
           [&] { k_filt_reduce_team<T, D, TSX>(fe[l].data(), cnt[l], 2, fe[l + 1].data(), cnt[l + 1]); });
  launch(1, BF::threads, order, poison,
         [&] { k_filt_top_team<T, D, TSX>(fe[nl - 1].data(), cnt[nl - 1], x0m, x0L, fs[nl - 1].data()); });
  for (int l = nl - 2; l >= 0; --l)
    launch(blocks(cnt[l + 1], BF::teams), BF::threads, order, poison, [&] {
      k_filt_down_team<T, D, TSX>(fe[l].data(), cnt[l], 2, fs[l + 1].data(), cnt[l + 1], fs[l].data());
    });
  {
    using B = TeamBlockH<L0KFWs<T, D, DY, PS>, TSN, FQHeader<T, D, PS>::bytes>;
    launch(blocks(n1, B::teams), B::threads, order, poison, [&] {
      k_filt_l0_down_team<T, D, DY, TSN, PS>(n, C0, sm, fs[0].data(), n1, means, chols, se.data(), part.data(), true);
    });
  }
  {
    using B = TeamBlock<SmoTeamWs<T, D>, TSN>;
    launch(blocks(n1, B::teams), B::threads, order, poison,
           [&] { k_smo_l0_reduce_team<T, D, TSN>(se.data(), n, C0, ge[0].data(), n1); });
  }
  for (int l = 0; l + 1 < nl; ++l)
    launch(blocks(cnt[l + 1], BS::teams), BS::threads, order, poison,
           [&] { k_smo_reduce_team<T, D, TSX>(ge[l].data(), cnt[l], 2, ge[l + 1].data(), cnt[l + 1]); });
  launch(1, BS::threads, order, poison, [&] {
    k_smo_top_team<T, D, TSX>(ge[nl - 1].data(), cnt[nl - 1], means + n * D, chols + n * D * D, gs[nl - 1].data());
  });
  for (int l = nl - 2; l >= 0; --l)
    launch(blocks(cnt[l + 1], BS::teams), BS::threads, order, poison, [&] {
      k_smo_down_team<T, D, TSX>(ge[l].data(), cnt[l], 2, gs[l + 1].data(), cnt[l + 1], gs[l].data());
    });
  {
    using B = TeamBlockH<SmoL0Ws<T, D, PS>, TSN, FQHeader<T, D, PS>::bytes>;
    memcpy(sm_means, means, (n + 1) * D * sizeof(T));
    memcpy(sm_chols, chols, (n + 1) * D * D * sizeof(T));
    launch(blocks(n1, B::teams), B::threads, order, poison, [&] {
      k_smo_l0_down_team<T, D, TSN, PS>(n, C0, static_cast<const T*>(sm.F), static_cast<const T*>(sm.QL),
                                        sm.ft_stride, StepDims<T, D, DY>::Q1, se.data(), gs[0].data(), n1, sm_means,
                                        sm_chols, (const T*)nullptr, (const T*)nullptr, 0.0, 0.0, part.data());
    });
  }
  for (int p = P_SSQ; p <= P_SOBJ; ++p) {
    sums[p] = 0.0;
    for (int64_t t = 0; t < n1; ++t) sums[p] += part[p * n1 + t];
  }
}

template <typename T, int D, int DY>
static void sequential(int order, int poison, int64_t n, const StepModel& sm, int field, const T* params, double p0,
                       double p1, const T* x0m, const T* x0L, T* means, T* chols, double* scalars) {
  static_assert(sizeof(SeqWs<T, D, DY>) <= sizeof host_smem, "");
  launch(1, 64, order, poison, [&] {
    k_seq_filtsmooth<T, D, DY>(n, sm, field, params, (T)p0, (T)p1, x0m, x0L, 1, means, chols, scalars);
  });
}

// The square-root factorizations alone: X (M x NC) -> L by lq_rows, [P | W] by
// lq_pivot and t_lq, with MB rows below that get the same reflectors.
template <typename T, int M, int MB, int NW, int TS>
static void factor(int which, int order, T* X) {
  constexpr int LD = M + NW;
  if (which == 0) {
    lq_rows<T, M, M + MB, LD, LD>(X);
  } else if (which == 1) {
    lq_pivot<T, M, NW, MB, 0, LD, LD, LD, LD>(X, X + M, X + M * LD, X + M * LD + M);
  } else {
    launch(1, TS, order, 0xff, [&] {
      const Team<TS> tm;
      t_lq<T, TS, M, MB, LD, LD>(tm, X, X + M * LD, TailFixed<M, M + NW>{});
    });
  }
}

extern "C" {

int team_cpu_deadlock() { return emu::deadlock; }

#define SHAPES(X) X(6, 2) X(8, 2) X(9, 3) X(12, 3)
// 0 when the shape is compiled in
int team_cpu_pass(int f32, int order, int poison, int64_t n, int C0, int D, int d, const void* F, const void* QL,
                  int64_t fts, const void* H, const void* c, const void* R, const void* x0m, const void* x0L,
                  void* means, void* chols, void* sm_means, void* sm_chols, double* sums) {
  const StepModel sm{F, QL, fts, H, c, R, R ? (int64_t)d * d : 0};
#define CASE(T, D_, d_, PS)                                                                                         \
  pass<T, D_, d_, PS>(order, poison, n, C0, sm, (const T*)x0m, (const T*)x0L, (T*)means, (T*)chols, (T*)sm_means, \
                      (T*)sm_chols, sums)
#define X(D_, d_)                                                  \
  if (D == D_ && d == d_) {                                        \
    if (f32)                                                       \
      fts ? CASE(float, D_, d_, true) : CASE(float, D_, d_, false); \
    else                                                           \
      fts ? CASE(double, D_, d_, true) : CASE(double, D_, d_, false); \
    return 0;                                                      \
  }
  SHAPES(X)
#undef X
  return 1;
}

int team_cpu_sequential(int f32, int order, int poison, int64_t n, int D, int d, const void* F, const void* QL,
                        int64_t fts, const void* H, const void* c, const void* R, int field, const void* params,
                        double p0, double p1, const void* x0m, const void* x0L, void* means, void* chols,
                        double* scalars) {
  const StepModel sm{F, QL, fts, H, c, R, R ? (int64_t)d * d : 0};
#define X(D_, d_)                                                                                                 \
  if (D == D_ && d == d_) {                                                                                       \
    if (f32)                                                                                                      \
      sequential<float, D_, d_>(order, poison, n, sm, field, (const float*)params, p0, p1, (const float*)x0m,     \
                                (const float*)x0L, (float*)means, (float*)chols, scalars);                        \
    else                                                                                                          \
      sequential<double, D_, d_>(order, poison, n, sm, field, (const double*)params, p0, p1, (const double*)x0m,  \
                                 (const double*)x0L, (double*)means, (double*)chols, scalars);                    \
    return 0;                                                                                                     \
  }
  SHAPES(X)
  X(2, 1) X(4, 1) X(3, 4)
#undef X
  return 1;
}

// B (nbr x K, row-major) <- L^{-1} B (upper: L upper triangular)
void team_cpu_trsm_diag(int f32, int nbr, int upper, int K, void* L, void* B) {
  auto go = [&](auto t) {
    using T = decltype(t);
    const dense::MV<T> Lv{(T*)L, nbr, 1, 0}, Bv{(T*)B, K, 1, 0};
    blockDim.x = 128;
    for (int b = 0; b < (K + 127) / 128; ++b) {
      blockIdx.x = b, blockIdx.y = 0;
      auto f = [&] { dense::k_trsm_diag<T>(nbr, Lv, upper != 0, Bv, K, 0); };
      emu::run_block(128, 0, [](void* p) { (*static_cast<decltype(f)*>(p))(); }, &f);
    }
    blockIdx.x = 0;
  };
  f32 ? go(1.f) : go(1.0);
}

// M = 4 rows with 3 rows below and a tail of 4 columns, teams of 8 and 32 lanes
int team_cpu_factor(int f32, int which, int order, void* X) {
  switch (which) {
    case 0: case 1: case 2:
      f32 ? factor<float, 4, 3, 4, 8>(which, order, (float*)X) : factor<double, 4, 3, 4, 8>(which, order, (double*)X);
      return 0;
    case 3:
      f32 ? factor<float, 4, 3, 4, 32>(2, order, (float*)X) : factor<double, 4, 3, 4, 32>(2, order, (double*)X);
      return 0;
  }
  return 1;
}
}
