// The chunk rule of passes and solves (even_c0 of csrc/pof_plan.h) and the plans
// it gives, at random step counts and at the multiples of its target.
#define main plan_props_main
#include "plan_props.cpp"
#undef main

static void check_even(int64_t n, int D, int DY, int esz, bool solver) {
  const int lanes = pof::l0_lanes(D, true), lo = lanes == 1 ? 4 : 2;
  const int64_t target = lanes == 1 ? 19456 : 48640 / lanes;
  const int c = pof::even_c0(n, lanes);
  CHECK(c >= lo && c <= 64, "n %lld D %d: C0 %d", (long long)n, D, c);
  if (c < 64) CHECK(cdiv(n, c) <= target, "n %lld D %d: %lld chunks", (long long)n, D, (long long)cdiv(n, c));
  if (c > lo) CHECK(cdiv(n, c - 1) > target, "n %lld D %d: C0 %d not the shortest", (long long)n, D, c);
  const pof::Plan p = pof::make_plan(n, D, DY, esz, solver, c, 0, false, 0);
  CHECK(p.C0 == c && p.cnt[1] == cdiv(n, c) && (p.cnt[1] - 1) * c < n, "n %lld: %lld chunks of %d", (long long)n,
        (long long)p.cnt[1], p.C0);
  std::vector<Region> r;
  const int64_t NF = 3LL * D * D + 2 * D, NS = D + (int64_t)D * D, NG = D + 2LL * D * D;
  for (int k = 1; k <= p.nlev; ++k) {
    r.push_back({p.felem[k], (size_t)(esz * NF * p.cnt[k])});
    r.push_back({p.fstate[k], (size_t)(esz * NS * p.cnt[k])});
    r.push_back({p.gelem[k], (size_t)(esz * NG * p.cnt[k])});
    r.push_back({p.gend[k], (size_t)(esz * NS * p.cnt[k])});
  }
  r.push_back({p.selem, (size_t)(esz * NG * n)});
  r.push_back({p.partials, sizeof(double) * 5 * (size_t)p.cnt[1]});
  const char* why = "";
  CHECK(regions_ok(r, p.total, &why), "n %lld D %d: %s", (long long)n, D, why);
}

int main() {
  std::mt19937_64 rng(1);
  for (int D : {2, 3, 4, 5, 6, 8, 9, 10, 12})
    for (int esz : {4, 8})
      for (bool solver : {false, true}) {
        const int lanes = pof::l0_lanes(D, true);
        const int64_t target = lanes == 1 ? 19456 : 48640 / lanes;
        check_even(1, D, 1, esz, solver);
        check_even(2, D, 1, esz, solver);
        for (int m : {1, 2, 3, 4, 5, 7, 8, 11, 63, 64, 65, 100})
          for (int o : {-1, 0, 1}) check_even(m * target + o, D, 1, esz, solver);
        for (int i = 0; i < 50; ++i)
          check_even((int64_t)std::exp(std::uniform_real_distribution<double>(0, 17)(rng)) + 1, D, 1, esz, solver);
      }
  if (g_fail) return 1;
  puts("ok");
  return 0;
}
