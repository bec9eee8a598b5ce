// The split search of k_small against the plain loops over every count, on the
// host.  Prints one line per problem of a sweep that differs, then for the
// allocation-free call's longest integrations the counts tried by both, then
// the chunks of single units in four planes.
#include <cstdio>
#include <cstdlib>

#include "small_split.h"

using namespace rsg;

static int fit_every(int turns, int gps, int ublocks, int c_lo, int c_hi, const SplitCost& k, double* cost_of, int* tried) {
  int best = c_lo;
  double best_cost = 1e300;
  for (int c = c_lo; c <= c_hi; ++c) {
    ++*tried;
    const int per = (turns + c - 1) / c;
    if (c > c_lo && (turns + per - 1) / per != c) continue;
    const double per_sm = std::ceil((double)ublocks * c / k.sms);
    const double load = std::max(per_sm, 1.5 * std::ceil(per_sm / k.occ));
    const double sum = c == 1 ? 0.0 : small_clustered(c, ublocks * c, k.sms) ? 0.5 + 0.15 * k.outputs / c : k.kernel ? 4.0 + c * (k.partial + 0.04) : 2.0 + c * (k.partial + k.serial);
    const double cost = ((per + gps - 1) / gps + 0.6) * k.unit * load + sum;
    if (cost < best_cost * 0.99) {
      best_cost = cost;
      best = c;
    }
  }
  *cost_of = best_cost;
  return best;
}

static Split every(const SplitProblem& p, int* tried) {
  auto pow2_floor = [](int x) { int q = 1; while (q * 2 <= x) q *= 2; return q; };
  const int most = std::min(p.groups, std::min(pow2_floor(p.planes * p.radix), pow2_floor(p.turns)));
  Split best;
  for (int gps = most; gps >= 1; gps /= 2) {
    const int sets = p.groups / gps;
    const int ub = (p.units + sets - 1) / sets;
    const int aim = std::max(1, (p.target_ctas + ub - 1) / ub);
    const long long floats = (long long)p.all_units * p.planes * p.n;
    int c_hi = (int)std::min<long long>((p.turns + gps - 1) / gps, std::max(8, 4 * aim));
    if (p.max_partial) c_hi = (int)std::min<long long>(c_hi, std::max<long long>(1, (long long)p.max_partial / floats));
    SplitCost k{p.unit_us, ub * ((double)sets * p.planes * p.n) * 2e-6, (double)sets * p.planes * p.n * 1.1e-4,
                (double)sets * p.planes * p.n / p.threads, p.sms, p.occ, !p.counters};
    Split s;
    s.gps = gps;
    s.chunks = fit_every(p.turns, gps, ub, 1, std::max(1, c_hi), k, &s.cost, tried);
    double cost = 0.0;
    if (p.counters && s.cost > kIdle * least_us(p, gps)) {
      k.kernel = true;
      const int c = fit_every(p.turns, gps, ub, 1, std::max(1, c_hi), k, &cost, tried);
      if (cost < s.cost) s.chunks = c, s.cost = cost;
    }
    if (gps == most || s.cost < 0.95 * best.cost) best = s;
  }
  return best;
}

static SplitProblem problem(int n, int planes, int units, int turns, bool limits) {
  SplitProblem p;
  p.n = n;
  p.planes = planes;
  p.radix = planes == 1 && (n == 32 || n == 512 || n == 1024) ? 32 : n < 16 ? n : 16;
  const int t = n / p.radix, tpb = t > 128 ? t : 128;
  p.groups = tpb / t;
  p.threads = tpb;
  p.units = p.all_units = units;
  p.turns = turns;
  p.sms = 152;
  p.occ = p.radix == 32 || planes == 4 ? 3 : 4;
  p.target_ctas = 152 * 4;
  p.unit_us = tpb * p.radix * 152 * 2.3e-6;
  if (limits) {
    p.max_partial = 1 << 20;
    p.counters = false;
  }
  return p;
}

int main() {
  int differ = 0, compared = 0;
  unsigned rng = 1;
  auto next = [&](unsigned m) { return (rng = rng * 1664525u + 1013904223u, (rng >> 8) % m); };
  for (int i = 0; i < 6000; ++i) {
    const int n = 1 << next(13), planes = next(2) ? 4 : 1;
    const int units = 1 + (int)next(1u << next(14)), turns = 1 + (int)next(1u << next(18));
    SplitProblem p = problem(n, planes, units, turns, next(2));
    if (next(4) == 0) p.units = std::max(1, p.units / 8);
    int a = 0, b = 0;
    const Split s = split_groups_and_chunks(p, &a), e = every(p, &b);
    ++compared;
    // without counters nothing but a cluster or a kernel sums the chunks
    const int sets = p.groups / s.gps, ub = (p.units + sets - 1) / sets;
    if (!p.counters && s.chunks > 1 && !s.finalize && !small_clustered(s.chunks, ub * s.chunks, p.sms)) {
      ++differ;
      printf("counters used: n %d planes %d units %d turns %d\n", n, planes, units, turns);
    }
    if (s.gps != e.gps || s.chunks != e.chunks || s.cost != e.cost) {
      if (++differ <= 10)
        printf("differ n %d planes %d units %d turns %d: %d x %d, every count %d x %d\n", n, planes, units, turns, s.gps,
               s.chunks, e.gps, e.chunks);
    }
  }
  printf("compared %d differ %d\n", compared, differ);
  const int shapes[][4] = {{256, 1, 1, 4096}, {64, 1, 1, 20000}, {8, 1, 1, 1000000}, {8, 1, 1, 131072}, {8, 4, 1, 131072},
                           {64, 1, 1, 100000}, {256, 1, 4, 8192}, {16, 1, 2, 65536}, {512, 4, 30, 640}, {64, 1, 3000, 4096}};
  for (const auto& s : shapes) {
    const SplitProblem p = problem(s[0], s[1], s[2], s[3], true);
    int a = 0, b = 0;
    split_groups_and_chunks(p, &a);
    every(p, &b);
    printf("tried %d of %d\n", a, b);
  }
  // One unit's partial sums, summed by one CTA, cost more than chunks beyond a
  // cluster's save.
  for (int n : {1024, 2048, 4096}) {
    const Split s = split_groups_and_chunks(problem(n, 4, 1, 64, false));
    printf("chunks %d %d\n", s.chunks, s.finalize ? 1 : 0);
  }
  // Two spectra whose sums within a pair of CTAs take longer than the second one.
  for (int n : {2048, 4096}) printf("pair %d\n", split_groups_and_chunks(problem(n, 4, 1, 2, false)).chunks);
  return differ != 0;
}
