// How k_small's units are split over groups and CTAs: plain host code.
//
// A unit's spectra are taken in turns (a spectrum, or two of one
// polarisation) by `gps` groups of threads of each of `chunks` CTAs.  The
// allocation-free entry point plans in every call, before a kernel of 8 to 30
// us, so the search looks only at counts that can win.  One channel of 10^6
// spectra of 8 points: every count of every number of groups 9124 and 80 us of
// an x86 core, these 320 and 4.8; 20000 spectra of 64 points 47 -> 3.0 us.  The
// split found is the same.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstddef>

namespace rsg {

// Whether a launch of `ctas` CTAs whose units are spread over `chunks` of them
// runs these as a cluster.  Up to 8 (what every GPU takes) while every CTA has
// an SM of its own, else pairs: a larger cluster waits for that many places in
// one cluster of SMs.  Four units of 8 x 2048 points in four planes: 28 us
// without, 27 with pairs, 12 with 8; 64 Mi samples of 2048 points in four
// planes, 1024 CTAs: 278 without, 256 with pairs, 259 with 4, 267 with 8; four
// products in four planes, 4096 to 8 points: 108, 110, 110, 121.  (Launches that
// share a grid have no clusters: their units' last CTAs sum.)
constexpr int kSmallCluster = 8;
inline bool small_clustered(int chunks, int ctas, int sms) {
  return chunks == 2 || (chunks > 1 && chunks <= kSmallCluster && ctas <= sms);
}

struct SplitProblem {
  int turns = 1;        // of a unit
  int units = 1;        // of the launch
  int all_units = 1;    // of the product (what the scratch is sized for)
  int groups = 1;       // of a CTA
  int planes = 1, n = 1, radix = 1;  // output planes, FFT length, values per thread
  int threads = 1;      // of a CTA
  int target_ctas = 1;  // CTAs that fill the GPU
  int sms = 0, occ = 0; // of the device, and resident CTAs per SM (0: unknown)
  double unit_us = 0;   // SM time of one iteration of a CTA
  std::size_t max_partial = 0;  // floats of partial sums (0: no limit)
  bool counters = true;         // arrival counters: a unit's last CTA may sum it
};
struct Split {
  int gps = 1, chunks = 1;
  bool finalize = false;  // the chunks are summed by a kernel of its own
  double cost = 0;  // microseconds
};

// Times in microseconds of a launch with every count of chunks.
struct SplitCost {
  double unit;     // SM time of one iteration of a CTA
  double partial;  // traffic of one chunk's partial sums of every unit
  double serial;   // the last CTA's reading of one chunk's partial sums
  double outputs;  // of a CTA's units, for each of its threads
  int sms, occ;
  bool kernel;     // chunks beyond a cluster are summed by a kernel, not by the last CTA

  // Iterations of a CTA with `per` turns.
  static int iterations(unsigned per, unsigned gps) { return (int)((per + gps - 1) / gps); }
  // CTAs of the most loaded SM with `ctas` in all.
  int on_one_sm(int ctas) const { return (int)((unsigned)(ctas + sms - 1) / (unsigned)sms); }
  bool finalize(int c, int ublocks) const { return kernel && c > 1 && !small_clustered(c, ublocks * c, sms); }
  double sum(int c, int ublocks) const {
    if (c == 1) return 0.0;
    if (small_clustered(c, ublocks * c, sms)) return 0.5 + 0.15 * outputs / c;
    return kernel ? 4.0 + c * (partial + 0.04) : 2.0 + c * (partial + serial);
  }
  // SM time of an iteration of all of them, over that of one
  double load(int per_sm) const {
    return std::max((double)per_sm, 1.5 * (int)((unsigned)(per_sm + occ - 1) / (unsigned)occ));
  }
  double cost(int iters, double load, double sum_us) const { return (iters + 0.6) * unit * load + sum_us; }
};

// Chunks per unit: the split with the shortest schedule.  A launch lasts as
// long as its most loaded SM: ceil(CTAs / SMs) CTAs of `iters` iterations each
// (an SM with fewer CTAs resident than it holds loses little, so a split over
// occupancy slots would be the wrong measure: 1024 CTAs of N = 64 run in
// 127 us, 512 twice as long ones in 143, 2560 in 124), plus about 0.6
// iterations for a CTA's start and reduction; a CTA alone on its SM is bound
// by its own latency, about 1.5 times its share of a full one.  A unit split
// within a cluster adds about 0.5 us and 0.15 for each output that a thread sums
// (two spectra of 4096 points in four planes: one CTA 10.3 us a call, a pair, 32
// outputs a thread, 14.4); one split over more CTAs the traffic of the partial
// sums, and an arrival and their sum by one CTA (36 GB/s) or a kernel over all
// outputs.
//
// Counts of a cluster are all looked at.  Of larger ones that load the SMs alike
// and leave a CTA as many iterations the smallest is the best (the sum costs more
// with every chunk), so the search goes from one such count to the next with few
// enough iterations to win, and over all that load them alike if the fewest among
// them would not.  *tried: counts looked at.
inline int fit_chunks(int turns, int gps, int ublocks, int c_lo, int c_hi, const SplitCost& k, double* cost_of,
                      int* tried = nullptr) {
  // (32-bit divisions: they are most of the search's time)
  auto ceil_div = [](unsigned a, unsigned b) { return (int)((a + b - 1) / b); };
  int best = c_lo;
  double best_cost = 1e300;
  int c = c_lo;
  for (; c <= std::min(c_hi, kSmallCluster); ++c) {
    const int per = ceil_div(turns, c);
    if (c > c_lo && ceil_div(turns, per) != c) continue;
    if (tried) ++*tried;
    const double cost = k.cost(SplitCost::iterations(per, gps), k.load(k.on_one_sm(ublocks * c)), k.sum(c, ublocks));
    if (cost < best_cost * 0.99) {
      best_cost = cost;
      best = c;
    }
  }
  // the first count from c that no smaller one equals in turns per chunk
  auto distinct = [&](int c) {
    const int per = ceil_div(turns, c);
    return ceil_div(turns, per) == c ? c : per > 1 ? ceil_div(turns, per - 1) : c_hi + 1;
  };
  for (c = distinct(c); c <= c_hi;) {
    // the counts from here that load the most loaded SM alike
    const int per_sm = k.on_one_sm(ublocks * c);
    const int beyond = std::min((int)((unsigned)(per_sm * k.sms) / (unsigned)ublocks), c_hi) + 1;
    const double load = k.load(per_sm);
    if (tried) ++*tried;
    if (k.cost(SplitCost::iterations(ceil_div(turns, beyond - 1), gps), load, k.sum(c, ublocks)) < best_cost * 0.99) {
      while (c < beyond) {
        if (tried) ++*tried;
        const int iters = SplitCost::iterations(ceil_div(turns, c), gps);
        const double sum = k.sum(c, ublocks), cost = k.cost(iters, load, sum);
        if (cost < best_cost * 0.99) {
          best_cost = cost;
          best = c;
        }
        const double most = (best_cost * 0.99 - sum) / (k.unit * load) + 0.4;  // iterations with which one could win
        const int fewer = most < iters - 1 ? (int)most : iters - 1;
        c = fewer >= 1 ? ceil_div(turns, gps * fewer) : beyond;
      }
    }
    c = distinct(beyond);
  }
  *cost_of = best_cost;
  return best;
}

// All turns of all units over all SMs: no split takes less.
inline double least_us(const SplitProblem& p, int gps) {
  const int sets = p.groups / gps, ub = (p.units + sets - 1) / sets;
  return p.turns * (double)ub * p.unit_us / ((double)gps * p.sms);
}

// Chunks of a launch with `gps` groups per unit.  A kernel of its own for the sum
// of the chunks is a launch behind a drained GPU, against a CTA that others' work
// can hide, so it is taken only where the GPU idles: where the best split without
// one takes kIdle times the least.  One channel, 64 spectra of 4096 points in four
// planes (a thirtieth of it busy): 8 chunks in a cluster 33 us, 32 and a kernel
// 19; 8 channels x 256 spectra (a third): a pass among others 36 us without the
// kernel, 41 with it.
constexpr double kIdle = 8.0;
inline Split split_chunks(const SplitProblem& p, int gps, int* tried = nullptr) {
  const int sets = p.groups / gps;
  const int ub = (p.units + sets - 1) / sets;
  const int aim = std::max(1, (p.target_ctas + ub - 1) / ub);  // chunks that fill the GPU
  // partial sums that fit the limit
  const long long floats = (long long)p.all_units * p.planes * p.n;
  int most = (int)std::min<long long>((p.turns + gps - 1) / gps, std::max(8, 4 * aim));
  if (p.max_partial) most = (int)std::min<long long>(most, std::max<long long>(1, (long long)p.max_partial / floats));
  most = std::max(1, most);
  Split s;
  s.gps = gps;
  if (p.occ <= 0) {
    s.chunks = std::min(aim, most);
    s.finalize = s.chunks > 1 && !p.counters;
    return s;
  }
  // partial sums are written and read at about 4 TB/s
  const double sums = (double)sets * p.planes * p.n;
  SplitCost k{p.unit_us, ub * sums * 2e-6, sums * 1.1e-4, sums / p.threads, p.sms, p.occ, !p.counters};
  s.chunks = fit_chunks(p.turns, gps, ub, 1, most, k, &s.cost, tried);
  s.finalize = k.finalize(s.chunks, ub);
  if (p.counters && s.cost > kIdle * least_us(p, gps)) {
    k.kernel = true;
    double cost = 0.0;
    const int c = fit_chunks(p.turns, gps, ub, 1, most, k, &cost, tried);
    if (cost < s.cost) {
      s.chunks = c;
      s.cost = cost;
      s.finalize = k.finalize(c, ub);
    }
  }
  return s;
}

// Groups per unit: at most one per spectrum (or pair of them), few enough that
// every thread of a set has an output to reduce (gps <= |P| * R), and fewer
// where their last iteration would leave too many of them idle (9 spectra on
// eight groups: 16 turns).  64 Mi samples, always as many / by the cost: 64
// points, 17 spectra a unit 264 / 129 us, 256 points in four planes, 9 spectra
// 413 / 240, 1024 points, 5 spectra 275 / 203; powers of two the same either way.
inline Split split_groups_and_chunks(const SplitProblem& p, int* tried = nullptr) {
  auto pow2_floor = [](int x) { int q = 1; while (q * 2 <= x) q *= 2; return q; };
  const int most = std::min(p.groups, std::min(pow2_floor(p.planes * p.radix), pow2_floor(p.turns)));
  Split best = split_chunks(p, most, tried);
  for (int gps = most / 2; gps >= 1 && p.occ > 0; gps /= 2) {
    if (0.999 * least_us(p, gps) >= 0.95 * best.cost) continue;
    const Split s = split_chunks(p, gps, tried);
    if (s.cost < 0.95 * best.cost) best = s;
  }
  return best;
}

}  // namespace rsg
