// How many blocks share the keys of every pair of query tiles in attention_prefill_pair.cu, and for how long such a launch leaves SMs
// idle: a model of the kernel's time (its numbers: ops.prefill_pair_shares), searched here because a step with prompts asks anew each
// time and its first layer waits for the answer. A step of one / two / four / eight portions takes the host 4 / 5 / 7 / 11 us with the call; in Python
// 45 / 77 / 138 / 269.
#include <algorithm>
#include <new>

#include "api.h"
#include "common.cuh"

namespace {

constexpr int BQ = 128, BK = 128, RUNS = 8;    // tokens of an item and keys of a tile; runs of blocks a portion is taken as, at most

struct Run { long long tiles, blocks; };       // key tiles of a block, blocks

struct Runs {
  Run* at = nullptr;
  int n = 0;
  ~Runs() { delete[] at; }
  // portions: (cached, new) tokens
  bool fill(const int* portions, int count, int nh, int nkv, int chunk, int window) {
    at = new (std::nothrow) Run[(size_t)count * RUNS + 1];
    if (!at) return false;
    const long long group = nh / nkv;
    for (int p = 0; p < count; ++p) {
      const long long cached = portions[2 * p], fresh = portions[2 * p + 1];
      const long long items = (fresh + BQ - 1) / BQ * group, pairs = (items + 1) / 2, runs = std::min<long long>(RUNS, pairs);
      for (long long i = 0; i < runs; ++i) {
        const long long a = pairs * i / runs, b = pairs * (i + 1) / runs;
        const long long first = cached + BQ * ((a + b - 1) / group), last = std::min(a + b, items - 1) / group;
        const long long end = std::min(cached + BQ * (last + 1), cached + fresh) - 1;
        long long seen = chunk > 0 ? first / chunk * chunk : 0;
        if (window > 0) seen = std::max(seen, first - window + 1);
        at[n++] = {end / BK - seen / BK + 1, (b - a) * nkv};
      }
    }
    std::sort(at, at + n, [](const Run& x, const Run& y) { return x.tiles > y.tiles; });      // the heaviest start first
    return true;
  }
};

bool bad(const int* portions, int n, int nh, int nkv, int chunk, int window, int sms) {
  if ((!portions && n > 0) || n < 0 || n > (1 << 24) || nkv <= 0 || nh <= 0 || nh % nkv != 0 || chunk < 0 || window < 0 || sms <= 0) return true;
  for (int p = 0; p < n; ++p)
    if (portions[2 * p] < 0 || portions[2 * p + 1] < 0) return true;
  return false;
}

}  // namespace

// portions [n][2] on the host: (cached, new) tokens of every request that brings more than one; rows: the step's. least .. most; 0: bad arguments or no memory.
extern "C" int hb_prefill_pair_shares(const int* portions, int n, int nh, int nkv, int hd, int chunk, int window, long long rows, int sms,
                                      int least, int most) {
  if (bad(portions, n, nh, nkv, chunk, window, sms) || least < 1 || most < least) return 0;
  Runs runs;
  if (!runs.fill(portions, n, nh, nkv, chunk, window)) return 0;
  if (runs.n == 0) return 1;
  const bool small = hd <= 64;
  const double numbers = (double)rows * nh * hd, fixed = small ? 7.75 : 8.4, tile = small ? 1.515 : 1.73;
  const double merge = small ? 1.46 : 1.27, share = small ? 0.6 : 0.63, whole = small ? 6.2 : 4.05;
  auto cost = [&](int k) {
    // a pair takes half a tile more than its share; the launch the longest block, all tiles over all SMs, or the last turn that starts in a run
    double longest = 0., all = 0.;
    long long before = 0, turn = 0;
    for (int i = 0; i < runs.n; ++i) {
      const double t = (double)((runs.at[i].tiles + k - 1) / k) + 0.5;
      const long long blocks = runs.at[i].blocks * k;
      if (i == 0) longest = t;
      all += t * (double)blocks;
      before += blocks;
      if (sms * turn < before) {
        turn = (before - 1) / sms + 1;
        longest = std::max(longest, (double)turn * t);
      }
    }
    return fixed + tile * std::max(longest, all / sms) + (k > 1 ? merge + (share * k + whole) * numbers / 1e6 : 0.);
  };
  int best = least;
  double took = cost(least);
  for (int k = least + 1; k <= most; ++k) {
    const double c = cost(k);
    if (c < took) { took = c; best = k; }
  }
  if (least > 1) return best;
  const double alone = cost(1);
  return took < std::min(0.93 * alone, alone - 8.0) ? best : 1;
}

// Us for which the SMs of such a launch, in one share, are idle on average; 0 for launches of less than `from` us; -1: bad arguments or no memory.
extern "C" double hb_prefill_pair_idle_us(const int* portions, int n, int nh, int nkv, int hd, int chunk, int window, int sms, double from) {
  if (bad(portions, n, nh, nkv, chunk, window, sms)) return -1.;
  Runs runs;
  if (!runs.fill(portions, n, nh, nkv, chunk, window)) return -1.;
  const double tile = hd <= 64 ? 1.515 : 1.73;
  long long longest = 0, all = 0;
  for (int i = 0; i < runs.n; ++i) {
    longest = std::max(longest, runs.at[i].tiles);
    all += runs.at[i].tiles * runs.at[i].blocks;
  }
  return tile * (double)longest >= from ? std::max(0., tile * ((double)longest - (double)all / sms)) : 0.;
}
