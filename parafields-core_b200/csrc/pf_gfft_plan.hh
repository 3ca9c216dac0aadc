// pf_gfft_plan.hh -- radix schedules and tile sizes of the any-length passes (pf_gfft.cuh).
#pragma once

#include <algorithm>
#include <map>
#include <mutex>
#include <vector>

#include "pf_gfft.cuh"

using namespace pf;

// Radix schedule of a transform length, descending; empty when it has a prime factor above 13.
// The cost of a stage per element: shared-memory access, twiddle and barrier (the constant),
// index arithmetic per butterfly (over R) and the butterfly itself.
static double g_radix_cost(int R) {
  static const double arith[14] = {0, 0, .05, .15, .1, .25, .25, .5, .25, .35, .35, 1.2, 9., 1.5};
  return 0.6 + 1.2 / R + arith[R];
}

static void g_search(int x, int top, std::vector<int>& cur, double cost, std::vector<int>& best, double& best_cost) {
  if (x == 1) {
    if (cost < best_cost) {
      best_cost = cost;
      best = cur;
    }
    return;
  }
  if ((int)cur.size() == kGStages) return;
  for (int R = std::min(top, x); R >= 2; R--)
    if (R != 12 && R != 9 && R != 10 && x % R == 0 && cost + g_radix_cost(R) < best_cost) {
      cur.push_back(R);
      g_search(x / R, R, cur, cost + g_radix_cost(R), best, best_cost);
      cur.pop_back();
    }
}

struct GSched {
  std::vector<int> r;
  double cost = 1e300;
};
static std::mutex g_sched_mu;

static const GSched& g_schedule_locked(int N) {  // entries stay in place
  static std::map<int, GSched> cache;
  auto it = cache.find(N);
  if (it != cache.end()) return it->second;
  GSched s;
  if (N == 1) {
    s.r.push_back(1);
    s.cost = g_radix_cost(1);
  } else {
    std::vector<int> cur;
    g_search(N, 13, cur, 0., s.r, s.cost);
  }
  return cache[N] = s;
}
static const GSched& g_schedule(int N) {
  std::lock_guard<std::mutex> lk(g_sched_mu);
  return g_schedule_locked(N);
}

// transform length of Bluestein's convolution for pencils of length L: the cheapest length
// >= 2 L - 1 with factors 2, 3, 5, 7 (cost per element times length)
static int g_blue_length(int L) {
  std::lock_guard<std::mutex> lk(g_sched_mu);
  static std::map<int, int> cache;
  auto it = cache.find(L);
  if (it != cache.end()) return it->second;
  const int lo = 2 * L - 1;
  int best = 0;
  double bc = 1e300;
  for (int n = lo; n <= lo + lo / 3 + 8; n++) {
    int x = n;
    for (int p : {2, 3, 5, 7})
      while (x % p == 0) x /= p;
    if (x != 1) continue;
    const GSched& s = g_schedule_locked(n);
    if (s.r.size() >= 2 && s.cost * n < bc) {
      bc = s.cost * n;
      best = n;
    }
  }
  cache[L] = best;
  return best;
}

static bool g_smooth(int L) {
  for (int p : {2, 3, 5, 7, 11, 13})
    while (L % p == 0) L /= p;
  return L == 1;
}

static unsigned g_magic(int d) { return d <= 1 ? 0u : (unsigned)(((1ull << 32) + (unsigned)d - 1) / (unsigned)d); }

constexpr size_t kGSmem = 227 * 1024;

// Slots per tile and threads.  Strided tiles take 8 slots (128-byte row segments) while three
// of them fit on an SM, fewer for longer pencils but at least 2 (one 32-byte sector) while two
// fit; row tiles up to 1024 elements, 2048 where the loader computes its values (complex-to-real rows
// of n0 x 96 x 80 fields at 17 lengths 32..512, tiles of 1024 against 2048 elements, us: FP32 192
// points 11.6 against 13.0, 256 13.1 / 14.5, 384 21.9 / 23.1, FP64 250 27.4 / 29.3, 500 46 / 50; the
// others within 3%, but 400 points 25.2 / 24.7 and 40.8 / 36.4; 192-point FP32 rows beside another
// stream's passes 74 / 87).  Fewer slots where the grid would leave SMs idle.  Threads: the count
// with the least estimated time, which is rounds of butterflies (and of loader pairs) per tile over
// the tiles that run at once on an SM within 1024 threads, the tile's shared memory and the grid.
static void g_tile(int slots, const std::vector<int>& r, bool rows, bool direct, int pitch, long long nslots,
                   long long nouter, int sms, int* B_out, int* nt_out) {
  const size_t per = (size_t)16 * pitch;
  int B = 1;
  if (rows) {
    while (B < 32 && 2 * B * slots <= (direct ? 1024 : 2048) && 2 * B * per <= kGSmem / 3) B *= 2;
  } else {
    B = 8;
    while (B > 2 && B * per > kGSmem / 3) B /= 2;
    while (B > 1 && B * per > kGSmem) B /= 2;
  }
  while (B > 1 && (nslots + B - 1) / B * nouter < 2LL * sms && (rows || B > 2 || nslots * nouter < sms)) B /= 2;
  const long long grid = (nslots + B - 1) / B * nouter;
  const long long fit = std::min<long long>(std::max<size_t>(1, kGSmem / (B * per + 1024)), (grid + sms - 1) / sms);
  // kernels that go through shared memory often share the SMs with others (ensembles): blocks of
  // at most half the threads unless there are only a few
  const int top = !direct && grid > sms / 4 ? kGThreads / 2 : kGThreads;
  // work items of the widest step
  const long long wide = (long long)B * slots / (direct ? *std::min_element(r.begin(), r.end()) : 2);
  double best = 1e300;
  *nt_out = 32;
  for (int nt = 32; nt <= top && nt < wide + 32; nt += 32) {
    double t = 0.;
    for (int R : r) t += (double)(((long long)B * (slots / R) + nt - 1) / nt) * (R + 4);
    if (!direct) t += (double)(((long long)B * slots / 2 + nt - 1) / nt) * 60.;
    t *= (1. + 32. / nt) / (double)std::min<long long>(kGThreads / nt, fit);
    if (t < best * 0.999) {
      best = t;
      *nt_out = nt;
    }
  }
  *B_out = B;
}

// lengths, stages and divisors of a pass (mode, mid: as in k_g; rows: row tiles)
template <typename T, bool ROWS>
static void g_fill(GArgs<T>& a, const GSched& sc, int N, int L, int Lout, int mode, bool mid) {
  a.N = N;
  a.S = (int)sc.r.size();
  a.L = L;
  a.Lout = Lout;
  int m = N, rest = 1, tw = 0;
  for (int s = 0; s < a.S; s++) {
    GStage& g = a.st[s];
    g.block = m;
    g.R = sc.r[s];
    m /= g.R;
    g.M = m;
    g.nb = N / g.R;
    if (s > 1) rest *= sc.r[s - 1];
    g.rest = rest;
    g.tw = tw;
    tw += (g.R - 1) * m;
    g.mM = g_magic(g.M);
    g.mnb = g_magic(g.nb);
    g.mrest = g_magic(g.rest);
    g.mR = g_magic(g.R);
  }
  const int M1 = a.st[0].M, R1 = a.st[0].R;
  // an odd distance of the sub-blocks of a row; rows that fill shared memory go without
  a.M1p = ROWS && M1 % 2 == 0 && (size_t)16 * (N + R1) <= kGSmem ? M1 + 1 : M1;
  a.pitch = a.M1p * R1;
  a.mL = g_magic(L);
  // items per slot of the store phase
  a.mLout = g_magic(mode == 1 ? L / 2 + 1 : (mode == 2 ? (Lout + 1) / 2 : (mid ? std::min(Lout, L) : Lout)));
}
