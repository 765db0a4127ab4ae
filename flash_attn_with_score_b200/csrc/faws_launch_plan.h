// Host side of the forward launches: the row count of a CTA and the work lists of persistent launches.  Plain C++, compiled
// into the library and, alone, into its tests.
#pragma once
#include <algorithm>
#include <cstdint>
#include <cstring>
#include <functional>
#include <queue>
#include <utility>
#include <vector>

namespace faws {

constexpr int kPlanTile = 128;  // query rows and keys of a tile

// Persistent launches: one CTA per SM walks a list of work items (an item is what one CTA of the
// plain launch does: a row block of one head), in the order of the plain launch's grid.  The
// lists are made on the host (longest item first onto the least loaded CTA) and travel as a
// kernel parameter, so that no device-side counter is shared between launches; launches with
// more items than the lists hold deal the items to the CTAs in rounds of alternating direction.
constexpr int kMaxListedItems = 2048;
constexpr int kMaxListCtas = 192;
struct WorkList {
  int n_items;  // 0: plain launch, every CTA does the item its block index names
  int listed;   // 1: CTA c does ids[start[c]] .. ids[start[c + 1] - 1]
  int gx, gy, gz;  // the grid of the plain launch; an item is a linear block index of it (x fastest)
  uint16_t start[kMaxListCtas + 1];
  uint16_t ids[kMaxListedItems];
};

// The plain launch a list is made for.
struct WorkShape {
  int gx, gy, gz, lpt, causal, p_seq, m_begin, m_end, N, rows, ctas, pack_m;
  bool operator==(const WorkShape& o) const { return std::memcmp(this, &o, sizeof(WorkShape)) == 0; }
};

// Cost of the work items of each row block, by the block's place on the grid's row-block axis, which is heaviest first.
inline std::vector<int> block_costs(const WorkShape& sh) {
  const int ncb = sh.lpt ? sh.gz : sh.gx;
  std::vector<int> cost(ncb);
  for (int slot = 0; slot < ncb; ++slot) {
    const int r0 = sh.m_begin + (ncb - 1 - slot) * sh.rows;
    int tiles = 0;
    for (int t = 0; t * kPlanTile < sh.rows; ++t) {
      const int r = r0 + t * kPlanTile;
      int hi = 0;
      if (r < sh.m_end)
        hi = sh.causal && sh.pack_m == 0 ? std::max(0, std::min(sh.N, sh.p_seq + std::min(r + kPlanTile, sh.m_end))) : sh.N;
      tiles = std::max(tiles, (hi + kPlanTile - 1) / kPlanTile);
    }
    cost[slot] = 19 * tiles + 30;  // measured on cfg3: 1.90 us per key tile + 3.0 us per item (unit 0.1 us)
  }
  return cost;
}

// Fewer than two items per CTA: heaviest item first, those of equal cost in launch order (neighbours share K and V: full S512
// H144 20.4 us, 20.9 row block by row block), each to the CTA with the least work so far (the first of them), and no exchanges after
// that (below), which would not make the heaviest CTA lighter.  A few microseconds at most, for kernels of 20 to 70;
// with a sort of the items, a heap of the CTAs and exchanges it was 65 to 160: sixteen lengths around causal S2048 H28
// D128, a call among others 122 us, the 128-row launch without a list 55.  The CTAs wait in bins of equal load, so that a step
// takes the lowest bit of the first bin.  (Pairing the items off from both ends is simpler still and makes no CTA heavier, but
// causal B5 H12 S1024 D128 took 32.1 us for 31.8, with row sums 34.9 for 34.1.)
inline void deal_short(const WorkShape& sh, const std::vector<int>& cost, WorkList* wl) {
  const int n = wl->n_items, ncb = (int)cost.size(), per_block = n / ncb;
  uint16_t order[2 * kMaxListCtas], of[2 * kMaxListCtas];  // the items, heaviest first; their CTAs
  for (int slot = 0, k = 0; slot < ncb;) {
    int end = slot + 1;
    while (end < ncb && cost[end] == cost[slot]) ++end;
    if (sh.lpt) {  // row blocks are the slowest axis of the grid: launch order
      for (const int to = end * per_block; k < to; ++k) order[k] = (uint16_t)k;
    } else {
      for (int rest = 0; rest < per_block; ++rest)
        for (int x = slot; x < end; ++x) order[k++] = (uint16_t)(x + rest * sh.gx);
    }
    slot = end;
  }
  struct Bin {
    int load;
    uint64_t ctas[kMaxListCtas / 64];
  };
  std::vector<Bin> bins;  // lightest last
  auto put = [&](int load, int cta) {
    size_t at = bins.size();
    while (at > 0 && bins[at - 1].load < load) --at;
    if (at == 0 || bins[at - 1].load != load) bins.insert(bins.begin() + at, Bin{load, {}});
    else --at;
    bins[at].ctas[cta >> 6] |= uint64_t(1) << (cta & 63);
  };
  for (int k = 0; k < n; ++k) {
    int cta = k, load = 0;
    if (k >= sh.ctas) {
      Bin& lightest = bins.back();
      int w = 0;
      while (lightest.ctas[w] == 0) ++w;
      cta = w * 64 + __builtin_ctzll(lightest.ctas[w]);
      load = lightest.load;
      lightest.ctas[w] &= lightest.ctas[w] - 1;
      bool empty = true;
      for (uint64_t word : lightest.ctas) empty = empty && word == 0;
      if (empty) bins.pop_back();
    }
    of[k] = (uint16_t)cta;
    put(load + cost[k / per_block], cta);
  }
  uint16_t count[kMaxListCtas] = {};
  for (int k = 0; k < n; ++k) ++count[of[k]];
  wl->start[0] = 0;
  for (int c = 0; c < kMaxListCtas; ++c) wl->start[c + 1] = (uint16_t)(wl->start[c] + count[c]);
  uint16_t at[kMaxListCtas];
  std::memcpy(at, wl->start, sizeof(at));
  for (int k = 0; k < n; ++k) wl->ids[at[of[k]]++] = order[k];  // (a CTA's items come heaviest first)
}

// Work lists of a persistent launch.  An item costs its key tiles plus a fixed part; the items, heaviest
// first, go one by one to the CTA with the least work so far (what the hardware does with the CTAs of a
// plain launch, here decided ahead).  Made once per problem geometry and kept for the next call.
// false: the launch should stay a plain one
inline bool make_work_list(const WorkShape& sh, WorkList* out) {
  const int n_items = sh.gx * sh.gy * sh.gz, ctas = sh.ctas;
  if (ctas > kMaxListCtas || n_items <= ctas || n_items > 65535) return false;
  const bool listed = n_items <= kMaxListedItems;
  if (!listed && sh.causal) return false;  // unequal items in no useful order: leave them to the hardware
  if (n_items < 2 * ctas) {
    *out = WorkList{n_items, 1, sh.gx, sh.gy, sh.gz, {}, {}};
    deal_short(sh, block_costs(sh), out);
    return true;
  }
  thread_local WorkShape last_shape{};
  thread_local WorkList last{};
  if (last.n_items > 0 && sh == last_shape) {
    *out = last;
    return true;
  }
  WorkList& wl = last;
  wl = WorkList{};
  wl.n_items = n_items;
  wl.listed = listed ? 1 : 0;
  wl.gx = sh.gx;
  wl.gy = sh.gy;
  wl.gz = sh.gz;
  if (listed) {
    const std::vector<int> cost = block_costs(sh);
    auto cost_of = [&](int item) {
      const int ix = item % wl.gx, iz = item / (wl.gx * wl.gy);
      return cost[sh.lpt ? iz : ix];
    };
    std::vector<int> order(n_items);
    for (int i = 0; i < n_items; ++i) order[i] = i;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return cost_of(a) > cost_of(b); });
    // Heaviest item first onto the CTA with the least work so far (what the hardware does with the CTAs
    // of a plain grid), then exchanges of single items between any two CTAs that bring their loads closer
    // together, fuller CTAs first against the emptiest.  Exchanges keep the number of items per CTA, so
    // the result does not lean on the fixed cost per item, which differs between the hooks (3 us plain,
    // 6 us with the column hook, measured on cfg3; packing to a capacity instead put up to 30 small items
    // on one CTA and was 30 % slower under the column hook).  cfg3: 48..56 key tiles per CTA -> 50..52.
    std::vector<std::vector<uint16_t>> mine(ctas);
    std::vector<long long> load(ctas, 0);
    {
      using Load = std::pair<long long, int>;  // (work so far, CTA)
      std::priority_queue<Load, std::vector<Load>, std::greater<Load>> heap;
      for (int c = 0; c < ctas; ++c) heap.push({0, c});
      for (int item : order) {
        Load l = heap.top();
        heap.pop();
        mine[l.second].push_back((uint16_t)item);
        load[l.second] = l.first + cost_of(item);
        heap.push({load[l.second], l.second});
      }
    }
    for (int round = 0; round < 32; ++round) {
      bool improved = false;
      std::vector<int> by_load(ctas);
      for (int c = 0; c < ctas; ++c) by_load[c] = c;
      std::stable_sort(by_load.begin(), by_load.end(), [&](int x, int y) { return load[x] > load[y]; });
      for (int ai = 0; ai < ctas; ++ai) {
        const int A = by_load[ai];
        for (int bi = ctas - 1; bi >= 0; --bi) {
          const int B = by_load[bi];
          const long long gap = load[A] - load[B];
          if (gap <= 0) break;  // (the order is the one before this round's exchanges: good enough)
          long long best_gain = 0, best_d = 0;
          int bia = -1, bib = -1;
          for (size_t ia = 0; ia < mine[A].size(); ++ia)
            for (size_t ib = 0; ib < mine[B].size(); ++ib) {
              const long long d = cost_of(mine[A][ia]) - cost_of(mine[B][ib]);
              if (d <= 0 || d >= gap) continue;
              const long long after = gap - 2 * d;
              const long long gain = gap - (after < 0 ? -after : after);  // how much closer the two get
              if (gain > best_gain) { best_gain = gain; best_d = d; bia = (int)ia; bib = (int)ib; }
            }
          if (bia < 0) continue;
          std::swap(mine[A][bia], mine[B][bib]);
          load[A] -= best_d;
          load[B] += best_d;
          improved = true;
        }
      }
      if (!improved) break;
    }
    for (int c = 0; c < ctas; ++c)  // heaviest item first within a CTA
      std::stable_sort(mine[c].begin(), mine[c].end(), [&](uint16_t x, uint16_t y) { return cost_of(x) > cost_of(y); });
    int at = 0;
    for (int c = 0; c < ctas; ++c) {
      wl.start[c] = (uint16_t)at;
      for (uint16_t id : mine[c]) wl.ids[at++] = id;
    }
    for (int c = ctas; c <= kMaxListCtas; ++c) wl.start[c] = (uint16_t)at;
  }
  last_shape = sh;
  *out = wl;
  return true;
}


// The row count of a CTA, for launches of fewer than two 256-row CTAs per SM (above, 256 rows always).  128-row CTAs, whose two
// warpgroups split the key tiles, shorten the chain of dependent key tiles of launches with few CTAs; they fetch each K / V
// tile twice as often and are launched plainly, where 256-row ones walk balanced lists.
struct RowChoice {
  long long heads;  // of all batches
  int m_begin, m_end, N, p_seq, causal, sms;
  int blocks(int rows) const { return (m_end - m_begin + rows - 1) / rows; }
};
enum RowChoiceKind { kPlainOut, kWithRowSums, kWithColSums };

// us: of a CTA, of a key tile, of a launch; how much the CTAs of unequal length of a launch of two waves and more add to it; of a
// CTA without a visible key; of a key tile of a last row block that is not whole (column sums: such a block reduces every
// tile itself)
struct LaunchFit {
  double fix, per, base, uneven, empty, ragged;
};
// Fitted to 1 576 launches of either row count, for the choice between the two more than for the times (fp16 and bf16,
// multi-head and grouped, head dims 32 to 128, M 129 to 4096 rows against 129 to 4096 keys, M < N, M = N and M > N, 75 to
// 295 256-row CTAs, causal and not).
inline const LaunchFit& launch_fit(bool d128, RowChoiceKind kind, int rows) {
  static constexpr LaunchFit kFits[3][2][2] = {  // [kind][D = 128][128 rows]
      {{{4.51, 1.59, 1.01, 1.00, 4.02, 0.0}, {4.51, 0.81, 0.27, 1.09, 1.66, 0.0}},
       {{4.66, 1.81, 2.08, 1.00, 0.01, 0.0}, {4.88, 0.98, 0.76, 1.12, 2.06, 0.0}}},
      {{{5.20, 1.70, 1.17, 1.05, 0.00, 0.0}, {4.89, 0.86, 0.58, 1.07, 1.93, 0.0}},
       {{5.58, 1.86, 2.01, 1.07, 0.00, 0.0}, {5.41, 1.04, 0.85, 1.08, 2.59, 0.0}}},
      {{{6.62, 1.77, 6.52, 1.36, 0.00, 1.21}, {7.30, 0.98, 4.18, 1.31, 1.49, 0.91}},
       {{7.96, 2.04, 6.75, 1.33, 0.00, 1.14}, {8.52, 1.14, 5.20, 1.24, 1.48, 0.89}}}};
  return kFits[kind][d128 ? 1 : 0][rows == 128 ? 1 : 0];
}

// A lower bound of the launch's makespan, one CTA per SM at a time (the longest CTA, the mean load, and what the j SMs + 1
// longest CTAs force onto one SM), lengthened where it takes several waves of unequal CTAs.  The row blocks of a head get
// heavier towards its end (causal) or are alike, and every head has the same ones.
inline double expected_us(const RowChoice& c, bool d128, RowChoiceKind kind, int rows) {
  const LaunchFit& f = launch_fit(d128, kind, rows);
  const int ncb = c.blocks(rows);
  const long long n = ncb * c.heads;
  auto job = [&](int cb) -> double {
    const int end = std::min(c.m_begin + (cb + 1) * rows, c.m_end);
    const int hi = c.causal ? std::max(0, std::min(c.N, c.p_seq + end)) : c.N;
    const int tiles = (hi + kPlanTile - 1) / kPlanTile;
    const bool ragged = cb == ncb - 1 && (c.m_end - c.m_begin) % kPlanTile != 0;
    return tiles == 0 ? f.empty : f.fix + (f.per + (ragged ? f.ragged : 0.0)) * tiles;
  };
  auto ranked = [&](long long i) -> double { return i < n ? job(ncb - 1 - (int)(i / c.heads)) : 0.0; };
  double total = 0.0;
  for (int cb = 0; cb < ncb; ++cb) total += job(cb);
  const double longest = job(ncb - 1);
  double us = std::max(longest, total * (double)c.heads / c.sms);
  for (int j = 1; j <= 3 && (long long)j * c.sms < n; ++j) {
    double sum = 0.0;
    for (int x = 0; x <= j; ++x) sum += ranked((long long)j * c.sms - x);
    us = std::max(us, sum);
  }
  if (n <= c.sms || longest <= 0.0) return f.base + us;
  return f.base + us * (1.0 + (f.uneven - 1.0) * (1.0 - job(0) / longest) * std::min(1.0, (double)(n - c.sms) / c.sms));
}

// 256 rows have to be expected 3 % faster, 4 % where there are column sums.  Of 4 605 such launches with each row count
// 2 943 take 256, 14 of which run more than 2 % slower than with 128 (5.5 % at most); the mean launch is 0.2 % behind the
// better of the two.  128 rows everywhere are 8 to 11 % slower in the mean, up to 1.5 times: causal D128 S2048 H32 48.4 and
// 39.4 us, full S512 H144 34.7 and 23.1, S1024 H64 48.0 and 36.5; the other way causal S2048 H8 19.2 and 33.4, full S2048
// H24 57.4 and 63.3, causal M2048 N700 H20 with column sums, where most row blocks see no key, 18.7 and 26.9.
inline bool prefer_256_rows(const RowChoice& c, bool d128, RowChoiceKind kind) {
  const double small = expected_us(c, d128, kind, 128), large = expected_us(c, d128, kind, 256);
  return small > (kind == kWithColSums ? 1.04 : 1.03) * large;
}
}  // namespace faws
