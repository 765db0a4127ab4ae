// Host side of the forward launches: the work lists of persistent launches.  Plain C++, compiled into the library and,
// alone, into its test.
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

// Fewer than two items per CTA: the heaviest items one to a CTA, then the rest back from the last CTA, so that the lightest
// of the first round get the heaviest that are left.  Along the grid's row-block axis the items come heaviest first, and
// every head has the same, so that nothing is sorted or weighed.  Over S 128 to 8192 and all head counts with 149 to 295 items the
// heaviest CTA is never heavier than in the list that greedy dealing and exchanges make (below), which takes 65 to 160 us of host time,
// three times the kernel where every call has another length: sixteen lengths around causal S2048 H28 D128, a call among
// others 122 us with that list; the 128-row launch without one 55.
inline void deal_pairs(const WorkShape& sh, WorkList* wl) {
  const int n = wl->n_items, ncb = sh.lpt ? sh.gz : sh.gx, per_block = n / ncb;
  auto ranked = [&](int k) -> uint16_t {  // k-th item, heaviest first
    if (sh.lpt) return (uint16_t)k;       // row blocks are the slowest axis: launch order
    return (uint16_t)(k / per_block + k % per_block * sh.gx);
  };
  int at = 0;
  for (int c = 0; c < sh.ctas; ++c) {
    wl->start[c] = (uint16_t)at;
    wl->ids[at++] = ranked(c);
    if (2 * sh.ctas - 1 - c < n) wl->ids[at++] = ranked(2 * sh.ctas - 1 - c);
  }
  for (int c = sh.ctas; c <= kMaxListCtas; ++c) wl->start[c] = (uint16_t)at;
}

// Work lists of a persistent launch.  An item costs its key tiles plus a fixed part; the items, heaviest
// first, go one by one to the CTA with the least work so far (what the hardware does with the CTAs of a
// plain launch, here decided ahead).  Made once per problem geometry and kept for the next call.
// (Fewer than two items per CTA are dealt in pairs.)
// false: the launch should stay a plain one
inline bool make_work_list(const WorkShape& sh, WorkList* out) {
  const int n_items = sh.gx * sh.gy * sh.gz, ctas = sh.ctas;
  if (ctas > kMaxListCtas || n_items <= ctas || n_items > 65535) return false;
  const bool listed = n_items <= kMaxListedItems;
  if (!listed && sh.causal) return false;  // unequal items in no useful order: leave them to the hardware
  if (n_items < 2 * ctas) {
    *out = WorkList{n_items, 1, sh.gx, sh.gy, sh.gz, {}, {}};
    deal_pairs(sh, out);
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

}  // namespace faws
