"""Work lists of persistent launches: every item once, no CTA heavier than greedy dealing makes one, and no more host time
than a launch of that size is worth."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flash_attn_with_score_b200", "csrc")

PROGRAM = r"""
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include "faws_launch_plan.h"
using namespace faws;

static int cost(const WorkShape& s, int item) {  // the cost model of the lists: 1.9 us a key tile, 3 us an item
  const int ncb = s.lpt ? s.gz : s.gx, slot = s.lpt ? item / (s.gx * s.gy) : item % s.gx;
  int tiles = 0;
  for (int t = 0; t * 128 < s.rows; ++t) {
    const int r = s.m_begin + (ncb - 1 - slot) * s.rows + t * 128;
    if (r >= s.m_end) continue;
    const int hi = s.causal ? std::max(0, std::min(s.N, s.p_seq + std::min(r + 128, s.m_end))) : s.N;
    tiles = std::max(tiles, (hi + 127) / 128);
  }
  return 19 * tiles + 30;
}

int main(int argc, char** argv) {
  // H B M N causal lpt m_begin
  const int H = atoi(argv[1]), B = atoi(argv[2]), M = atoi(argv[3]), N = atoi(argv[4]), causal = atoi(argv[5]);
  const int lpt = atoi(argv[6]), m_begin = atoi(argv[7]), ctas = 148, ncb = (M - m_begin + 255) / 256;
  const WorkShape s{lpt ? H : ncb, lpt ? B : H, lpt ? ncb : B, lpt, causal, N - M, m_begin, M, N, 256, ctas, 0};
  const int n = s.gx * s.gy * s.gz;
  WorkList wl;
  if (!make_work_list(s, &wl) || !wl.listed || wl.n_items != n) return printf("no list\n"), 1;
  std::vector<int> seen(n, 0), load;
  for (int c = 0; c < ctas; ++c) {
    int sum = 0, last = 1 << 30;
    for (int k = wl.start[c]; k < wl.start[c + 1]; ++k) {
      if (wl.ids[k] >= n || seen[wl.ids[k]]++) return printf("item %d twice or out of range\n", wl.ids[k]), 1;
      if (cost(s, wl.ids[k]) > last) return printf("a CTA's heaviest item is not its first\n"), 1;
      last = cost(s, wl.ids[k]);
      sum += last;
    }
    if (wl.start[c] == wl.start[c + 1]) return printf("a CTA without work\n"), 1;
    load.push_back(sum);
  }
  if (wl.start[0] != 0 || wl.start[ctas] != n) return printf("%d of %d items\n", wl.start[ctas], n), 1;
  std::vector<int> all;
  for (int i = 0; i < n; ++i) all.push_back(cost(s, i));
  std::sort(all.rbegin(), all.rend());
  std::priority_queue<int, std::vector<int>, std::greater<int>> heap;
  for (int c = 0; c < ctas; ++c) heap.push(0);
  int greedy = 0;
  for (int x : all) {
    const int l = heap.top() + x;
    heap.pop();
    heap.push(l);
    greedy = std::max(greedy, l);
  }
  const int heaviest = *std::max_element(load.begin(), load.end());
  if (heaviest > greedy) return printf("heaviest CTA %d, greedy %d\n", heaviest, greedy), 1;
  // every call another geometry (the window's end moves within the last row block)
  std::vector<double> us;
  for (int k = 0; k < 200; ++k) {
    WorkShape t = s;
    t.N -= k & 1;
    t.p_seq -= k & 1;
    const auto a = std::chrono::steady_clock::now();
    make_work_list(t, &wl);
    us.push_back(std::chrono::duration<double, std::micro>(std::chrono::steady_clock::now() - a).count());
  }
  std::sort(us.begin(), us.end());
  printf("%f\n", us[100]);
  return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("lists")
    src, exe = str(d / "lists.cpp"), str(d / "lists")
    with open(src, "w") as f:
        f.write(PROGRAM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-Wall", "-Werror", "-I", CSRC, "-o", exe, src], check=True)
    return exe


SHORT = [  # fewer than two items for each of 148 CTAs
    (28, 1, 2048, 2048, 1), (40, 1, 1531, 1531, 1), (16, 1, 4096, 4096, 1), (144, 1, 512, 512, 0), (75, 1, 300, 300, 1),
    (149, 1, 130, 777, 1), (5, 59, 256, 100, 1), (1, 149, 700, 33, 0), (8, 1, 9400, 9400, 1), (295, 1, 200, 4096, 0)]
LONG = [(32, 1, 8192, 8192, 1), (28, 1, 4096, 4096, 1), (37, 4, 512, 512, 0)]


@pytest.mark.parametrize("lpt", [0, 1])
@pytest.mark.parametrize("H,B,M,N,causal", SHORT + LONG)
def test_list(program, H, B, M, N, causal, lpt):
    for m_begin in (0, 128):
        items = H * B * -(-(M - m_begin) // 256)
        if not 148 < items <= 2048:
            continue
        r = subprocess.run([program] + [str(x) for x in (H, B, M, N, causal, lpt, m_begin)], capture_output=True, text=True)
        assert r.returncode == 0, r.stdout
        if items < 2 * 148:  # kernels of 20 to 70 us: a list may not take a tenth of one (10 times what it takes here)
            assert float(r.stdout) < 5.0, r.stdout
