// Runs ds_warp_gather.cuh as 32 fibres: between two __syncwarp() the lanes go one after
// another, in every order given, so two stores to one address that no __syncwarp()
// orders land either way round.  Exits 1 where the indices placed are not those of the
// bits, in order.
#include <ucontext.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#define __device__
#define __forceinline__ inline
static int __popc(uint32_t x) { return __builtin_popcount(x); }
static void __syncwarp();
#include "../../diffsplat_b200/csrc/ds_warp_gather.cuh"

static ucontext_t g_main, g_lane[32];
static int g_now;
static bool g_done[32];
static void __syncwarp() { swapcontext(&g_lane[g_now], &g_main); }

static std::vector<uint32_t> g_words;
static uint16_t g_buf[64];
static std::vector<std::vector<int>> g_placed;  // per lane: the index it read at each place()

static void run_lane(int lane) {
  int pend = 0;
  auto place = [&](int n) {
    if (lane < n) g_placed[lane].push_back(g_buf[lane]);
  };
  for (size_t i = 0; i < g_words.size(); ++i)
    if (g_words[i]) pend = ds::warp_gather(g_buf, pend, g_words[i], (int)(32 * i), lane, place);
  __syncwarp();
  if (pend > 0) place(pend);
  g_done[lane] = true;
  swapcontext(&g_lane[lane], &g_main);
}

static std::vector<int> gather(const std::vector<int>& order) {
  static std::vector<std::vector<char>> stacks(32, std::vector<char>(1 << 16));
  g_placed.assign(32, {});
  for (int l = 0; l < 32; ++l) {
    g_done[l] = false;
    getcontext(&g_lane[l]);
    g_lane[l].uc_stack.ss_sp = stacks[l].data();
    g_lane[l].uc_stack.ss_size = stacks[l].size();
    g_lane[l].uc_link = &g_main;
    makecontext(&g_lane[l], (void (*)())run_lane, 1, l);
  }
  while (!std::all_of(g_done, g_done + 32, [](bool d) { return d; }))
    for (int l : order)
      if (!g_done[l]) {
        g_now = l;
        swapcontext(&g_main, &g_lane[l]);
      }
  std::vector<int> out;
  for (size_t p = 0; p < g_placed[0].size(); ++p)
    for (int l = 0; l < 32; ++l)
      if (p < g_placed[l].size()) out.push_back(g_placed[l][p]);
  return out;
}

int main() {
  std::mt19937 rng(1);
  for (int trial = 0; trial < 400; ++trial) {
    g_words.resize(1 + rng() % 32);
    std::vector<int> want;
    const int dense = trial % 4;
    for (size_t i = 0; i < g_words.size(); ++i) {
      g_words[i] = dense == 0 ? rng() & rng() & rng() : dense == 1 ? rng()
                   : dense == 2 ? rng() | rng() : (rng() % 3 ? 0xffffffffu : 0u);
      for (int b = 0; b < 32; ++b)
        if (g_words[i] >> b & 1u) want.push_back((int)(32 * i) + b);
    }
    std::vector<int> order(32);
    for (int l = 0; l < 32; ++l) order[l] = trial & 1 ? l : 31 - l;
    if (trial % 3 == 2) std::shuffle(order.begin(), order.end(), rng);
    std::fill(g_buf, g_buf + 64, (uint16_t)0xeeee);
    if (gather(order) != want) {
      std::printf("trial %d: wrong indices\n", trial);
      return 1;
    }
  }
  std::puts("ok");
  return 0;
}
