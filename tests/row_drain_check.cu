// Host check of the row tiles' give-up protocol (rows_drain in
// gpu-sims_b200/csrc/phys_rows.cuh).  Service warps, the collision and the copies
// of a block advance in random order and stop at random tiles, as after a wait
// that ran out; then every warp must see all loads of the block land, through
// waits that end, whatever the warps had begun.  Runs on the CPU.
#include <algorithm>
#include <cstdio>
#include <random>
#include <vector>

#include "../gpu-sims_b200/csrc/phys_rows.cuh"

using namespace lbm;

struct Barrier {  // phase number, arrivals still to come and bytes in flight of the current phase
  uint32_t phase = 0, pending, count, bytes = 0;
  void settle() {
    if (!pending && !bytes) {
      ++phase;
      pending = count;
    }
  }
};

int main() {
  std::mt19937 r(11);
  auto pick = [&](uint32_t n) { return (uint32_t)(r() % n); };
  constexpr uint32_t W = ROWS_SERV;
  long bad = 0, uneven = 0;
  for (int trial = 0; trial < 200000; ++trial) {
    const uint32_t stages = trial & 1 ? 2 : 5, tiles = 1 + pick(14), stop = 1 + pick(120);
    std::vector<Barrier> full(stages), done(stages);
    for (auto& b : full) b.pending = b.count = W;  // a warp's 33 arrivals as one
    for (auto& b : done) b.pending = b.count = 1;
    uint32_t loaded[W] = {}, at[W] = {}, consumed = 0;
    std::vector<std::pair<uint32_t, uint32_t>> copies;  // stage, warp: issued, not landed
    auto load = [&](uint32_t w) {
      const uint32_t s = loaded[w]++ % stages;
      --full[s].pending;
      ++full[s].bytes;
      copies.push_back({s, w});
    };
    auto land = [&] {
      const uint32_t k = pick((uint32_t)copies.size());
      --full[copies[k].first].bytes;
      full[copies[k].first].settle();
      copies.erase(copies.begin() + k);
    };
    auto passed = [](const Barrier& b, uint32_t parity) { return (b.phase & 1u) != parity; };
    for (uint32_t w = 0; w < W; ++w)
      if (pick(8))  // a warp may be stopped before its first loads
        while (loaded[w] < std::min(stages, tiles)) load(w);
    for (uint32_t step = 0; step < stop; ++step) {
      const uint32_t what = pick(W + 2);
      if (what < W) {  // a service warp's tile: its store, then the refill of rows_service
        uint32_t& j = at[what];
        if (loaded[what] < std::min(stages, tiles)) {
          load(what);
          continue;
        }
        if (j < tiles && passed(done[j % stages], j / stages & 1)) {
          if ((j > 0 || stages <= 2) && loaded[what] < tiles) load(what);
          ++j;
        }
      } else if (what == W) {  // the collision
        if (consumed < tiles && passed(full[consumed % stages], consumed / stages & 1)) {
          --done[consumed % stages].pending;
          done[consumed % stages].settle();
          ++consumed;
        }
      } else if (!copies.empty()) {
        land();
      }
    }
    // all give up here
    const uint32_t most = *std::max_element(loaded, loaded + W);
    uneven += *std::min_element(loaded, loaded + W) != most;
    uint32_t order[W] = {0, 1, 2, 3};
    std::shuffle(order, order + W, r);
    std::vector<std::pair<uint32_t, uint32_t>> waits[W];
    for (uint32_t w : order)
      rows_drain(
          loaded[w], most, stages,
          [&](uint32_t s) {
            bad += full[s].pending == 0;  // an arrival too many for the phase
            --full[s].pending;
            full[s].settle();
          },
          [&](uint32_t s, uint32_t parity) { waits[w].push_back({s, parity}); });
    for (uint32_t w = 0; w < W; ++w)  // no wait passes while one of its loads is in flight
      for (auto& c : copies)
        if (c.second == w) {
          bool held = false;
          for (auto& q : waits[w]) held = held || (q.first == c.first && !passed(full[q.first], q.second));
          bad += !held;
        }
    while (!copies.empty()) land();
    for (uint32_t w = 0; w < W; ++w)  // ... and with all landed, all pass
      for (auto& q : waits[w]) bad += !passed(full[q.first], q.second);
  }
  std::printf("%ld stops at uneven tiles, %ld errors\n", uneven, bad);
  return bad != 0 || uneven < 1000;
}
