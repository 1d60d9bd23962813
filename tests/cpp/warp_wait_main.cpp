// 32 threads as a warp's lanes: waits whose looks answer differently from lane to
// lane, each followed by a collective of its own (as the sweeps' shuffles follow
// their waits).  A collective that lanes enter from different places is a fault.
#include <condition_variable>
#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <thread>
#include <vector>

#include "../../xfluid_b200/csrc/xfp_warp_wait.h"

struct Warp {
  std::mutex m;
  std::condition_variable cv;
  int arrived = 0, place = 0;
  long turn = 0;
  bool value = true, result = false;
  bool all(int where, bool v) {
    std::unique_lock<std::mutex> lock(m);
    if (arrived == 0) {
      place = where;
      value = true;
    } else if (where != place) {
      std::fprintf(stderr, "lanes at %d and %d in one collective\n", place, where);
      std::_Exit(1);
    }
    value = value && v;
    const long mine = turn;
    if (++arrived == 32) {
      arrived = 0;
      result = value;
      ++turn;
      cv.notify_all();
    } else {
      cv.wait(lock, [&] { return turn != mine; });
    }
    return result;
  }
};

int main() {
  Warp w;
  std::vector<int> gave_up(32, 0);
  auto lane = [&](int id) {
    unsigned rng = 12345u + 977u * (unsigned)id;
    for (int round = 0; round < 300; ++round) {
      // lane `id` sees the phase complete from its look number `first` on; one lane
      // in some rounds never does, or is the only one that loses patience
      rng = rng * 1664525u + 1013904223u;
      const int first = (int)(rng >> 28);
      const bool never = round % 7 == 3 && id == round % 32;
      const int patience = round % 7 == 3 ? (id == (round + 5) % 32 ? 4 : 1000) : 1000;
      int looks = 0, turns = 0;
      const bool ok = xfp::warp_wait([&] { return !never && looks++ >= first; },
                                     [&](bool v) { return w.all(2 * round, v); },
                                     [&] { return ++turns < patience; });
      if (!ok) ++gave_up[id];
      if (ok != (round % 7 != 3)) std::_Exit(2);
      w.all(2 * round + 1, true);   // the step's shuffle
    }
  };
  std::vector<std::thread> lanes;
  for (int id = 0; id < 32; ++id) lanes.emplace_back(lane, id);
  for (auto& t : lanes) t.join();
  for (int id = 1; id < 32; ++id)
    if (gave_up[id] != gave_up[0]) return 3;
  std::printf("ok\n");
  return 0;
}
