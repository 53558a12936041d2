"""The verdict of a bounded wait (waits.cuh), compiled for the host: 32 lanes whose tries and clock readings
fall at times of their own wait for a phase that completes around the limit.  With the warp's vote
all lanes agree; each for itself they do not, for some completion times, which is what the vote is for."""
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "aero2d_b200" / "csrc"

PROGRAM = r"""
#include <barrier>
#include <cstdio>
#include <thread>
#include <vector>
#include "waits.cuh"

using u64 = unsigned long long;
constexpr int kLanes = 32;
constexpr u64 kStep = 20000000;   // ns between a lane's tries

struct Vote {   // __all_sync of the lanes
  std::barrier<> in{kLanes}, out{kLanes};
  bool flag[kLanes];
  bool all(int lane, bool b) {
    flag[lane] = b;
    in.arrive_and_wait();
    bool r = true;
    for (bool f : flag) r = r && f;
    out.arrive_and_wait();
    return r;
  }
};

// verdicts of the lanes for a phase that completes `complete` ns after their first try
int accepted(u64 complete, bool vote) {
  Vote v;
  bool got[kLanes];
  auto lane = [&](int l) {
    u64 now = (u64)l * (kStep / kLanes);   // this lane's own time
    auto done = [&] { now += kStep; return now >= complete; };
    auto clock = [&] { now += kStep / 7; return now; };
    if (vote) got[l] = a2d::bounded_wait(done, clock, [&](bool b) { return v.all(l, b); });
    else got[l] = a2d::bounded_wait(done, clock, [](bool b) { return b; });
  };
  if (vote) {
    std::vector<std::thread> t;
    for (int l = 0; l < kLanes; ++l) t.emplace_back(lane, l);
    for (auto& x : t) x.join();
  } else {
    for (int l = 0; l < kLanes; ++l) lane(l);
  }
  int n = 0;
  for (bool g : got) n += g;
  return n;
}

int main() {
  int split_vote = 0, split_lane = 0, yes = 0, no = 0;
  const u64 limit = a2d::kWaitLimitNs + (a2d::kWaitTries + 1) * kStep;
  for (u64 c = limit - 4 * kStep; c < limit + 8 * kStep; c += kStep / 8) {
    const int a = accepted(c, false);
    split_lane += a != 0 && a != kLanes;
  }
  for (u64 c = limit - 4 * kStep; c < limit + 8 * kStep; c += kStep / 2) {
    const int a = accepted(c, true);
    split_vote += a != 0 && a != kLanes;
    yes += a == kLanes;
    no += a == 0;
  }
  yes += accepted(0, true) == kLanes;
  std::printf("%d %d %d %d\n", split_vote, split_lane > 0, yes > 0, no > 0);
}
"""


def test_a_warp_has_one_verdict(tmp_path):
    src, exe = tmp_path / "w.cpp", tmp_path / "w"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-O2", "-std=c++20", "-pthread", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=120).stdout
    assert out.split() == ["0", "1", "1", "1"]
