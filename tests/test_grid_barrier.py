"""The barrier of a cooperative grid (csrc/gridbar.cuh) compiled for the host, threads in place of CTAs: with waits
that run out at any moment, the threads of a launch agree on whether its last barrier was passed."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent

PROGRAM = r"""
#include <atomic>
#include <cstdio>
#include <random>
#include <thread>
#include <vector>
#include "gridbar.cuh"

struct Word {
  std::atomic<unsigned>* at;
  std::mt19937 rng;
  void idle() { if (rng() % 3 == 0) std::this_thread::yield(); }
  unsigned add(unsigned v) { idle(); return at->fetch_add(v); }
  unsigned load() { idle(); return at->load(); }
  bool swap(unsigned was, unsigned to) { idle(); return at->compare_exchange_strong(was, to); }
  void pause(int) { idle(); }
};

int main() {
  int passed = 0, gave_up = 0;
  for (int trial = 0; trial < 4000; ++trial) {
    const int ctas = 2 + trial % 4, barriers = 1 + trial % 3;
    const int turns = trial % 2 ? 1 + trial % 9 : 1 << 20;  // every other launch runs out of turns easily
    std::atomic<unsigned> word{0};
    std::vector<int> through(ctas, 0);
    std::vector<std::thread> t;
    for (int c = 0; c < ctas; ++c)
      t.emplace_back([&, c] {
        Word w{&word, std::mt19937(trial * 16 + c)};
        for (int b = 1; b <= barriers; ++b) {
          if (w.rng() % 4 == 0) for (int k = w.rng() % 20; k > 0; --k) std::this_thread::yield();
          if (!hb::grid_barrier(w, b * ctas, turns)) return;
        }
        through[c] = 1;
      });
    for (auto& x : t) x.join();
    for (int c = 1; c < ctas; ++c)
      if (through[c] != through[0]) return std::printf("trial %d: the threads disagree\n", trial), 1;
    if (turns > 1000 && !through[0]) return std::printf("trial %d: gave up\n", trial), 1;
    (through[0] ? passed : gave_up) += 1;
  }
  std::printf("%d %d\n", passed, gave_up);
  return passed > 100 && gave_up > 100 ? 0 : 1;
}
"""


def test_the_ctas_agree_on_the_last_barrier(tmp_path):
    (tmp_path / "bar.cpp").write_text(PROGRAM)
    exe = tmp_path / "bar"
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I", str(ROOT / "hades_b200" / "csrc"),
                    str(tmp_path / "bar.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
