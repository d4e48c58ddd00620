"""The softmax warps' loop (csrc/block_loop.h) with threads in the place of warps: whichever wait runs out, every warp has
to come to every barrier, or the others wait there without end."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "multimodal_training_b200" / "csrc"

PROGRAM = r"""
#include <chrono>
#include <condition_variable>
#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <thread>
#include <vector>
#include "block_loop.h"

// A barrier that reports instead of waiting for ever.
struct Barrier {
  std::mutex m;
  std::condition_variable cv;
  int n, here = 0, round = 0;
  bool stuck = false;
  explicit Barrier(int n) : n(n) {}
  void operator()() {
    std::unique_lock<std::mutex> l(m);
    const int mine = round;
    if (++here == n) {
      here = 0;
      ++round;
      cv.notify_all();
      return;
    }
    if (!cv.wait_for(l, std::chrono::seconds(5), [&] { return round != mine || stuck; }) || stuck) {
      stuck = true;
      cv.notify_all();
    }
  }
};

int main(int argc, char** argv) {
  const int warps = 4, blocks = atoi(argv[1]), bad_warp = atoi(argv[2]), bad_block = atoi(argv[3]);
  Barrier bar(warps);
  std::vector<int> worked(warps, 0), result(warps, -1);
  std::vector<std::thread> t;
  for (int w = 0; w < warps; ++w)
    t.emplace_back([&, w] {
      // the products of a block are published only when every warp has worked on the block before
      auto wait = [&](int it) { return bad_block < 0 || (it <= bad_block && !(w == bad_warp && it == bad_block)); };
      result[w] = attn::for_blocks_in_step(blocks, wait, [&](int) { bar(); ++worked[w]; }, [&] { bar(); });
    });
  for (auto& x : t) x.join();
  for (int w = 0; w < warps; ++w) printf("%d %d ", worked[w], result[w]);
  printf("%d %d\n", bar.round, (int)bar.stuck);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("block_loop")
    (d / "main.cpp").write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-O1", "-pthread", "-I", str(CSRC), str(d / "main.cpp"), "-o", str(d / "main")],
                   check=True)
    return d / "main"


@pytest.mark.parametrize("blocks,warp,block", [(0, 0, -1), (1, 0, -1), (7, 0, -1), (1, 2, 0), (7, 0, 0), (7, 3, 4), (7, 1, 6)])
def test_every_warp_comes_to_every_barrier(program, blocks, warp, block):
    out = [int(v) for v in subprocess.run([str(program), str(blocks), str(warp), str(block)], capture_output=True,
                                          text=True, timeout=60, check=True).stdout.split()]
    worked, result, (rounds, stuck) = out[0:8:2], out[1:8:2], out[8:]
    assert not stuck and rounds == blocks
    for w in range(4):
        if block < 0:
            assert worked[w] == blocks and result[w] == 1
        else:
            assert worked[w] == (block if w == warp else min(block + 1, blocks))
            assert result[w] == int(w != warp and block + 1 >= blocks)
