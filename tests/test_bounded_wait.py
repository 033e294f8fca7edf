"""Waits that run out (csrc/bounded_wait.h), compiled for the host: a block of warps that wait on copies which never land."""
import os
import subprocess

from serve_b200.kernels.build import CSRC

PROGRAM = r"""
#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <thread>
#include <vector>
#include "bounded_wait.h"

std::atomic<int> flag, counted, read, landed;           // a block's flag; the host's count; chunks read; copies landed so far
struct Notes {
  bool raise() { return flag.exchange(1) == 0; }
  bool raised() const { return flag.load() != 0; }
  void count() { ++counted; }
};

// The walk of ``chunks`` chunks through two stages, as chunked_recurrence.cu has it: one thread fetches, the other reads, and copies from
// number ``lost`` on never land; those from ``late`` on land only once the fetching thread has asked for them many times.
int main(int argc, char** argv) {
  const int chunks = atoi(argv[1]), lost = atoi(argv[2]), late = atoi(argv[3]);
  const unsigned LIMIT = 500000;
  flag = counted = read = landed = 0;
  std::atomic<int> issued(0), stored(0), left_with(0), asked(0);
  auto full = [&](int c) { std::this_thread::yield(); return landed.load() > c; };
  auto land = [&](int c) { if (c < lost && c < late) landed = c + 1; };
  std::thread fetching([&] {
    Notes notes;
    int c = 0;
    for (; c < chunks; ++c) {
      sb::wait_in_step([&] { std::this_thread::yield(); return c < 2 || read.load() >= c - 1; }, notes, LIMIT);
      if (notes.raised()) break;
      issued = c + 1;
      land(c);
    }
    for (int i = std::max(0, c - 2); i < c; ++i)
      sb::wait_landed([&] { if (++asked > 5000 && i < lost) landed = std::max(landed.load(), i + 1); return full(i); }, notes, LIMIT);
    left_with = issued.load() - landed.load();          // copies still under way when the thread that asked for them leaves
  });
  std::thread reading([&] {
    Notes notes;
    for (int c = 0; c < chunks; ++c) {
      sb::wait_in_step([&] { return full(c); }, notes, LIMIT);
      read = c + 1;
    }
    if (!notes.raised()) stored = 1;
  });
  fetching.join();
  reading.join();
  printf("%d %d %d\n", counted.load(), stored.load(), left_with.load());
}
"""


def _walk(tmp_path, chunks, lost, late):
    exe = os.path.join(tmp_path, "walk")
    if not os.path.isfile(exe):
        source = os.path.join(tmp_path, "walk.cc")
        with open(source, "w") as f:
            f.write(PROGRAM)
        subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, "-o", exe, source], check=True)
    out = subprocess.run([exe, str(chunks), str(lost), str(late)], check=True, capture_output=True, text=True, timeout=60)
    return tuple(int(x) for x in out.stdout.split())


def test_a_copy_that_never_lands_is_reported(tmp_path):
    """Counted once, whichever chunk it is (after the last copy has been asked for too), and the state is not stored."""
    for chunks in (1, 2, 3, 7):
        assert _walk(tmp_path, chunks, chunks, chunks) == (0, 1, 0)
        for lost in range(chunks):
            counted, stored, _ = _walk(tmp_path, chunks, lost, chunks)
            assert (counted, stored) == (1, 0), (chunks, lost)


def test_copies_under_way_land_before_the_block_leaves(tmp_path):
    for chunks in (1, 2, 5):
        assert _walk(tmp_path, chunks, chunks, chunks - 1)[2] == 0
