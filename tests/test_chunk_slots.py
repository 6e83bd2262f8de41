"""The slots that lanes reserve a chunk at a time (chunk_slots.hpp), run on the host: every slot below
min(counter, capacity), which is what the kernels' readers take, is written once or marked empty, whatever the
capacity and wherever the counter stands."""
from __future__ import annotations

import subprocess

import pytest

from hpgbwt.build import CSRC

_MAIN = r"""
#include <cstdio>
#include <cstdlib>
#include <map>
#include <random>
#include <vector>
#include "chunk_slots.hpp"

using namespace hpgbwt;

// argv: lanes, entries, capacity, counter at the start
int main(int, char** argv) {
  const unsigned lanes = atoi(argv[1]), entries = atoi(argv[2]);
  const uint32_t cap = strtoul(argv[3], nullptr, 0), from = strtoul(argv[4], nullptr, 0);
  uint32_t counter = from;
  std::map<uint32_t, int> seen;  // of the slots from `from` on: times written or marked
  auto claim = [&](unsigned n) { const uint32_t c = counter; counter += n; return c; };
  auto note = [&](uint32_t s) {
    if (s < cap) ++seen[s];
  };
  std::vector<uint32_t> state(lanes, 0);
  std::mt19937 rng(7);
  unsigned refused = 0;
  for (unsigned i = 0; i < entries; ++i) {
    const uint32_t s = SLOT(cap, state[rng() % lanes], claim, note);
    if (s >= cap) ++refused;
    else note(s);
  }
  for (uint32_t w : state) chunk_leave(cap, w, note);
  const uint32_t end = counter < cap ? counter : cap;
  unsigned unwritten = 0, twice = 0, outside = 0;
  for (uint32_t s = from; s < end; ++s) unwritten += !seen.count(s);
  for (auto& kv : seen) {
    twice += kv.second > 1;
    outside += kv.first < from || kv.first >= end;
  }
  std::printf("%u %u %u %u\n", refused, unwritten, twice, outside);
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    d = tmp_path_factory.mktemp("chunk_slots")
    (d / "main.cpp").write_text(_MAIN)

    def build(slot: str):
        exe = d / slot
        if not exe.exists():
            subprocess.run(["g++", "-O1", "-std=c++17", f"-I{CSRC}", f"-DSLOT={slot}", str(d / "main.cpp"),
                            "-o", str(exe)], check=True)

        def call(*args) -> list[int]:
            return [int(x) for x in subprocess.run([str(exe), *map(str, args)], capture_output=True, text=True,
                                                   check=True).stdout.split()]
        return call
    return build


@pytest.mark.parametrize("cap", [1, 7, 8, 9, 100, 1004, 1005, 1008, 1011, (1 << 28) - 1])
@pytest.mark.parametrize("entries", [0, 5, 900, 5000])
def test_bounded_queue_leaves_no_slot_unwritten(run, cap, entries):
    call = run("chunk_slot")
    for from_ in {0, max(0, cap - 40), max(0, cap - 3)}:
        refused, unwritten, twice, outside = call(13, entries, cap, from_)
        assert (unwritten, twice, outside) == (0, 0, 0)
        if entries > cap - from_:
            assert refused


@pytest.mark.parametrize("cap", [1, 100, 1005, (1 << 28) - 5, 1 << 28, (1 << 28) + 777, (1 << 32) - 17])
@pytest.mark.parametrize("from_", [0, 3, (1 << 28) - 2000, (1 << 28) - 8, (1 << 28) - 3, 1 << 28, (1 << 31) + 5])
def test_pool_leaves_no_slot_unwritten(run, cap, from_):
    """Past 2^28, what a state's word holds, a lane takes one slot a claim."""
    for lanes, entries in ((1, 9), (13, 3000), (300, 5000)):
        refused, unwritten, twice, outside = run("pool_slot")(lanes, entries, cap, from_)
        assert (unwritten, twice, outside) == (0, 0, 0)
        if cap > from_ + 8 * (entries + lanes):
            assert refused == 0
