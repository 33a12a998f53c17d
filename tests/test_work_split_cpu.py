"""The tickets of groups that several CTAs share (csrc/work_split.cuh) are back at zero after every launch, also when CTAs stop
early: compiled for the host, over many splits and stopping points."""
import pathlib
import shutil
import subprocess

import pytest

CSRC = pathlib.Path(__file__).resolve().parent.parent / "frisk_b200" / "csrc"

PROGRAM = r"""
#include <cstdio>
#include <random>
#include <vector>
#include "work_split.cuh"

int main() {
  std::mt19937 rng(7);
  auto pick = [&](unsigned lo, unsigned hi) { return lo + rng() % (hi - lo + 1); };
  for (int round = 0; round < 20000; ++round) {
    const unsigned groups = pick(1, 40), size = pick(1, 70), units = groups * size;
    const unsigned ctas = units < 148 ? pick(1, units) : pick(1, 148);
    const fb::WorkSplit w{units / ctas, units % ctas};
    std::vector<unsigned> ticket(groups, 0), draws(groups, 0), merged(groups, 0);
    std::vector<unsigned> from(groups, ctas), to(groups, 0);
    auto draw = [&](unsigned g, unsigned partners) {
      ++draws[g];
      const bool last = ticket[g]++ == partners;
      if (last) { ticket[g] = 0; ++merged[g]; }
    };
    const bool stops = round % 2;
    if (w.start(0) != 0 || w.start(ctas) != units) return 1;
    for (unsigned c = 0; c < ctas; ++c) {
      const unsigned begin = w.start(c), end = w.start(c + 1);
      if (begin >= end) return 2;
      for (unsigned u = begin; u < end; ++u) {
        if (w.worker_of(u) != c) return 3;
        const unsigned g = u / size;
        if (c < from[g]) from[g] = c;
        if (c > to[g]) to[g] = c;
      }
      // group by group, as far as the CTA gets; then what it owes
      unsigned u = begin;
      while (u < end && !(stops && rng() % 4 == 0)) {
        const unsigned g = u / size, left = size - u % size, n = w.partners(g * size, size);
        if (n > 0) draw(g, n);
        u += left < end - u ? left : end - u;
      }
      w.draw_owed(u, end, size, draw);
    }
    for (unsigned g = 0; g < groups; ++g) {
      const unsigned contributors = to[g] - from[g] + 1;
      if (ticket[g] != 0) return 4;
      if (draws[g] != (contributors > 1 ? contributors : 0)) return 5;
      if (merged[g] != (contributors > 1 ? 1u : 0u)) return 6;
    }
  }
  puts("ok");
  return 0;
}
"""


def test_every_ticket_is_drawn_exactly_once_by_each_contributor(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    src, exe = tmp_path / "split.cpp", tmp_path / "split"
    src.write_text(PROGRAM)
    subprocess.run([gxx, "-std=c++17", "-O1", "-Wall", "-Werror", "-I", str(CSRC), "-o", str(exe), str(src)], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True)
    assert res.returncode == 0 and res.stdout.strip() == "ok", res.returncode
