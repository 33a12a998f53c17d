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
  // tiles: whole rounds, then clusters that share the K of the rest
  for (int round = 0; round < 20000; ++round) {
    const int splits = 1 << pick(0, 3), sms = 148, kb = (int)pick(2 * splits, 64), tiles_n = (int)pick(1, 30);
    const int tiles = tiles_n * (int)pick(1, 30), full = sms / splits * splits;
    int grid, n_whole;
    if (splits == 1) {
      grid = tiles < sms ? tiles : sms;
      n_whole = tiles;
    } else {
      const int rest = tiles % full;
      if (rest == 0 || rest > full / splits) continue;
      n_whole = tiles - rest;
      grid = n_whole > 0 ? full : rest * splits;
    }
    const fb::TileWalk w{tiles, kb, n_whole, splits, grid};
    std::vector<int> blocks(tiles, 0);
    std::vector<unsigned> ticket(tiles / tiles_n, 0), merged(tiles / tiles_n, 0);
    auto draw = [&](int tile) {
      const bool last = ticket[tile / tiles_n]++ == (unsigned)tiles_n - 1;
      if (last) { ticket[tile / tiles_n] = 0; ++merged[tile / tiles_n]; }
    };
    const bool stops = round % 2;
    for (int c = 0; c < grid; ++c) {
      fb::TileItem it;
      int drawn = 0, i = 0;
      bool stopped = false;
      for (; w.get(c, c % splits, i, it); ++i) {
        blocks[it.tile] += it.kb1 - it.kb0;
        if (it.kb0 >= it.kb1 || it.kb1 > kb || (it.shared && (splits == 1 || w.get(c, c % splits, i + 1, it)))) return 7;
        if (stops && rng() % 4 == 0) stopped = true;
        if (stopped) continue;
        if (!it.shared || c % splits == 0) draw(it.tile);
        ++drawn;
      }
      w.draw_owed(c, c % splits, drawn, draw);
    }
    for (int t = 0; t < tiles; ++t)
      if (blocks[t] != kb) return 8;
    for (size_t m = 0; m < ticket.size(); ++m)
      if (ticket[m] != 0 || merged[m] != 1) return 9;
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
