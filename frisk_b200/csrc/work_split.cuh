// How work is dealt to CTAs, and which tickets a CTA owes.  Plain arithmetic, for the host as well.
//
// WorkSplit: units, numbered group after group (a group: the key tiles of a head), in contiguous ranges.
// TileWalk: output tiles, whole ones round by round and the rest to clusters that share each one's K.
//
// What several CTAs work on has a ticket, zero between launches: each contributor draws it EXACTLY ONCE, whatever
// happens to the CTA in between (draw_owed), and the last draw puts it back to zero.
#pragma once
#ifdef __CUDACC__
#define FB_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define FB_HOST_DEVICE inline
#endif

namespace fb {

struct WorkSplit {
  unsigned q, r;  // units = CTAs * q + r: the first r CTAs take q + 1
  FB_HOST_DEVICE unsigned start(unsigned c) const { return c * q + (c < r ? c : r); }
  FB_HOST_DEVICE unsigned worker_of(unsigned u) const {
    const unsigned big = r * (q + 1);
    return u < big ? u / (q + 1) : r + (u - big) / q;
  }
  // the other contributors of a group of `size` units that begins at unit u0 (0: its one CTA draws no ticket)
  FB_HOST_DEVICE unsigned partners(unsigned u0, unsigned size) const { return worker_of(u0 + size - 1) - worker_of(u0); }
  // draw(group, partners) for every group that units [u, end) of one CTA belong to and that it shares
  template <typename Draw>
  FB_HOST_DEVICE void draw_owed(unsigned u, unsigned end, unsigned size, Draw&& draw) const {
    while (u < end) {
      const unsigned group = u / size, n = partners(group * size, size);
      if (n > 0) draw(group, n);
      const unsigned left = size - u % size;  // units of the group from u on
      if (left >= end - u) break;
      u += left;
    }
  }
};

struct TileItem {
  int tile, kb0, kb1;  // 64-k blocks [kb0, kb1) of the tile
  bool shared;         // the other blocks are the cluster's other CTAs'
};

struct TileWalk {
  int tiles, num_kb;          // in all; 64-k blocks of a tile
  int n_whole, splits, grid;  // tiles [0, n_whole) are walked whole; a cluster of `splits` CTAs shares each of the others
  // item i of CTA `cta`, which has `rank` in its cluster: its whole tiles, then its part of one shared tile
  FB_HOST_DEVICE bool get(int cta, int rank, int i, TileItem& it) const {
    const int whole = cta + i * grid;
    if (whole < n_whole) {
      it = TileItem{whole, 0, num_kb, false};
      return true;
    }
    const int n_mine = cta < n_whole ? (n_whole - 1 - cta) / grid + 1 : 0;
    const int tile = n_whole + cta / splits;
    if (i > n_mine || splits == 1 || tile >= tiles) return false;
    it = TileItem{tile, (int)((long long)num_kb * rank / splits), (int)((long long)num_kb * (rank + 1) / splits), true};
    return true;
  }
  // draw(tile) for the tiles from item i on whose tickets this CTA draws: all of its own, and rank 0 the cluster's
  template <typename Draw>
  FB_HOST_DEVICE void draw_owed(int cta, int rank, int i, Draw&& draw) const {
    TileItem it;
    for (; get(cta, rank, i, it); ++i)
      if (!it.shared || rank == 0) draw(it.tile);
  }
};

}  // namespace fb
