// How work is dealt to CTAs, and which tickets a CTA owes.  Plain arithmetic, for the host as well.
//
// WorkSplit: units, numbered group after group (a group: the key tiles of a head), in contiguous ranges.
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

}  // namespace fb
