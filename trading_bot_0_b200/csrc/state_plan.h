// How the state scans (k_state_scan_ps) are spread over the SMs: the host rule, and the order in which a block walks its
// chunks.  No CUDA in here beyond the function qualifiers, so that a host program can go through both.
#pragma once

#ifdef __CUDACC__
#define SSD_HD __host__ __device__ __forceinline__
#else
#define SSD_HD inline
#endif

namespace ssd {

// A unit is the sequence of one batch row for 128 (h,p) rows of a group.
struct StatePlan {
  int nseg, seglen;   // segments that the sequence is cut into, chunks in each (the last may be shorter)
  bool shares;        // every block gets the same number of chunks (only with one segment)
};

// The one rule for both.  More units than SMs: one segment, and even shares where they save more than a twentieth (a hand-over
// costs a state's write and read per block); a share has to be longer than a unit, so that a unit is cut at most once.
// Fewer units: segments.  A launch takes (units per block, rounded up) x (chunks of a segment) steps; cutting costs a second
// launch over all segments but the last, whose steps are 0.7 of the others' (nothing is written), the launch itself (about
// three steps) and a fold per segment.  Fewer than 16 chunks: one segment, the second launch would cost what it saves.
inline StatePlan state_plan(int nc, int units, int sms) {
  auto up = [](int a, int b) { return (a + b - 1) / b; };
  StatePlan p{1, nc, false};
  if (units > sms) {
    p.shares = up(units, sms) * sms > units + units / 20 && (long long)units * nc / sms > nc;
    return p;
  }
  if (nc < 16) return p;
  double least = 1e30;
  for (int n = 1; n <= nc / 2; ++n) {
    const int len = up(nc, n), seg = up(nc, len);
    const double t = (double)up(units * seg, sms) * len + (seg > 1 ? 0.7 * up(units * (seg - 1), sms) * len + 3 + 0.3 * seg : 0.);
    if (t < least) { least = t; p.nseg = seg; p.seglen = len; }
    if ((long long)units * n > 4LL * sms) break;
  }
  return p;
}

// A block's tiles in order: the chunks of a unit (or of a segment of one) in scan order, unit after unit; neighbouring units
// share a B/C tile.  BAL (even shares): the unit cut at the end of the share first, then the whole units, then the rest of the
// unit that the block before cut.  `nunits` counts segments; G has B, G, hpg and nc.  (Few members: the consumers hold a walk
// beside the running state.)
template <int P, bool BAL>
struct StateWalk {
  int u, b, h0, grp, seg, s, s0, s1;
  template <class G>
  SSD_HD StateWalk(const G& g, int seglen, int nunits, int block, int grid) {
    if constexpr (BAL) {
      const long long a1 = (long long)(block + 1) * nunits * g.nc / grid;
      u = (int)(a1 / g.nc);
      piece(g, 0, (int)(a1 - (long long)u * g.nc));
      if (s == s1) next_unit(g, seglen, nunits, block, grid);
    } else {
      u = block;
      place(g, seglen);
    }
  }
  template <class G>
  SSD_HD void place(const G& g, int seglen) {
    const int MT = g.hpg * P / 128;
    int r = u / MT;
    h0 = (u - r * MT) * (128 / P);
    grp = r % g.G; r /= g.G;
    h0 += grp * g.hpg;
    b = r % g.B;
    seg = BAL ? 0 : r / g.B;
    s = s0 = seg * seglen;
    s1 = s + seglen < g.nc ? s + seglen : g.nc;
  }
  template <class G>
  SSD_HD void piece(const G& g, int from, int to) {
    place(g, g.nc);
    s = s0 = from;
    s1 = to;
  }
  template <class G>
  SSD_HD void next_unit(const G& g, int seglen, int nunits, int block, int grid) {
    if constexpr (BAL) {
      const long long T = (long long)nunits * g.nc, a0 = block * T / grid, a1 = (block + 1) * T / grid;
      const int first = (int)(a0 / g.nc), off = (int)(a0 - (long long)first * g.nc), last = (int)(a1 / g.nc);
      u = u == last ? first + (off > 0) : u + 1;
      if (u < last) {
        piece(g, 0, g.nc);
      } else {
        u = first;
        piece(g, off, g.nc);
      }
    } else {
      u += grid;
      place(g, seglen);
    }
  }
  template <class G>
  SSD_HD void next(const G& g, int seglen, int nunits, int block, int grid) {
    if (++s == s1) next_unit(g, seglen, nunits, block, grid);
  }
  // tiles of a block; `segs` = segments of a unit among the `nunits`
  template <class G>
  static SSD_HD int total(const G& g, int seglen, int nunits, int segs, int block, int grid) {
    if constexpr (BAL) {
      const long long T = (long long)nunits * g.nc;
      return (int)((block + 1) * T / grid - block * T / grid);
    } else {
      int n = 0;
      for (int u = block; u < nunits; u += grid) {
        const int s0 = u / (nunits / segs) * seglen;
        n += seglen < g.nc - s0 ? seglen : g.nc - s0;
      }
      return n;
    }
  }
};

}  // namespace ssd
