// How the state scans (k_state_scan_ps) are spread over the SMs: the host rule, and the order in which a block walks its
// chunks.  No CUDA in here beyond the function qualifiers, so that a host program can go through both.
#pragma once

#ifdef __CUDACC__
#define SSD_HD __host__ __device__ __forceinline__
#else
#define SSD_HD inline
#endif

namespace ssd {

// A unit is the sequence of one batch row for 128 (h,p) rows of a group.  Whichever way is taken, every element goes through the
// same operations in the same order, chunk after chunk: a row's bits depend neither on how many rows a call has nor on how far
// its sequence goes on.
enum class StatePlan {
  walks,    // a block walks whole units
  shares,   // every block gets the same number of chunks; a unit cut between two is handed over
  split     // products and scan as two kernels, the fp32 states of all chunks in memory between them
};

// The one rule; `n` = dstate.  State kernels of a forward and a backward pass, us on 148 SMs, sequences of 64 chunks:
//                  24 heads of 64 x 128 (12 units a row)       8 heads of 32 x 64 (2 units a row)
//   units           12    24    48    60    72    96            8    32    64    74    84    96
//   walks          339   341   340   340   335   342          271   277   277   277   279   280
//   split           96   142   253   336   373   490           67   125   229   257   279   299
// A walk takes the time of one unit's chunks behind one another, the two kernels the time of the states they move: the lines cross
// near 60 and 84 units, at 8 to 128 chunks alike (bounds: 2/5 and 1/2 of the SMs).  Below 8 chunks the second launch weighs more, and
// they cross near 50 (2 chunks, 48 units of 24 heads: 37 against 44 us, but whole passes 92.2 against 91.1; 1/3); a single chunk has
// nothing to walk.  The longest sequences stay with it (1024 chunks, 24 units: 2030 against 4870).
// Whole forwards since the products of k_state_ps got faster, walks and split: 64 chunks, 24 heads, 48, 60, 72 units 226, 248, 264 and
// 198, 260, 300 us; 8 heads, 64, 74, 84 units 259, 279, 303 and 234, 266, 322; 16 chunks, 60 and 72 units 75, 78 and 74, 79.
// More units than SMs: even shares where they save more than a twentieth (192 units of 32 chunks: 413 -> 311; a hand-over costs a
// state's write and read per block); a share has to be longer than a unit, so that a unit is cut at most once.
inline StatePlan state_plan(int nc, int units, int n, int sms) {
  if (units > sms) {
    const int rounds = (units + sms - 1) / sms;
    return rounds * sms > units + units / 20 && (long long)units * nc / sms > nc ? StatePlan::shares : StatePlan::walks;
  }
  const int per6 = nc < 8 ? 18 : n > 64 ? 15 : 12;   // a third, two fifths, a half of the SMs
  return nc > 1 && units * per6 <= 6 * sms ? StatePlan::split : StatePlan::walks;
}

// A block's tiles in order: the chunks of a unit in scan order, unit after unit; neighbouring units share a B/C tile.  BAL (even
// shares): the unit cut at the end of the share first, then the whole units, then the rest of the unit that the block before
// cut.  G has B, G, hpg and nc.  (Few members: the consumers hold a walk beside the running state.)
template <int P, bool BAL>
struct StateWalk {
  int u, b, h0, grp, s, s0, s1;
  template <class G>
  SSD_HD StateWalk(const G& g, int nunits, int block, int grid) {
    if constexpr (BAL) {
      const long long a1 = (long long)(block + 1) * nunits * g.nc / grid;
      u = (int)(a1 / g.nc);
      piece(g, 0, (int)(a1 - (long long)u * g.nc));
      if (s == s1) next_unit(g, nunits, block, grid);
    } else {
      u = block;
      piece(g, 0, g.nc);
    }
  }
  template <class G>
  SSD_HD void piece(const G& g, int from, int to) {
    const int MT = g.hpg * P / 128, r = u / MT;
    grp = r % g.G;
    b = r / g.G;
    h0 = grp * g.hpg + (u - r * MT) * (128 / P);
    s = s0 = from;
    s1 = to;
  }
  template <class G>
  SSD_HD void next_unit(const G& g, int nunits, int block, int grid) {
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
      piece(g, 0, g.nc);
    }
  }
  template <class G>
  SSD_HD void next(const G& g, int nunits, int block, int grid) {
    if (++s == s1) next_unit(g, nunits, block, grid);
  }
  // tiles of a block
  template <class G>
  static SSD_HD int total(const G& g, int nunits, int block, int grid) {
    const long long T = (long long)nunits * g.nc;
    if constexpr (BAL) return (int)((block + 1) * T / grid - block * T / grid);
    else return (nunits - block + grid - 1) / grid * g.nc;
  }
};

}  // namespace ssd
