// Host check of how the state scans are spread over the SMs (csrc/state_plan.h): the rule over a range of sizes, and the walks
// of all blocks of a launch replayed for a part of them.  Exit code 0 when everything holds, else 1 and the first failure.
#include <cstdio>
#include <vector>

#include "../../trading_bot_0_b200/csrc/state_plan.h"

using namespace ssd;

struct G { int B, G, hpg, nc; };

#define REQUIRE(c)                                                                                              \
  do {                                                                                                          \
    if (!(c)) {                                                                                                 \
      std::printf("%s: units %d chunks %d sms %d, plan %d\n", #c, units, nc, sms, (int)p);                      \
      return false;                                                                                             \
    }                                                                                                           \
  } while (0)

static bool check_rule(int units, int nc, int sms, StatePlan p) {
  REQUIRE(p != StatePlan::shares || (units > sms && (long long)units * nc / sms > nc));   // a unit is cut at most once
  REQUIRE(p != StatePlan::split || (units < sms && nc > 1));
  return true;
}

// All blocks of one launch: every (unit, chunk) once and in order, the hand-over slots inside their array and used by
// neighbouring blocks only (published by the one before as its first piece), the end of every unit reached once.
template <int P, bool BAL>
static bool check_walk(const G& g, int sms, StatePlan p) {
  const int MT = g.hpg * P / 128, units = g.B * g.G * MT, nc = g.nc, hand_len = g.B * g.G * g.hpg * P / 128;
  const int grid = BAL || units > sms ? sms : units;
  std::vector<char> seen((size_t)units * nc, 0);
  std::vector<int> published(units, -1), cut(units, 0), ends(units, 0);
  long long all = 0;
  for (int blk = 0; blk < grid; ++blk) {
    using Walk = StateWalk<P, BAL>;
    const int total = Walk::total(g, units, blk, grid);
    Walk t(g, units, blk, grid);
    int pieces = 0, su = -1, ss = -1;
    all += total;
    for (int k = 0; k < total; ++k, t.next(g, units, blk, grid)) {
      REQUIRE(t.u >= 0 && t.u < hand_len);
      REQUIRE(t.b >= 0 && t.b < g.B && t.grp >= 0 && t.grp < g.G && t.h0 >= 0 && t.h0 + 128 / P <= g.G * g.hpg);
      REQUIRE(t.s >= t.s0 && t.s < t.s1 && t.s1 <= nc);
      REQUIRE((t.b * g.G + t.grp) * MT + (t.h0 - t.grp * g.hpg) * P / 128 == t.u);
      if (t.s == t.s0) {
        ++pieces;
        REQUIRE(BAL || t.s0 == 0);
        if (t.s0 > 0) {   // taken over, by the last piece of the block behind the one that published it
          REQUIRE(published[t.u] == blk - 1 && cut[t.u] == t.s0 && t.s1 == nc);
          REQUIRE(k + (t.s1 - t.s0) == total);
        }
      } else {
        REQUIRE(su == t.u && ss == t.s - 1);
      }
      char& c = seen[(size_t)t.u * nc + t.s];
      REQUIRE(!c);
      c = 1;
      if (t.s + 1 == t.s1) {
        if (t.s1 < nc) {
          REQUIRE(BAL && pieces == 1 && published[t.u] < 0);
          published[t.u] = blk;
          cut[t.u] = t.s1;
        } else {
          ++ends[t.u];
        }
      }
      su = t.u;
      ss = t.s;
    }
  }
  REQUIRE(all == (long long)units * nc);
  for (int u = 0; u < units; ++u) REQUIRE(ends[u] == 1);
  return true;
}

template <int P>
static bool check_all(const G& g, int sms) {
  const StatePlan p = state_plan(g.nc, g.B * g.G * (g.hpg * P / 128), 64, sms);
  return p == StatePlan::shares ? check_walk<P, true>(g, sms, p) : check_walk<P, false>(g, sms, p);
}

int main() {
  for (int sms : {148, 132})
    for (int units = 1; units <= 2000; ++units)
      for (int nc = 1; nc <= 1200; ++nc)
        for (int n : {64, 128})
          if (!check_rule(units, nc, sms, state_plan(nc, units, n, sms))) return 1;
  const int chunks[] = {1, 2, 3, 8, 15, 16, 17, 31, 32, 33, 63, 87, 88, 89, 120, 147, 148, 149, 255, 256, 511, 1024, 1200};
  for (int sms : {148, 132})
    for (int nc : chunks) {
      for (int B = 1; B <= 300; ++B)
        if (!check_all<32>(G{B, 1, 4, nc}, sms)) return 1;        // one unit per batch row
      for (int B = 1; B <= 100; B += nc > 256 ? 7 : 1) {
        if (!check_all<32>(G{B, 1, 8, nc}, sms)) return 1;        // 8 heads of 32: 2 units
        if (!check_all<64>(G{B, 2, 4, nc}, sms)) return 1;        // two groups of 4 heads of 64
        if (B <= 40 && !check_all<64>(G{B, 1, 24, nc}, sms)) return 1;   // 24 heads of 64: 12 units
      }
    }
  std::puts("ok");
  return 0;
}
