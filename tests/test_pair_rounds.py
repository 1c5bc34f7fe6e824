"""The barriers of two warps that share rows (csrc/pair_rounds.h), on the CPU: whatever wait of either warp gives up at whatever tile,
both take the same barriers in the same order and leave the walk together."""

import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "edgerag_b200" / "csrc"

# A warp's walk as the kernels have it, stopped at each of its barriers.  `rule` 0: leaves at once where a wait gives up; 1: the header's.
DRIVER = r"""
#include <cstdio>
#include "pair_rounds.h"
using namespace erb;

const int kTiles = 4;
enum At { kExchange, kVote, kEnd };

struct Warp {
  int rule, fails_tile, fails_site;                // site 0: the wait for the scores, 1: the wait before O is rescaled
  unsigned low;                                    // tiles whose sum asks for a higher reference
  volatile int* flag;                              // the block's
  int tile = 0;
  bool ok = true, alone = false, left = false;     // alone: the wait for the scores gave up
  PairRounds pair{true};

  void fail() { ok = false; *flag = 1; }
  At start_tile() {
    if (left || tile == kTiles) return kEnd;
    pair = PairRounds(tile == 0);
    if (fails_tile == tile && fails_site == 0) { fail(); alone = true; }
    if (!ok && rule == 0) { left = true; return kEnd; }
    return pair.search() ? kExchange : kVote;
  }
  At after_exchange() {
    if (fails_tile == tile && fails_site == 1 && tile > 0 && !alone) fail();
    if (!ok && rule == 0) { left = true; return kEnd; }
    return kVote;
  }
  bool vote() const { return alone || pair.vote(low >> tile & 1, flag); }
  At after_vote(bool any) {
    if (any && pair.again()) return kExchange;
    if (any) { ok = false; left = true; return kEnd; }
    ++tile;
    return start_tile();
  }
};

// 0: both end together; 1: one waits at a barrier that the other never comes to
int meet(Warp a, Warp b, bool& both_ok) {
  At x = a.start_tile(), y = b.start_tile();
  for (int barriers = 0; barriers < 4 * kTiles; ++barriers) {
    if (x != y) return 1;
    if (x == kEnd) { both_ok = a.ok && b.ok && a.tile == kTiles && b.tile == kTiles; return a.left != b.left; }
    if (x == kExchange) { x = a.after_exchange(); y = b.after_exchange(); }
    else { const bool any = a.vote() || b.vote(); x = a.after_vote(any); y = b.after_vote(any); }
  }
  return 1;
}

int main() {
  int stuck[2] = {0, 0}, cases = 0, wrong = 0;
  for (int rule = 0; rule < 2; ++rule)
    for (int fa = -1; fa < kTiles; ++fa) for (int sa = 0; sa < 2; ++sa)
      for (int fb = -1; fb < kTiles; ++fb) for (int sb = 0; sb < 2; ++sb)
        for (unsigned la = 0; la < 1u << kTiles; ++la) for (unsigned lb = 0; lb < 1u << kTiles; ++lb) {
          bool both_ok = false;
          volatile int flag = 0;
          Warp a{rule, fa, sa, la, &flag}, b{rule, fb, sb, lb, &flag};
          const int s = meet(a, b, both_ok);
          stuck[rule] += s;
          if (rule == 1) {
            ++cases;
            // a wait is reached where the walk has not ended before it and, the second, where the tile is searched behind the first
            const bool none = fa < 0 && fb < 0;
            if (none && !both_ok) ++wrong;
            if ((fa >= 0 && sa == 0) || (fb >= 0 && sb == 0)) wrong += both_ok;
          }
        }
  std::printf("%d %d %d %d\n", stuck[0], stuck[1], cases, wrong);
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no g++")
def test_two_warps_meet_at_the_same_barriers(tmp_path):
    source, program = tmp_path / "meet.cpp", tmp_path / "meet"
    source.write_text(DRIVER)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", f"-I{CSRC}", str(source), "-o", str(program)], check=True)
    stuck_before, stuck, cases, wrong = map(int, subprocess.run([str(program)], check=True, capture_output=True, text=True).stdout.split())
    assert cases == 25600 and stuck == 0 and wrong == 0
    assert stuck_before > 0                                    # (the driver sees a warp that leaves alone)


@pytest.mark.parametrize("kernel", ["attention_prefill.cu", "attention_wide.cu"])
def test_kernels_leave_the_tiles_by_the_vote_alone(kernel):
    """From the wait for a tile's scores to the vote no warp leaves by itself: one that gave up comes to the pair's barriers first."""
    text = (CSRC / kernel).read_text()
    head, rest = text.split("PairRounds pair(")
    walk, behind = rest.split("pair.vote(!(l_tile < kSumLimit), s_abort)", 1)
    assert "if (!ok) break;" not in head[head.rindex("for (int j ="):] + walk
    given_up = walk.index("named_barrier_any(pair_barrier, 64, true);")     # the one way out before the vote has the pair's barriers in it
    assert walk[given_up:].index("while (pair.again());") < walk[given_up:].index("break;")
    assert behind.index("if (!pair.again()) { ok = false; break; }") < behind.index("mbar_arrive")
