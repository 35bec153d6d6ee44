"""What the pipeline's autotuner decides from its times: a bin is merged into a larger one only where the shape
that it keeps runs as fast there (the decisions are host code, compiled here by itself)."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "custingeralg_b200", "csrc")
# arguments: bin, arm, ms, updates of each sample; output: per bin its best arm, next arms and server
PROGRAM = """
#include <cstdio>
#include <cstdlib>
#include "tc_pipe_tune.h"
int main(int argc, char** argv) {
  tc::BinTimes t[4];
  int serve[4];
  for (int i = 1; i + 3 < argc; i += 4)
    t[std::atoi(argv[i])].add(std::atoi(argv[i + 1]), std::atof(argv[i + 2]), std::atoll(argv[i + 3]));
  tc::merge_bins(t, 4, serve);
  for (int i = 0; i < 4; ++i)
    std::printf("%d %d %d %d\\n", t[i].best(4), t[i].next(tc::kPipeArms), t[i].next(tc::kPipeCands), serve[i]);
}
"""
UP = 5  # the arm in the next bin's graph


@pytest.fixture(scope="module")
def decide(tmp_path_factory):
    d = tmp_path_factory.mktemp("tune")
    (d / "t.cpp").write_text(PROGRAM)
    exe = str(d / "t")
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", CSRC, str(d / "t.cpp"), "-o", exe], check=True)

    def run(samples):
        args = [str(x) for s in samples for x in s]
        out = subprocess.run([exe] + args, check=True, capture_output=True, text=True).stdout.split("\n")
        return [tuple(map(int, line.split())) for line in out[:4]]
    return run


def _bin(i, times, updates=1000):
    return [(i, arm, ms, updates) for arm, ms in times]


def test_merge_compares_the_shape_that_the_bin_keeps(decide):
    # items of 1024 entries: 10 alone and 10.2 padded; of 64: 1.0 alone, 1.5 padded
    best, _, _, serve = decide(_bin(0, [(0, 10.0), (4, 1.0), (UP, 1.5)]))[0]
    assert (best, serve) == (4, 0)
    best, _, _, serve = decide(_bin(0, [(0, 10.0), (4, 1.0), (UP, 1.02)]))[0]
    assert (best, serve) == (4, 1)
    # means over the samples, by update
    samples = _bin(0, [(4, 1.0), (4, 3.0), (2, 1.9)]) + _bin(0, [(UP, 3.88)], updates=2000)
    best, _, _, serve = decide(samples)[0]
    assert (best, serve) == (2, 1)


def test_a_chain_of_merges_adds_up(decide):
    def serves(*ms):  # bins of ms a batch, each step of 0.02 ms more
        return [r[3] for r in decide([s for i, t in enumerate(ms) for s in _bin(i, [(4, t), (UP, t + 0.02)])])]
    assert serves(8.0, 8.0, 8.0) == [3, 3, 3, 3]  # 0.06 of 8
    assert serves(1.0, 1.0, 1.0) == [1, 1, 3, 3]
    assert serves(1.0, 2.0, 4.0) == [0, 3, 3, 3]  # 0.06 of 1, 0.04 of 2, 0.02 of 4
    assert serves(0.5, 0.5, 4.0) == [0, 1, 3, 3]
    # a step that measured faster counts as nothing, not as a credit for the others
    fast = _bin(2, [(4, 4.0), (UP, 3.0)])
    assert [r[3] for r in decide(fast + _bin(1, [(4, 1.0), (UP, 1.1)]))] == [0, 1, 3, 3]


def test_nothing_is_merged_or_changed_without_samples(decide):
    assert decide([]) == [(4, 0, 0, i) for i in range(4)]
    assert decide(_bin(1, [(UP, 1.0)]))[1][::3] == (4, 1)
    assert decide(_bin(1, [(1, 1.0)]))[1][::3] == (1, 1)


def test_arms_take_turns(decide):
    assert decide(_bin(2, [(0, 1.0)]))[2][1:3] == (1, 1)
    assert decide(_bin(2, [(a, 1.0) for a in range(5)]))[2][1:3] == (UP, 0)
    assert decide(_bin(2, [(a, 1.0) for a in range(6)]))[2][1:3] == (0, 0)
