"""What the pipeline's autotuner decides from its times: a bin is merged into the next one only where the
shape that it keeps runs as fast there (the decisions are host code, compiled here by itself)."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "custingeralg_b200", "csrc")
PROGRAM = """
#include <cstdio>
#include <cstdlib>
#include "tc_pipe_tune.h"
int main(int argc, char** argv) {
  tc::BinTimes t;
  for (int i = 1; i + 1 < argc; i += 2) t.add(std::atoi(argv[i]), std::atof(argv[i + 1]));
  std::printf("%d %d %d %d", t.best(4), (int)t.merges(), t.next(tc::kPipeArms), t.next(tc::kPipeCands));
}
"""
UP = 5  # the arm in the next bin's graph


@pytest.fixture(scope="module")
def decide(tmp_path_factory):
    d = tmp_path_factory.mktemp("tune")
    (d / "t.cpp").write_text(PROGRAM)
    exe = str(d / "t")
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", CSRC, str(d / "t.cpp"), "-o", exe], check=True)

    def run(*samples):
        args = [str(x) for s in samples for x in s]
        best, merges, nxt, nxt_own = map(int, subprocess.run([exe] + args, check=True, capture_output=True,
                                                             text=True).stdout.split())
        return best, bool(merges), nxt, nxt_own
    return run


def test_merge_compares_the_shape_that_the_bin_keeps(decide):
    # items of 1024 entries: 10 alone and 10.2 padded; of 64: 1.0 alone, 1.5 padded
    assert decide((0, 10.0), (4, 1.0), (UP, 1.5))[:2] == (4, False)
    assert decide((0, 10.0), (4, 1.0), (UP, 1.02))[:2] == (4, True)
    assert decide((4, 1.0), (4, 3.0), (2, 1.9), (UP, 1.94))[:2] == (2, True)  # means, not single samples


def test_nothing_is_merged_or_changed_without_samples(decide):
    assert decide() == (4, False, 0, 0)
    assert decide((UP, 1.0))[:2] == (4, False)
    assert decide((1, 1.0))[:2] == (1, False)


def test_arms_take_turns(decide):
    assert decide((0, 1.0))[2:] == (1, 1)
    assert decide(*[(a, 1.0) for a in range(5)])[2:] == (UP, 0)
    assert decide(*[(a, 1.0) for a in range(6)])[2:] == (0, 0)
