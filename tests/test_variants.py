"""What the launch variants' numbers stand for (variants.cuh)."""
import os
import subprocess

import pytest

from conftest import ROOT

FLOW, METRO, OBS = 0, 1, 2


@pytest.fixture(scope="module")
def lines(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("native") / "variants")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "glac_b200", "csrc"),
                    os.path.join(ROOT, "tests", "native", "variants.cpp"), "-o", exe], check=True)

    def run(*args):
        out = subprocess.run([exe, *map(str, args)], check=True, capture_output=True, text=True).stdout
        return [tuple(int(x) for x in line.split()) for line in out.splitlines()]

    return run


def test_numbers_keep_their_meaning(lines):
    # a tuning is kept by its numbers, so these do not move (the defaults, number 0, may)
    forms = {x[:3]: x[3:] for x in lines()}
    assert {k[:2]: 1 + max(v for f, p, v in forms if (f, p) == k[:2]) for k in forms} == {
        (FLOW, 0): 4, (FLOW, 1): 4, (METRO, 0): 2, (METRO, 1): 4, (OBS, 0): 2, (OBS, 1): 3}
    want = {(FLOW, 0): {1: (128, 0), 2: (0, 1), 3: (128, 2)}, (FLOW, 1): {1: (80, 0), 2: (0, 3), 3: (96, 0)},
            (METRO, 0): {1: (128, 0)}, (METRO, 1): {1: (96, 0), 2: (80, 0), 3: (128, 0)},
            (OBS, 0): {1: (128, 0)}, (OBS, 1): {1: (128, 0), 2: (168, 0)}}
    for (f, p), per in want.items():
        for v, form in per.items():
            assert forms[f, p, v] == form, (f, p, v)


@pytest.mark.parametrize("case, flow64, flow32, metro64, metro32", [
    # split, Morningstar, learned, blocks of a sub-sweep
    ((1, 1, 0, 32), (0, 1, 2, 3), (0, 1, 2, 3), (0, 1), (0, 1, 2, 3)),          # several warps to a link
    ((0, 1, 0, 5 * 148), (0, 0, 2, 3), (0, 0, 2, 3), (0, 1), (0, 1, 2, 0)),     # one wave: 128 registers
    ((0, 1, 0, 5 * 148 + 1), (0, 0, 2, 3), (0, 0, 2, 3), (0, 1), (0, 0, 2, 3)),  # 96
    ((0, 1, 1, 8192), (0, 0, 2, 3), (0, 0, 2, 3), (0, 0), (0, 1, 2, 0)),        # learned; FP64 beyond ten blocks per SM
    ((0, 0, 0, 1480), (0, 0, 0, 0), (0, 0, 2, 0), (0, 1), (0, 0, 2, 3)),        # another exponential
    ((0, 0, 0, 1481), (0, 0, 0, 0), (0, 0, 2, 0), (0, 0), (0, 0, 2, 3))])
def test_variants_that_launch_the_same_kernel(lines, case, flow64, flow32, metro64, metro32):
    assert lines(*case) == [(FLOW, 0, *flow64), (FLOW, 1, *flow32), (METRO, 0, *metro64), (METRO, 1, *metro32)]
