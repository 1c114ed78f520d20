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

    def run(*blocks):
        out = subprocess.run([exe, *map(str, blocks)], check=True, capture_output=True, text=True).stdout
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
