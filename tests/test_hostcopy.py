"""The copies of fields between pageable host memory and the device by several
threads (hostcopy.cu), on the host with a fake CUDA runtime
(native/hostcopy_fake.cpp)."""
import os
import subprocess

import pytest

from conftest import ROOT

MB = 1 << 20


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("native") / "hostcopy_fake")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-O3", "-x", "c++", "-I", os.path.join(cuda, "include"), "-I",
                    os.path.join(ROOT, "glac_b200", "csrc"),
                    os.path.join(ROOT, "tests", "native", "hostcopy_fake.cpp"), "-o", exe, "-lpthread"], check=True)

    def run(*steps, cores=16):
        out = subprocess.run([exe, str(cores), *map(str, steps)], capture_output=True, text=True, timeout=60)
        assert out.returncode == 0, (out.returncode, out.stdout, out.stderr)
        return [[int(x) for x in line.split()] for line in out.stdout.splitlines()]

    return run


@pytest.mark.parametrize("way", ["up", "down"])
def test_no_memory_for_a_thread(fake, way):
    # a thread that cannot be made leaves its pieces to the others; 400 MB are taken
    # in pieces whatever the memory held so far
    assert fake("hold", "fail", way, 400 * MB + 7, "drop")[0][0] == 401


PINNED = 16 * MB


def test_short_lived_contexts_pin_nothing(fake):
    # a context per configuration of 24 MB: pinning for its two copies would cost more than they take
    life = ["hold", "up", 24 * MB, "down", 24 * MB, "pinned", "drop"]
    assert fake(*(life * 4)) == [[1], [1], [0, 0], [0]] * 4


def test_buffers_come_with_a_large_copy_and_go_with_the_last_holder(fake):
    out = fake("hold", "hold", "up", 63 * MB, "pinned", "up", 64 * MB, "pinned", "down", 24 * MB + 1, "drop", "down",
               80 * MB, "drop", "pinned")
    assert out == [[1], [0, 0], [64], [PINNED, 1], [25], [PINNED], [80], [0], [0, 1]]


def test_buffers_come_after_enough_small_copies(fake):
    # 40 MB at a time: the seventh copy passes 256 MB; what small copies moved counts from the last holder's end
    seven = ["up", 40 * MB] * 3 + ["down", 40 * MB] * 3 + ["pinned", "up", 40 * MB, "pinned"]
    before, after = [[1]] * 6 + [[0, 0]], [[40], [PINNED, 1]]
    assert fake("hold", *seven, "drop") == before + after + [[0]]
    part = ["hold", *seven[:12], "drop"]
    assert fake(*part, *part) == ([[1]] * 6 + [[0]]) * 2


@pytest.mark.parametrize("cores, least", [(1, None), (2, 128 * MB), (3, 16 * MB), (4, 10 * MB), (16, 10 * MB),
                                          (-2, 128 * MB), (-8, 10 * MB), (0, None)])
def test_few_cores_copy_plainly(fake, cores, least):
    # one transfer each just below the size from which copies are split and, where
    # they never are, of 400 MB; with the buffers there, a transfer per MB from it on
    make = ["hold"] + ["up", 400 * MB] * 2
    if least is None:
        assert fake(*make, "pinned", cores=cores) == [[1], [1], [0, 0]]
    else:
        out = fake(*make, "up", least - 1, "down", least - 1, "up", least, "down", least, cores=cores)
        assert out == [[400], [400], [1], [1], [least // MB], [least // MB]]


def test_a_forked_child_leaves_the_buffers_alone(fake):
    assert fake("hold", "up", 64 * MB, "forked", "up", 64 * MB, "drop") == [[64], [0], [64], [0]]
