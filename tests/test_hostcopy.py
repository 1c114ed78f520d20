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
    subprocess.run(["g++", "-std=c++17", "-O1", "-x", "c++", "-I", os.path.join(cuda, "include"), "-I",
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
