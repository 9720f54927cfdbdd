"""The staging of host arrays (csrc/host_io.hpp) against a stand-in for the CUDA
runtime, on the CPU: every size class with pageable, pinned and device arrays in
every place, and the pinned pool at its limits."""
import os
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def host_io(tmp_path_factory):
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    exe = str(tmp_path_factory.mktemp("host_io") / "host_io")
    subprocess.run(["g++", "-O1", "-std=c++17", "-Wall", "-Wextra", "-Werror", "-Wno-unknown-pragmas", "-fopenmp",
                    "-isystem", os.path.join(cuda, "include"), os.path.join(ROOT, "tests", "cpp", "host_io.cpp"),
                    "-o", exe], check=True)

    def run(*args):
        return subprocess.run([exe, *map(str, args)], check=True, capture_output=True, text=True).stdout.split("\n")
    return run


# bytes of each of four arrays: around 64 KB and 1 MB in all, one and several chunks
SIZES = (1, 16384, 16385, 262144, 262145, 3000001)


@pytest.mark.parametrize("kinds", ["hhhh", "phhh", "hphh", "hhph", "hhhp", "pppp"])
def test_host_arrays_arrive_and_return(host_io, kinds):
    for n in SIZES:
        assert host_io("copy", n, kinds)[0] == "ok", n


@pytest.mark.parametrize("kinds", ["dhhh", "hdhh", "hhdh", "hhhd", "dddd", "pdph"])
def test_device_memory_is_left_to_the_cuda_copy(host_io, kinds):
    """A device pointer among host arrays: the host never reads or writes it; the
    CUDA copy with the call's direction takes it or refuses it (here: refuses)."""
    for n in SIZES:
        assert host_io("copy", n, kinds)[0] == "error 1", n


def test_pool_limits(host_io):
    assert host_io("pool")[:-1] == ["blocks 16 4 pinned 20",
                                    "out ok", "out ok", "out ok", "pinned by them 0",
                                    "after the last scene 0",
                                    "none ok", "none ok", "none ok"]
