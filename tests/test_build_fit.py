"""A cooperative launch that the context cannot hold as a whole is refused
before it runs; the tree build's is then tried with half as many blocks.  The
launches here are a fake that holds `room` blocks, so no GPU is needed."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = "/usr/local/cuda/include"

SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include "fa2_internal.cuh"
static int last = 0;
extern "C" cudaError_t cudaGetLastError() { last = 0; return cudaSuccess; }
int main(int argc, char **argv) {
    const int room = atoi(argv[2]), fails = atoi(argv[3]);
    int blocks = atoi(argv[1]), tried = 0;
    const cudaError_t e = fa2::launch_fitting(blocks, [&](int n) {
        ++tried;
        if (fails) return cudaErrorLaunchFailure;
        if (n <= room) return cudaSuccess;
        last = cudaErrorCooperativeLaunchTooLarge;
        return cudaErrorCooperativeLaunchTooLarge;
    });
    printf("%d %d %d %d\n", blocks, tried, (int)(e == cudaSuccess), last);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    if not shutil.which("g++") or not os.path.isdir(CUDA):
        pytest.skip("needs g++ and the CUDA headers")
    d = tmp_path_factory.mktemp("fit")
    (d / "fit.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-I", CUDA, "-I",
                    os.path.join(ROOT, "gpugraphlayout_b200", "csrc"), "-o", str(d / "fit"),
                    str(d / "fit.cpp")], check=True)
    return str(d / "fit")


@pytest.mark.parametrize("blocks,room,fails,want", [
    (148, 296, 0, "148 1 1 0"),   # the whole device
    (148, 148, 0, "148 1 1 0"),
    (148, 74, 0, "74 2 1 0"),     # no error is left behind
    (148, 30, 0, "19 4 1 0"),
    (10, 1, 0, "1 5 1 0"),
    (1, 1, 0, "1 1 1 0"),
    (148, 148, 1, "148 1 0 0"),   # another error is not one of size
])
def test_blocks_halve_until_they_fit(program, blocks, room, fails, want):
    out = subprocess.run([program, str(blocks), str(room), str(fails)], check=True,
                         capture_output=True, text=True).stdout
    assert out.strip() == want


def test_one_block_that_does_not_fit_is_an_error(program):
    out = subprocess.run([program, "4", "0", "0"], check=True, capture_output=True, text=True).stdout
    blocks, tried, ok, _ = map(int, out.split())
    assert (blocks, tried, ok) == (1, 3, 0)
