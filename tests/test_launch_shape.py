"""The launch shape of the flux form's kernel A (flux_shape of csrc/p2de_launch.h), compiled for
the host: the block width follows the device's multiprocessor count, and both layouts' defaults
lie where its comment says."""
import shutil
import subprocess
from pathlib import Path

import pytest

from conftest import ROOT

SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include "p2de_launch.h"
int main(int argc, char** argv) {
  const p2de::FluxShape s = p2de::flux_shape(std::atoi(argv[1]), std::atoi(argv[2]), std::atoi(argv[3]),
                                             std::atoi(argv[4]), std::atoi(argv[5]), std::atoi(argv[6]));
  std::printf("%d %d %d", s.split, s.epb, s.threads);
}
"""


@pytest.fixture(scope="module")
def flux_shape(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    include = Path(nvcc).resolve().parent.parent / "include"
    if shutil.which("g++") is None or not (include / "cuda_runtime.h").exists():
        pytest.skip("needs g++ and the CUDA headers")
    d = tmp_path_factory.mktemp("shape")
    (d / "shape.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-I", str(include), "-I", str(ROOT / "p2de.jl_gb300" / "csrc"),
                    str(d / "shape.cpp"), "-o", str(d / "shape")], check=True)

    def call(n1d, K, epb, ext, acc64, sms):
        out = subprocess.run([str(d / "shape"), *(str(int(v)) for v in (n1d, K, epb, ext, acc64, sms))], check=True,
                             capture_output=True, text=True).stdout
        return tuple(int(v) for v in out.split())

    return call


def test_block_width_follows_the_multiprocessors(flux_shape):
    # N = 3, 4 elements a block: ten blocks an SM are 40 elements an SM
    for sms in (8, 76, 152):
        assert flux_shape(4, 40 * sms - 4, 4, True, False, sms) == (0, 4, 128)
        assert flux_shape(4, 40 * sms, 4, True, False, sms) == (0, 4, 64)


@pytest.mark.parametrize("n1d,epb,first", [(2, 16, 16384), (3, 10, 7282), (4, 4, 4096), (5, 6, 4400), (6, 5, 3056)])
def test_split_ends_at_its_node_count(flux_shape, n1d, epb, first):
    assert flux_shape(n1d, first - 1, epb, False, False, 152)[0] == 1
    assert flux_shape(n1d, first, epb, False, False, 152)[0] == 0
    assert flux_shape(n1d, first - 1, epb, True, False, 152)[0] == 0
