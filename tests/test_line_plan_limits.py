"""Index limits of the plans of tiles of lines, on the host.

The pivots' sweep keeps two values a position in a vector that its kernels
index by int, so it must refuse plans of 2^30 positions or more (a factor of
some 540 million rows in lines of uneven length); ILU(0) is then made by levels.
"""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "matrix-toolkits-java_gb300", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def _run(tmp_path, body):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text('#include <cstdio>\n#include "lines.cuh"\nint main() {\n' + body + "\n}\n")
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, "-I", os.path.join(ROOT, "include"),
                    "-I", os.path.join(CUDA, "include"), "-o", str(exe), str(src)], check=True)
    return subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()


@pytest.mark.parametrize("positions", [0, 1, 2**29, 2**30 - 1, 2**30, 2**30 + 1, 1431650000, 2**31 - 1])
def test_pivot_pairs(tmp_path, positions):
    out = _run(tmp_path, f'std::printf("%d", (int)mtjg::pivot_pairs_fit({positions}LL));')
    last = 2 * (positions - 1) + 1  # the largest index used
    assert out == ["1" if last < 2**31 - 1 or positions == 0 else "0"]
