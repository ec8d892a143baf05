"""Compile-time switches refuse the values that the kernels cannot take."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "kairos_engine_b200", "csrc")


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="no CUDA compiler")
def test_parts_smaller_than_a_tile_do_not_compile(tmp_path):
    """A tile of eight routed pairs waits for the part of its first pair: parts of four would be multiplied before they land."""
    r = subprocess.run(["nvcc", "-std=c++17", "-cuda", "-gencode", "arch=compute_100a,code=sm_100a", "-DSP_DS_LP=2", os.path.join(CSRC, "decode_staged.cu"), "-o", str(tmp_path / "x.ii")],
                       capture_output=True, text=True)
    assert r.returncode != 0 and "whole tiles of eight pairs" in r.stderr, r.stderr[-2000:]
