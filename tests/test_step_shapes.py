"""The 2D grid stepper's CTAs hold whole tiles: a shape whose lines per CTA do not
divide the length must not compile, since a thread of its last CTA would own a row
without owning a column (or the reverse) and would add stale registers to the norm."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="needs nvcc")
@pytest.mark.parametrize("lines,ok", [(8, True), (7, False)])
def test_lines_per_cta_divide_the_length(tmp_path, lines, ok):
    src = tmp_path / "shape.cu"
    src.write_text('#include "stepper.cuh"\n'
                   "size_t bytes() { return gpue::StepShape<float, 1024, 16, 4, 0, 64, %d>"
                   "::fixed_bytes(); }\n" % lines)
    r = subprocess.run(["nvcc", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a",
                        "-I", os.path.join(ROOT, "gpue_b200", "csrc"), "-c", "-o", os.devnull,
                        str(src)], capture_output=True, text=True)
    assert (r.returncode == 0) == ok, r.stderr[-2000:]
    if not ok:
        assert "whole rows" in r.stderr
