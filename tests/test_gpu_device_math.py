"""Device arithmetic helpers checked against CUDA's own results on the GPU."""

import subprocess
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
HERE = Path(__file__).resolve().parent


def test_fast_reciprocal_within_two_ulps(tmp_path):
    """sapb::fast_recip (Newton-Raphson from the hardware's approximation, used
    for the pivots of a factor handed in) stays within 2 ulps of the IEEE
    quotient 1.0/d over 1e-35..1e35."""
    exe = tmp_path / "recip_check"
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-o", str(exe),
                    str(HERE / "cuda" / "recip_check.cu")], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout
    worst = int(out.split("max_ulps")[1].split()[0])
    assert worst <= 2, out


def test_pivot_reciprocals(tmp_path):
    """The factorizations' pivot reciprocals over the whole range of both types.
    Newton-Raphson squares the seed's error (two steps from the FP64 seed's
    1e-6, one from the FP32 seed's ulp) and rounds the last step once: within
    2 ulps of the IEEE quotient wherever the result counts as positive and
    normal; where it must not (d not positive, subnormal or not finite, or a
    quotient that is not normal) it does not."""
    exe = tmp_path / "pivot_check"
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-o", str(exe),
                    str(HERE / "cuda" / "pivot_check.cu")], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout
    rows = {line.split()[0]: [int(x) for x in line.split()[2::2]] for line in out.splitlines()}
    assert set(rows) == {"fp64", "fp32"}, out
    for worst, taken, wrong in rows.values():
        assert worst <= 2 and wrong == 0 and taken > 0, out
