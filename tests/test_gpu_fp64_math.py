"""The FP64 FMA build's reciprocals, roots, limiter and integer-pipe minima
(ek_common.cuh, ek_hydro.cuh) against CUDA's own functions."""

import os
import subprocess

import pytest

from euler_kokkos_gb300 import build as B

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("fp64") / "fp64_math")
    subprocess.run([B._nvcc(), os.path.join(HERE, "fp64_math.cu"), "-o", exe, "-I" + B.CSRC, "-std=c++17", "-O2",
                    "-DEK_NS=ek_fast", "--fmad=true"] + B.ARCH, check=True)
    return exe


@pytest.mark.gpu
@pytest.mark.parametrize("spread", [4, 40, 300])
def test_fp64_helpers(program, spread):
    out = subprocess.run([program, str(spread)], check=True, capture_output=True, text=True).stdout.split()
    rcp, rsqrt, root, ratio, scale, slope, minmax, special = (float(x) for x in out)
    # in 2^-53: the last rounding, and under 0.05 of series remainder (seeds of 2^-19 or better, third order);
    # the root also carries half the rounding of x y; the ratio's roundings n d (half), rsqrt, product, and CUDA's
    # own quotient (half) and root: 0.5 + 1.05 + 1 + 0.5 + 1
    assert rcp <= 1.05 and rsqrt <= 1.05 and root <= 1.55 and ratio <= 4.1
    assert scale == 0 and slope == 0 and minmax == 0 and special == 0
