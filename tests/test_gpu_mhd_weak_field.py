"""Mixed MHD over the range of its field, density and pressure: the FP32 HLLD
flux and corner emf against the FP64 ones, and runs with a field so weak that
its square times a density leaves FP32's range."""

import os
import subprocess

import numpy as np
import pytest

import euler_kokkos_gb300 as ek
from euler_kokkos_gb300 import build as B
from euler_kokkos_gb300 import problems as P
from helpers import interior, rel_l1

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.gpu
def test_fp32_speeds_over_exponents(tmp_path):
    exe = str(tmp_path / "fp32_speeds")
    subprocess.run([B._nvcc(), os.path.join(HERE, "fp32_speeds.cu"), "-o", exe, "-I" + B.CSRC, "-std=c++17", "-O2",
                    "-DEK_NS=ek_fast", "--fmad=true", "--ftz=true", "--prec-div=false", "--prec-sqrt=false"] + B.ARCH,
                   check=True)
    emf, flux, faces = (float(x) for x in subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split())
    # relative to (|u| + c) |B| and to the flux of the state: about 40 roundings of 2^-24 (2.4e-6), star quotients
    # that amplify them up to four times at these contrasts, approximate roots and reciprocals of 2 ulp; a speed
    # that is infinite, zero or off by 2^(1/2) is an error above 1e-1
    assert emf <= 1e-4 and flux <= 1e-4
    assert faces > 1000  # solved in FP32, not left to the repair pass


@pytest.mark.gpu
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("field", [1e-19, 1e-18, 1e-17])
def test_weak_field_in_thin_gas(dim, field):
    n = 48 if dim == 2 else 24
    ini, U0 = P.smooth_random(dim=dim, mhd=True, nx=n, seed=5, bc=(3, 3, 2, 2, 1, 1), nsteps=10)
    b = U0[5:].copy()
    U0[1] -= 0.5 * sum((0.5 * (b[c] + np.roll(b[c], -1, axis=2 - c))) ** 2 if c < dim else b[c] ** 2 for c in range(3))
    U0[:5] *= 1e-3  # density and pressure; the magnetic energy is nothing beside it
    U0[5:] = field * b
    out = []
    for prec in (ek.EK_PREC_FP64, ek.EK_PREC_MIXED):
        with ek.Solver(ek.params_from_ini(ini, precision=prec)) as s:
            s.set_state(U0)
            assert s.run(10) == 10
            out.append(interior(s.get_state(), 3, dim))
    assert np.isfinite(out[1]).all()
    err = rel_l1(out[1], out[0])
    # density and energy: the mixed form's bound.  The field: the FP32 limiter's product of two differences flushes to
    # zero below 1e-19, and such a field is advected to first order; ten steps of that smooth a wave of 24 cells by
    # v (1 - v) (2 pi / 24)^2 / 2 each, up to 8 % in all at a Courant number of a half
    assert max(err[:2]) <= 1e-5 and max(err[5:5 + dim]) <= 8e-2, err
