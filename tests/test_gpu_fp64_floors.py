"""Floors of the FP64 FMA build: a density or energy that is not a number, a
negative pressure with smallc = 0.  The exact build (the reference's fmax) is
the result to agree with."""

import os
import subprocess

import numpy as np
import pytest

import euler_kokkos_gb300 as ek
from euler_kokkos_gb300 import build as B
from euler_kokkos_gb300 import problems as P
from helpers import interior, rel_linf

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))

# tile kernels and passes of both dimensions
GRIDS = [(2, False, (40, 24, 1)), (2, False, (520, 512, 1)), (3, False, (20, 18, 12)), (2, True, (40, 24, 1)),
         (2, True, (200, 180, 1)), (3, True, (20, 18, 12))]
IDS = ["%s%dd_%dx%d" % ("mhd" if m else "hydro", d, n[0], n[1]) for d, m, n in GRIDS]


def _both(ini, U0, gw, dim, steps):
    out = []
    for exact in (1, 0):
        with ek.Solver(ek.params_from_ini(ini, exact_fp=exact)) as s:
            s.set_state(U0)
            s.run(steps, allow_nonfinite=True)
            out.append((interior(s.get_state(), gw, dim), s.dt_history()))
    return out


def _state(dim, mhd, n, gw):
    ini, U0 = P.smooth_random(dim=dim, mhd=mhd, nx=n[0], ny=n[1], nz=n[2], seed=9, nsteps=2)
    k = n[2] // 2 + gw if dim == 3 else 0
    return ini, U0, (k, n[1] // 2 + gw, n[0] // 2 + gw)

@pytest.fixture(scope="module")
def limits(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("fp64") / "fp64_limits")
    subprocess.run([B._nvcc(), os.path.join(HERE, "fp64_limits.cu"), "-o", exe, "-I" + B.CSRC, "-std=c++17", "-O2",
                    "-DEK_NS=ek_fast", "--fmad=true"] + B.ARCH, check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split()
    return dict(zip(out[::2], map(float, out[1::2])))


def test_floor_helpers(limits):
    assert limits["floors"] == 0 and limits["nan"] == 0  # values of fmax


def test_roots_of_quotients(limits):
    # as test_gpu_fp64_math.py's ratio, whose bound holds where n d leaves the range too (reciprocal 1.05 and product 0.5,
    # halved by the root, and the root 1.55); the fast speed: two roots of at most 1.55, sums and the difference, of which
    # the discriminant is no less than 0.3 of its first term
    assert limits["ratio"] <= 4.1 and limits["larger"] <= 4.1 and limits["fast"] <= 8


# scales beyond the roots of the number range: LLF takes no products of two densities
@pytest.mark.parametrize("dim,mhd,n", GRIDS, ids=IDS)
@pytest.mark.parametrize("power", [-512, 520])
def test_densities_beyond_the_root_of_the_range(dim, mhd, n, power):
    gw = 3 if mhd else 2
    ini, U0, _ = _state(dim, mhd, n, gw)
    ini = ini.replace("riemann=hlld", "riemann=llf").replace("riemann=hllc", "riemann=llf")
    ini = ini.replace("[hydro]", "[hydro]\nsmallr=0.0")
    U0 = U0 * 2.0 ** power
    U0[5:] *= 2.0 ** (-power // 2)
    (Ue, de), (Uf, df) = _both(ini, U0, gw, dim, 1)
    assert np.isfinite(Ue).all() and np.isfinite(Uf).all()
    assert np.max(np.abs(df / de - 1)) <= 1e-13
    assert np.max(rel_linf(Uf, Ue)[[0, 1]]) <= 1e-11


@pytest.mark.parametrize("var", [0, 1], ids=["density", "energy"])
@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("dim,mhd,n", GRIDS, ids=IDS)
def test_nan_is_floored(dim, mhd, n, var, sign):
    gw = 3 if mhd else 2
    ini, U0, at = _state(dim, mhd, n, gw)
    U0[(slice(2, 5 if U0.shape[0] > 4 else 4),) + at] = 0.0  # a density of smallr with a momentum would be a jet
    U0[(var,) + at] = np.copysign(np.nan, sign)
    (Ue, de), (Uf, df) = _both(ini, U0, gw, dim, 2)
    assert np.array_equal(np.isnan(Ue), np.isnan(Uf))
    assert np.isnan(Ue).sum() == 1  # the cell itself: its neighbours see the floor
    ok = ~np.isnan(Ue)
    assert np.max(rel_linf(np.where(ok, Uf, 0.0), np.where(ok, Ue, 0.0))[[0, 1]]) <= 1e-11
    assert np.max(np.abs(df / de - 1)) <= 1e-13


@pytest.mark.parametrize("dim,mhd,n", GRIDS, ids=IDS)
def test_negative_pressure_with_zero_floor(dim, mhd, n):
    gw = 3 if mhd else 2
    ini, U0, (k, j, i) = _state(dim, mhd, n, gw)
    ini = ini.replace("[hydro]", "[hydro]\nsmallc=0.0")
    U0[:5 if U0.shape[0] > 4 else 4] *= 0.1  # densities below a half
    U0[5:] *= 0.3
    U0[1, k, j - 3:j + 3, i - 3:i + 3] -= 0.3  # negative pressures
    p = ek.params_from_ini(ini)
    assert p.smallc == 0.0 and p.smallp == 0.0
    (Ue, de), (Uf, df) = _both(ini, U0, gw, dim, 1)
    assert np.array_equal(np.isnan(Ue), np.isnan(Uf))
    assert np.max(np.abs(df / de - 1)) <= 1e-13
    ok = ~np.isnan(Ue)
    assert np.max(rel_linf(np.where(ok, Uf, 0.0), np.where(ok, Ue, 0.0))[[0, 1]]) <= 1e-11
