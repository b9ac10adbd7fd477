"""Gas without pressure (smallc = 0): the FP64 FMA build against the exact build.
Where such gas expands the star state is 0 / 0, and the upwind state is the flux."""

import numpy as np
import pytest

import euler_kokkos_gb300 as ek
from euler_kokkos_gb300 import problems as P
from helpers import interior, rel_linf

pytestmark = pytest.mark.gpu


# 2D tile kernel, 2D and 3D passes
@pytest.mark.parametrize("dim,n", [(2, (40, 24, 1)), (2, (520, 512, 1)), (3, (20, 18, 12))])
@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_cold_expansion(dim, n, sign):
    ini, U0 = P.smooth_random(dim=dim, nx=n[0], ny=n[1], nz=n[2], seed=9, bc=(2,) * 6, nsteps=3)
    ini = ini.replace("[hydro]", "[hydro]\nsmallc=0.0")
    # velocities that grow along each axis, of short significands: the pressure of E = rho u^2 / 2 is exactly zero
    axes = np.meshgrid(*[np.arange(m) for m in U0.shape[1:]], indexing="ij")
    vel = [sign * (1.0 + (a // 8 % 8) / 16.0) for a in axes[::-1]]
    U0[0] = 1.0
    for d in range(dim):
        U0[2 + d] = vel[d]
    U0[1] = 0.5 * sum(v ** 2 for v in vel[:dim])
    out = []
    for exact in (1, 0):
        with ek.Solver(ek.params_from_ini(ini, exact_fp=exact)) as s:
            s.set_state(U0)
            s.run(1, allow_nonfinite=True)
            out.append((interior(s.get_state(), 2, dim), s.dt_history()))
    (Ue, de), (Uf, df) = out
    assert np.isfinite(Ue).mean() > 0.5
    assert np.array_equal(np.isfinite(Ue), np.isfinite(Uf))
    ok = np.isfinite(Ue)
    assert np.max(rel_linf(np.where(ok, Uf, 0.0), np.where(ok, Ue, 0.0))[[0, 1]]) <= 1e-11
    assert np.max(np.abs(df / de - 1)) <= 1e-13
