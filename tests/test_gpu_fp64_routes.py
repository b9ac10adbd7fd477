"""FP64 3D steps: in passes, or by the tile kernels where the planes per CTA are
given.  The FMA build's tile kernels against the oracle, by the tolerances of the
passes (test_gpu_tiles.py)."""

import numpy as np
import pytest

import eko
import euler_kokkos_gb300 as ek
from euler_kokkos_gb300 import problems as P
from helpers import interior, rel_linf

pytestmark = pytest.mark.gpu

# kernels of a step: hydro prims, trace, flux, update; MHD prims, E, trace, flux, update; tiles: one, or trace and update
# (and the CFL before the first step)
LAUNCHES = {(False, 0): 4, (False, 8): 1, (True, 0): 5, (True, 8): 2}


@pytest.mark.parametrize("kchunk", [0, 8])
@pytest.mark.parametrize("mhd,riemann", [(False, "hllc"), (False, "approx"), (False, "llf"), (True, "hlld"), (True, "llf"),
                                         (True, "hll")])
@pytest.mark.parametrize("n", [(17, 16, 9), (36, 19, 21)])
def test_tile_kernels_run_when_asked_for(mhd, riemann, kchunk, n):
    ini, U0 = P.smooth_random(dim=3, mhd=mhd, nx=n[0], ny=n[1], nz=n[2], seed=sum(n), bc=(1, 2, 3, 3, 2, 1), nsteps=4,
                              riemann=riemann)
    o = eko.Oracle(eko.params_from_ini(ini), U0)
    dts = o.run(4)
    gw = 3 if mhd else 2
    ref = interior(o.state(), gw, 3)
    for exact in (1, 0):
        with ek.Solver(ek.params_from_ini(ini, exact_fp=exact, kchunk=kchunk)) as s:
            s.set_state(U0)
            assert s.run(1) == 1
            before = s.launch_count()
            assert s.run(3) == 3
            assert s.launch_count() - before == 3 * LAUNCHES[mhd, kchunk]
            U, d = interior(s.get_state(), gw, 3), s.dt_history()
        if exact:
            assert np.array_equal(U, ref) and np.array_equal(d, dts)
        else:
            assert np.max(rel_linf(U, ref)[[0, 1]]) <= 1e-11 and np.max(np.abs(d / dts - 1)) <= 1e-13
