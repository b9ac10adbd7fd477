"""The ways of an FP64 step against the oracle, bitwise in the exact build and by the
tolerances of test_gpu_tiles.py in the FMA build: 3D in passes, or by the tile
kernels where the planes per CTA are given; grids of several slabs; ensembles."""

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


# a little more than one slab of 1 GiB
@pytest.mark.parametrize("dim,mhd,n,slabs", [(3, False, (320, 300, 33), 2), (3, True, (203, 200, 52), 2),
                                             (2, False, (2201, 2300, 1), 2), (2, True, (1801, 1850, 1), 2)])
def test_several_slabs(dim, mhd, n, slabs):
    ini, U0 = P.smooth_random(dim=dim, mhd=mhd, nx=n[0], ny=n[1], nz=n[2], seed=sum(n), bc=(1, 2, 3, 3, 2, 1), nsteps=2)
    o = eko.Oracle(eko.params_from_ini(ini), U0)
    dts = o.run(1)
    gw = 3 if mhd else 2
    ref = interior(o.state(), gw, dim)
    for exact in (1, 0):
        with ek.Solver(ek.params_from_ini(ini, exact_fp=exact)) as s:
            s.set_state(U0)
            before = s.launch_count()
            assert s.run(1) == 1
            assert s.launch_count() - before == (2 + 3 * slabs if mhd else 4 * slabs)
            U, d = interior(s.get_state(), gw, dim), s.dt_history()
        if exact:
            assert np.array_equal(U, ref) and np.array_equal(d, dts)
        else:
            assert np.max(rel_linf(U, ref)[[0, 1]]) <= 1e-11 and np.max(np.abs(d / dts - 1)) <= 1e-13


def test_fp64_ensemble():
    """The FMA build's marching warps in FP64 (a single FP64 run takes tiles or passes)."""
    cases = [P.smooth_random(dim=2, nx=x, ny=y, seed=x + y, bc=(1, 2, 3, 3, 1, 1), nsteps=4)
             for x, y in [(2, 2), (29, 9), (57, 33), (84, 130)]]
    with ek.Ensemble([ek.params_from_ini(ini) for ini, _ in cases]) as e:
        for i, (_, U0) in enumerate(cases):
            e.set_state(i, U0)
        e.run(4)
        e.synchronize()
        for i, (ini, U0) in enumerate(cases):
            o = eko.Oracle(eko.params_from_ini(ini), U0)
            dts = o.run(4)
            ref = interior(o.state(), 2, 2)
            assert np.max(rel_linf(interior(e.get_state(i), 2, 2), ref)[[0, 1]]) <= 1e-11, i
            assert np.max(np.abs(e.dt_history(i) / dts - 1)) <= 1e-13, i
