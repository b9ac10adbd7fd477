"""The kernels' choices by grid: sizes at the edges of tiles and blocks and on
both sides of the lines between them, exact build against the oracle (bitwise)
and FP64 FMA build within its tolerances."""

import numpy as np
import pytest

import eko
import euler_kokkos_gb300 as ek
from euler_kokkos_gb300 import problems as P
from helpers import interior, rel_linf

pytestmark = pytest.mark.gpu

# 2D hydro: 8 x 8 tiles up to six per SM (240^2: 900 tiles on 152 SMs), 16 x 16 above (248 x 240: 930), passes from
# 2^18 cells (512^2)
CASES = [(2, False, s) for s in [(2, 2, 1), (8, 8, 1), (9, 7, 1), (17, 16, 1), (240, 240, 1), (248, 240, 1), (511, 513, 1),
                                 (512, 512, 1)]]
# 2D MHD: 8 x 8 tiles up to three per SM (170 x 160: 440), then passes
CASES += [(2, True, s) for s in [(3, 3, 1), (8, 9, 1), (17, 8, 1), (170, 160, 1), (171, 178, 1)]]
# 3D: passes; blocks of 128 threads
CASES += [(3, False, s) for s in [(2, 2, 2), (16, 16, 33), (17, 33, 9), (127, 2, 3)]]
CASES += [(3, True, s) for s in [(3, 3, 3), (16, 8, 21), (33, 9, 14), (129, 3, 4)]]


@pytest.mark.parametrize("dim,mhd,n", CASES, ids=["%s%dd_%dx%dx%d" % ("mhd" if m else "hydro", d, *n) for d, m, n in CASES])
def test_tiles_match_the_oracle(dim, mhd, n):
    ini, U0 = P.smooth_random(dim=dim, mhd=mhd, nx=n[0], ny=n[1], nz=n[2], seed=sum(n), bc=(1, 2, 3, 3, 2, 1), nsteps=3)
    p = eko.params_from_ini(ini)
    o = eko.Oracle(p, U0)
    dts = o.run(3)
    ref = interior(o.state(), p.gw, dim)
    for exact in (1, 0):
        with ek.Solver(ek.params_from_ini(ini, exact_fp=exact)) as s:
            s.set_state(U0)
            assert s.run(3) == 3
            U, d = interior(s.get_state(), p.gw, dim), s.dt_history()
        if exact:
            assert np.array_equal(U, ref) and np.array_equal(d, dts)
        else:
            assert np.max(rel_linf(U, ref)[[0, 1]]) <= 1e-11 and np.max(np.abs(d / dts - 1)) <= 1e-13


# 2D marches: strips of 28 columns, four runs of rows per CTA
ROW_SIZES = [(2, 2), (27, 5), (28, 8), (29, 9), (57, 3), (5, 131), (84, 33)]


@pytest.mark.parametrize("more", [0, 12], ids=["one row", "longer runs"])
def test_marching_warps_match_the_oracle(more):
    """An ensemble's instances run the march: bitwise in the exact build, with runs of one row (few cells) and longer
    ones (the added instances)."""
    cases = [P.smooth_random(dim=2, nx=x, ny=y, seed=x + y, bc=(1, 2, 3, 3, 1, 1) if x % 2 else (3, 3, 2, 1, 1, 1), nsteps=3)
             for x, y in ROW_SIZES + more * [(128, 130)]]
    with ek.Ensemble([ek.params_from_ini(ini, exact_fp=1) for ini, _ in cases]) as e:
        for i, (_, U0) in enumerate(cases):
            e.set_state(i, U0)
        e.run(3)
        e.synchronize()
        for i, (ini, U0) in enumerate(cases[:len(ROW_SIZES) + 1]):
            o = eko.Oracle(eko.params_from_ini(ini), U0)
            dts = o.run(3)
            assert np.array_equal(e.dt_history(i), dts), i
            assert np.array_equal(interior(e.get_state(i), 2, 2), interior(o.state(), 2, 2)), i


@pytest.mark.parametrize("prec", [ek.EK_PREC_FP64, ek.EK_PREC_MIXED], ids=["fp64", "mixed"])
def test_runs_of_rows_do_not_show(prec):
    """A cell's result does not depend on the rows per run: the same instances beside few and many others, bitwise, and
    no mass is lost at the ends of runs."""
    cases = [P.smooth_random(dim=2, nx=x, ny=y, seed=x + y, bc=(3, 3, 3, 3, 1, 1), nsteps=20) for x, y in ROW_SIZES + [(100, 120)]]
    out = []
    for more in (0, 40):
        with ek.Ensemble([ek.params_from_ini(ini, precision=prec) for ini, _ in cases + more * cases[-1:]]) as e:
            for i, (_, U0) in enumerate(cases + more * cases[-1:]):
                e.set_state(i, U0)
            e.run(20)
            e.synchronize()
            out.append([(e.get_state(i), e.dt_history(i)) for i in range(len(cases))])
    for (U, d), (V, f), (_, U0) in zip(*out, cases):
        assert np.array_equal(U, V) and np.array_equal(d, f)
        # 20 updates of n cells, each rounded to half an ulp of about its value
        n, m = interior(U, 2, 2)[0].size, interior(U0, 2, 2)[0].sum()
        ulp = 2.0 ** -52 if prec == ek.EK_PREC_FP64 else 2.0 ** -23
        assert abs(interior(U, 2, 2)[0].sum() / m - 1) <= 20 * 8 * ulp / np.sqrt(n) + 8 * ulp


@pytest.mark.parametrize("n", ROW_SIZES + [(400, 301)])
def test_mixed_marching_warps(n):
    ini, U0 = P.smooth_random(dim=2, nx=n[0], ny=n[1], seed=sum(n), bc=(1, 2, 3, 3, 1, 1), nsteps=3)
    o = eko.Oracle(eko.params_from_ini(ini), U0)
    o.run(3)
    ref = interior(o.state(), 2, 2)
    with ek.Solver(ek.params_from_ini(ini, precision=ek.EK_PREC_MIXED)) as s:
        s.set_state(U0)
        assert s.run(3) == 3
        U = interior(s.get_state(), 2, 2)
    for v in (0, 1):  # density and energy, the mixed form's bound
        assert np.abs(U[v] - ref[v]).sum() / np.abs(ref[v]).sum() <= 1e-5


# mixed 2D MHD: 8 x 8 tiles up to seven per SM (264 x 256: 1056), 16 x 16 above (272 x 266: 1156)
@pytest.mark.parametrize("n", [(3, 3), (8, 9), (17, 8), (33, 25), (264, 256), (272, 266)])
def test_mixed_mhd2d_tiles(n):
    ini, U0 = P.smooth_random(dim=2, mhd=True, nx=n[0], ny=n[1], seed=sum(n), bc=(1, 2, 3, 3, 1, 1), nsteps=3)
    o = eko.Oracle(eko.params_from_ini(ini), U0)
    o.run(3)
    ref = interior(o.state(), 3, 2)
    with ek.Solver(ek.params_from_ini(ini, precision=ek.EK_PREC_MIXED)) as s:
        s.set_state(U0)
        assert s.run(3) == 3
        U = interior(s.get_state(), 3, 2)
    for v in (0, 1):  # density and energy, the mixed form's bound
        assert np.abs(U[v] - ref[v]).sum() / np.abs(ref[v]).sum() <= 1e-5


def test_mixed_mhd2d_repair_in_16x16_tiles():
    # the repair test's low-beta blast (tests/test_gpu_mhd2d.py) on a grid of 16 x 16 tiles
    ini, U0 = P.mhd_blast_2d(n=272, nsteps=30)
    with ek.Solver(ek.params_from_ini(ini, precision=ek.EK_PREC_MIXED)) as s, ek.Solver(ek.params_from_ini(ini)) as d:
        s.set_state(U0)
        d.set_state(U0)
        assert s.run(30) == d.run(30) == 30
        U, V = interior(s.get_state(), 3, 2), interior(d.get_state(), 3, 2)
    for v in (0, 1):
        assert np.abs(U[v] - V[v]).sum() / np.abs(V[v]).sum() <= 1e-5


@pytest.mark.parametrize("mhd", [False, True], ids=["hydro", "mhd"])
def test_slabs_do_not_show(mhd):
    """A grid whose workspace takes several slabs of passes (the trace of 262144-cell planes, 1 GiB a slab): the mixed
    form's tile kernels are the independent result, within the mixed form's tolerance, and symmetric halves of a
    z-periodic state stay equal bit for bit across the slab boundaries."""
    ini, U0 = P.smooth_random(dim=3, mhd=mhd, nx=512, ny=512, nz=10, seed=3, nsteps=2)
    gw = 3 if mhd else 2
    k = np.arange(10 + 2 * gw)
    U0 = np.ascontiguousarray(U0[:, (k - gw) % 2 + gw])  # period two in z
    if mhd:
        U0[7] = 0.0
    with ek.Solver(ek.params_from_ini(ini)) as s, ek.Solver(ek.params_from_ini(ini, precision=ek.EK_PREC_MIXED)) as m:
        s.set_state(U0)
        m.set_state(U0)
        assert s.run(2) == m.run(2) == 2
        U, V = interior(s.get_state(), gw, 3), interior(m.get_state(), gw, 3)
    for z in range(2, 10):
        assert np.array_equal(U[:, z], U[:, z % 2])
    assert np.abs(U[0] - V[0]).sum() / np.abs(U[0]).sum() <= 1e-5
