"""The kernels' tile and chunk choices: grids at the edges of the tiles and on
both sides of the lines between them, exact build against the oracle (bitwise)
and FP64 FMA build within its tolerances."""

import numpy as np
import pytest

import eko
import euler_kokkos_gb300 as ek
from euler_kokkos_gb300 import problems as P
from helpers import interior, rel_linf

pytestmark = pytest.mark.gpu

# 2D: 8 x 8 tiles up to six per SM (240^2: 900 tiles on 152 SMs), 16 x 16 above (248 x 240: 930)
CASES = [(2, False, s) for s in [(2, 2, 1), (8, 8, 1), (9, 7, 1), (17, 16, 1), (240, 240, 1), (248, 240, 1), (257, 241, 1)]]
# 2D MHD: 8 x 8 up to three per SM (170 x 165: 462 tiles, 160 x 160: 400), 16 x 8 up to three (240 x 240: 450), then 16 x 16
CASES += [(2, True, s) for s in [(3, 3, 1), (8, 9, 1), (17, 8, 1), (160, 160, 1), (170, 165, 1), (240, 240, 1), (250, 243, 1)]]
# 3D: planes per CTA from the grid (kchunk 0)
CASES += [(3, False, s) for s in [(2, 2, 2), (16, 16, 33), (17, 33, 9)]]
CASES += [(3, True, s) for s in [(3, 3, 3), (16, 8, 21), (33, 9, 14)]]


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
