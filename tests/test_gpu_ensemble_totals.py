"""Totals of an ensemble whose instances end at different steps: they are those
of the state that get_state returns, whichever buffer an instance stopped in."""

import numpy as np
import pytest

import euler_kokkos_gb300 as ek
from euler_kokkos_gb300 import problems as P
from helpers import interior

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [ek.EK_PREC_FP64, ek.EK_PREC_MIXED], ids=["fp64", "mixed"])
def test_totals_of_finished_instances(prec):
    ini, U0 = P.implode_2d(n=24, nsteps=100)
    ends = ["0.004", "0.006", "1e30"]
    # open sides: the totals change with every step
    open_ = ini
    for side in ("xmin", "xmax", "ymin", "ymax"):
        open_ = open_.replace("boundary_type_%s=1" % side, "boundary_type_%s=2" % side)
    assert open_ != ini
    params = [ek.params_from_ini(open_.replace("tEnd=1e30", "tEnd=" + e), precision=prec) for e in ends]
    U0[0] *= np.linspace(1.0, 1.5, U0.shape[-1])
    U0[2] = 0.3 * U0[0]
    U0[1] += 0.5 * U0[2] ** 2 / U0[0]
    with ek.Ensemble(params) as e:
        for i in range(3):
            e.set_state(i, U0)
        e.run(20)
        for _ in range(2):  # an even and an odd number of steps launched after the instances' last
            e.run(1)
            e.synchronize()
            assert e.time(0)[2] < 20 and e.time(1)[2] < 20
            tot = e.totals()
            for i in range(3):
                U = interior(e.get_state(i), 2, 2)
                for v in (0, 1):  # integrals: sums of 576 FP64 values in another order
                    assert abs(tot[i, v] / (U[v].sum() * params[i].dx * params[i].dy) - 1) <= 1e-13, (i, v)
