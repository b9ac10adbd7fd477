"""Clock and state reads: more solvers than page-locked clock slots (128), and
threads reading the instances of one ensemble, which share a staging buffer."""

import threading

import numpy as np
import pytest

import euler_kokkos_gb300 as ek
from euler_kokkos_gb300 import problems as P

pytestmark = pytest.mark.gpu


def test_more_solvers_than_clock_slots():
    ini, U0 = P.implode_2d(n=8, nsteps=4)
    p = ek.params_from_ini(ini)
    for _ in range(2):  # the slots come back
        solvers = [ek.Solver(p) for _ in range(131)]
        for s in solvers:
            s.set_state(U0)
            s.next_iteration()
            s.run(2)
        assert {(s.m_t, s.m_iteration) for s in solvers} == {(solvers[0].m_t, 3)}
        assert all(np.array_equal(s.get_state(), solvers[0].get_state()) for s in solvers)
        for s in solvers:
            s.close()


def test_threads_read_an_ensemble():
    cases = P.kh_ensemble(n_inst=8, sizes=(16, 40, 64), nsteps=4)
    with ek.Ensemble([ek.params_from_ini(ini, precision=ek.EK_PREC_MIXED) for ini, _ in cases]) as e:
        for i, (_, U0) in enumerate(cases):
            e.set_state(i, U0)
        e.run(4)
        ref = [e.get_state(i) for i in range(8)]
        got = [[] for _ in range(8)]

        def read(i):
            got[i] = [(e.get_state(i), e.time(i)[2]) for _ in range(20)]

        threads = [threading.Thread(target=read, args=(i,)) for i in range(8)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert all(len(g) == 20 and all(np.array_equal(U, ref[i]) and it == 4 for U, it in g) for i, g in enumerate(got))
