"""FP64 solvers on a device with little memory left: the workspace of the passes
gives way, in shorter slabs or to the tile kernels, and the results stay."""

import contextlib

import numpy as np
import pytest

import euler_kokkos_gb300 as ek
from euler_kokkos_gb300 import problems as P

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

MB = 1 << 20


@contextlib.contextmanager
def _left(nbytes):
    """All but about nbytes of the device's memory is taken (a failing cudaMalloc is an ordinary error)."""
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    held = []
    try:
        try:
            held.append(torch.empty(torch.cuda.mem_get_info()[0] - nbytes, dtype=torch.uint8, device="cuda"))
        except torch.OutOfMemoryError:
            pytest.skip("the device's memory cannot be taken")
        if abs(torch.cuda.mem_get_info()[0] - nbytes) > 4 * MB:
            pytest.skip("the device's free memory is not the test's to set")
        yield
    finally:
        held.clear()
        torch.cuda.empty_cache()


def _state(mhd, dim):
    n = (64, 64, 64) if mhd and dim == 3 else (128, 128, 64) if dim == 3 else (1024, 1024, 1)
    ini, U0 = P.smooth_random(dim=dim, mhd=mhd, nx=n[0], ny=n[1], nz=n[2], seed=7, nsteps=3)
    return ek.params_from_ini(ini), U0


def _run(s):
    before = s.launch_count()
    assert s.run(2) == 2
    return (s.launch_count() - before) // 2, s.get_state(), s.dt_history()


# MB left beside the states; one slab takes 445 MB (hydro 3D), 236 (2D), 186 (MHD 3D), 464 (MHD 2D), of one plane or row 20, 1,
# 45, 103
@pytest.mark.parametrize("dim,mhd,room", [(3, False, 160), (3, False, 24), (2, False, 100), (2, False, 16), (3, True, 110),
                                          (2, True, 200), (2, True, 60)])
def test_workspace_in_shorter_slabs(dim, mhd, room):
    p, U0 = _state(mhd, dim)
    with ek.Solver(p) as s:
        s.set_state(U0)
        launches, U, d = _run(s)
    state = 2 * U0.nbytes
    with _left(state + room * MB):
        with ek.Solver(p) as s:
            s.set_state(U0)
            few, V, f = _run(s)
    # the passes of more slabs, or a tile kernel (and, 2D MHD, its CFL kernel before the first step)
    assert few > launches or few <= 1
    # every value is computed as before, whichever slab it is in; the tile kernels' may differ by rounding
    if few > 1:
        assert np.array_equal(U, V) and np.array_equal(d, f)
    else:
        assert np.max(np.abs(U - V)) <= 1e-11 and np.max(np.abs(d / f - 1)) <= 1e-13


def test_staging_beside_the_workspace():
    """A row-major state goes through a staging buffer, allocated when it is first needed."""
    p, U0 = _state(False, 3)
    R = np.ascontiguousarray(np.transpose(U0, (3, 2, 1, 0)))
    out = []
    for little in (False, True):
        with ek.Solver(p) as s:
            s.set_state(U0)
            assert s.run(1) == 1
            with _left(20 * MB) if little else contextlib.nullcontext():
                s.set_state(R, layout=ek.EK_LAYOUT_RIGHT)  # 45 MB
                out.append(_run(s))
                assert np.array_equal(np.transpose(s.get_state(layout=ek.EK_LAYOUT_RIGHT), (3, 2, 1, 0)), out[-1][1])
    assert out[1][0] > out[0][0]
    assert np.array_equal(out[0][1], out[1][1]) and np.array_equal(out[0][2], out[1][2])


@pytest.mark.parametrize("mhd", [False, True], ids=["hydro", "mhd"])
def test_what_does_not_fit_leaves_the_solver_as_it_was(mhd):
    """The staging buffer fits in no way: the call is refused, and the solver goes on."""
    n = (64, 64, 64) if mhd else (96, 96, 96)
    ini, U0 = P.smooth_random(dim=3, mhd=mhd, nx=n[0], ny=n[1], nz=n[2], seed=7, nsteps=3)
    p = ek.params_from_ini(ini, kchunk=4)  # tile kernels: no workspace to give way in hydro
    with ek.Solver(p) as s:
        s.set_state(U0)
        assert s.run(1) == 1
        U = s.get_state()
        with _left(4 * MB):
            with pytest.raises(ek.EkError) as err:
                s.get_state(layout=ek.EK_LAYOUT_RIGHT)
            assert err.value.status == ek.EK_ERR_NO_MEMORY
            assert np.array_equal(s.get_state(), U)
            assert s.run(1) == 1


def test_gravity_field_beside_the_workspace():
    ini, U0 = P.rayleigh_taylor(dim=3, nx=96, ny=96, nz=96, nsteps=3)
    p = ek.params_from_ini(ini)
    G = np.zeros((3,) + U0.shape[1:])
    G[2] = -0.1 * (1.0 + 0.1 * np.cos(np.arange(U0.shape[1]))[:, None, None])
    out = []
    for little in (False, True):
        with ek.Solver(p) as s:
            s.set_state(U0)
            with _left(8 * MB) if little else contextlib.nullcontext():
                s.set_gravity_field(G)  # 24 MB
                out.append(_run(s))
    assert out[1][0] > out[0][0]
    assert np.array_equal(out[0][1], out[1][1]) and np.array_equal(out[0][2], out[1][2])
