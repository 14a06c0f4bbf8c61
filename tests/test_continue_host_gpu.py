"""Steps that go on after gasatt_sim_run_host: the same as those of a new cell
loaded with the state and fields that the call left behind."""
import ctypes

import numpy as np
import pytest

from gasatt import _lib
from gasatt._lib import check, lib
from gasatt.sim import Batch, Sim, births, config

pytestmark = pytest.mark.gpu

NR, NZ, D, C = 32, 64, 5e-6, 299792458.0


def cell(precision, ctx=None):
    # no gas: a collision would depend on the step's number, which differs
    return Sim(config(NR, NZ, D, 1e-14, 0.0, precision=precision, capacity=8000, seed=7, sort_period=6, FN=1e3), ctx=ctx)


def after_host_call(precision, nsteps, step):
    """(state after run_host and `step`, state of a new cell after `step`)"""
    r, z, ur, ut, uz, _ = births(1500, 8.0, NZ * D, seed=3, sigma_r=30e-6, Rp=0.98 * NR * D)
    n0, cap = r.size, 8000
    sim = cell(precision)
    g = np.sqrt(1 + (ur**2 + ut**2 + uz**2) / C**2)
    io = np.zeros((6, cap))
    io[:, :n0] = r, 0 * r, z, ur / g, ut / g, uz / g
    n, p = ctypes.c_int64(n0), io.ctypes.data
    check(sim.ctx.handle, lib.gasatt_sim_run_host(sim.h, ctypes.c_void_p(p), ctypes.c_void_p(p + 3 * cap * 8),
                                                  ctypes.byref(n), cap, nsteps))
    st = sim.read()
    new = cell(precision, sim.ctx)
    new.load(*(st[k] for k in ("r", "z", "ur", "ut", "uz", "id")))
    new.set_fields(*sim.fields())
    out = []
    for s in (sim, new):
        step(s)
        a = s.read()
        o = np.argsort(a["id"])
        out.append([a[k][o] for k in ("id", "r", "z", "ur", "ut", "uz")] + list(s.fields()) + list(s.current()))
    sim.close()
    new.close()
    return out


def by_batch(sim):
    b = Batch([sim], sort_period=6)
    b.step(5)
    b.close()


STEPS = [lambda s: s.step(0), lambda s: s.step(1), lambda s: s.step(14), by_batch]


@pytest.mark.parametrize("step", STEPS)
@pytest.mark.parametrize("nsteps", [1, 4, 5])
def test_fp64(nsteps, step):
    got, want = after_host_call(_lib.FP64, nsteps, step)
    assert np.abs(want[-1]).max() > 0
    for g, w in zip(got, want):
        np.testing.assert_array_equal(g, w)


@pytest.mark.parametrize("step", STEPS)
@pytest.mark.parametrize("nsteps", [1, 4, 5])
def test_fp32(nsteps, step):
    """The stochastic rounding draws differ, so the momenta differ by float
    roundings (6e-8 of c a step at most, so 1e-5 of 0.17 c in 14 steps with
    room) and the positions by what these move an electron: far less than the
    half drift of 0.05 cells that a missing prologue costs."""
    got, want = after_host_call(_lib.FP32_SPLIT, nsteps, step)
    np.testing.assert_array_equal(got[0], want[0])
    for k in (1, 2):
        assert np.abs(got[k] - want[k]).max() < 1e-4 * D
    for k in (3, 4, 5):
        assert np.abs(got[k] - want[k]).max() < 1e-5 * 0.17 * C
    for g, w in zip(got[6:], want[6:]):
        assert np.abs(w).max() > 0
        assert np.abs(g - w).max() < 1e-4 * np.abs(w).max()
