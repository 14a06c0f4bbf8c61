"""gasatt_sim_run_host in the FP32 form: each collision is applied once, also
where the call's step counter and the resident one differ in parity."""
import ctypes

import numpy as np
import pytest

from gasatt import _lib
from gasatt._lib import check, lib
from gasatt.sim import Sim, births, config

pytestmark = pytest.mark.gpu

NR, NZ, D, C = 32, 64, 5e-6, 299792458.0


def run_host(precision, calls):
    r, z, ur, ut, uz, _ = births(3000, 8.0, NZ * D, seed=3, sigma_r=30e-6, Rp=0.98 * NR * D)
    n0, cap = r.size, 4 * r.size
    cfg = config(NR, NZ, D, 1e-14, 200.0, precision=precision, capacity=cap, seed=7, sort_period=3)
    sim = Sim(cfg)
    g = np.sqrt(1 + (ur**2 + ut**2 + uz**2) / C**2)
    out = []
    for steps in calls:
        io = np.zeros((6, cap))
        io[:, :n0] = r, 0 * r, z, ur / g, ut / g, uz / g
        n = ctypes.c_int64(n0)
        p = io.ctypes.data
        check(sim.ctx.handle, lib.gasatt_sim_run_host(sim.h, ctypes.c_void_p(p), ctypes.c_void_p(p + 3 * cap * 8),
                                                      ctypes.byref(n), cap, steps))
        d = sim.diag()
        k = io[:, :n.value]
        out.append((n.value, d["n_ionizations"], d["n_elastic"], k[:, np.lexsort((k[2], k[0]))]))
    sim.close()
    return out


@pytest.mark.parametrize("calls", [(8,), (7, 6, 5), (6, 8)])
def test_collisions_applied_once(calls):
    """Run to run the same, and in the first call the FP32 form takes the FP64
    form's collisions (a few in a thousand may fall on the other side of a
    branch).  Later calls number their steps, and so draw, differently in the
    two forms."""
    a, b, c = run_host(_lib.FP32_SPLIT, calls), run_host(_lib.FP32_SPLIT, calls), run_host(_lib.FP64, calls[:1])
    for x, y in zip(a, b):
        assert x[:3] == y[:3]
        np.testing.assert_array_equal(x[3], y[3])
    x, w = a[0], c[0]
    assert w[1] > 100
    for k in range(3):
        assert abs(x[k] - w[k]) <= 3 + 0.003 * w[k], (k, x[:3], w[:3])


def test_fp64_queues_survive_alternating_steps():
    """FP64 cells stepped by a batch, on their own (odd counts, with reads in
    between that apply pending collisions) and by the batch again end where
    they end alone: every queue is emptied before it is filled again."""
    from gasatt.dropin import Context
    from gasatt.sim import Batch
    ctx = Context(0)

    def make(seed):
        cfg = config(NR, NZ, D, 1e-14, 200.0, precision=_lib.FP64, capacity=20000, seed=seed, sort_period=4)
        sim = Sim(cfg, ctx=ctx)
        sim.load(*births(1500, 8.0, NZ * D, seed=seed, sigma_r=30e-6, Rp=0.98 * NR * D))
        return sim

    def state(sim):
        st, d = sim.read(), sim.diag()
        a = st["r"] >= 0
        o = np.argsort(st["id"][a])
        return [st[k][a][o] for k in ("id", "r", "z", "ur", "ut", "uz")] + list(sim.fields()) + [
            np.array([d[k] for k in ("n_alive", "n_ionizations", "n_elastic", "n_excitation", "n_null")])]

    alone = []
    for seed in (3, 4):
        sim = make(seed)
        sim.step(16)
        alone.append(state(sim))
        sim.close()
    sims = [make(3), make(4)]
    batch = Batch(sims, sort_period=4)
    for kind, n in (("batch", 3), ("own", 1), ("batch", 2), ("read", 0), ("own", 3), ("read", 0), ("batch", 1), ("own", 2),
                    ("batch", 4)):
        if kind == "batch":
            batch.step(n)
        for sim in sims:
            if kind == "own":
                sim.step(n)
            elif kind == "read":
                sim.read()
    for sim, want in zip(sims, alone):
        for g, w in zip(state(sim), want):
            np.testing.assert_array_equal(g, w)
    batch.close()
    for sim in sims:
        sim.close()

