"""Steps taken several per graph launch give what single ones give: step counts
around the ten of a graph, sorts and ion pushes in between, odd starts."""
import numpy as np
import pytest

from gasatt import _lib
from gasatt.dropin import Context
from gasatt.sim import Batch, Sim, births, config

pytestmark = pytest.mark.gpu

NR, NZ, D = 32, 64, 5e-6


def make(precision, sort, ions, ctx=None, seed=3):
    cfg = config(NR, NZ, D, 1e-14, 200.0, precision=precision, capacity=20000, seed=seed, sort_period=sort,
                 ion_capacity=20000 if ions else 0, ion_subcycle=ions or 50)
    sim = Sim(cfg, ctx=ctx)
    sim.load(*births(1500, 8.0, NZ * D, seed=seed, sigma_r=30e-6, Rp=0.98 * NR * D))
    return sim


def state(sim):
    st, d = sim.read(), sim.diag()
    a = st["r"] >= 0
    o = np.argsort(st["id"][a])
    i = sim.read_ions()
    p = np.argsort(i["id"])
    return [st[k][a][o] for k in ("id", "r", "z", "ur", "ut", "uz")] + [i["r"][p], i["uz"][p]] + list(sim.fields()) + \
        list(sim.current()) + [np.array([d[k] for k in ("n_alive", "n_ionizations", "n_elastic", "steps", "n_ions")])]


@pytest.mark.parametrize("precision", [_lib.FP64, _lib.FP32_SPLIT])
@pytest.mark.parametrize("sort,ions,calls", [(0, 0, (10, 21)), (10, 0, (31,)), (12, 0, (9, 11, 12)), (20, 15, (45,)),
                                             (30, 10, (3, 37)), (5, 0, (22,))])
def test_same_as_single_steps(precision, sort, ions, calls):
    one, many = make(precision, sort, ions), make(precision, sort, ions)
    l0 = many.ctx.launches
    for n in calls:
        many.step(n)
        for _ in range(n):
            one.step(1)
    for a, b in zip(state(many), state(one)):
        np.testing.assert_array_equal(a, b)
    assert many.ctx.launches - l0 > sum(calls)
    ctx = Context(0)
    sims = [make(precision, sort, ions, ctx), make(_lib.FP32_SPLIT, sort, 0, ctx, seed=4)]
    batch = Batch(sims, sort_period=sort)
    for n in calls:
        batch.step(n)
    for a, b in zip(state(sims[0]), state(one)):
        np.testing.assert_array_equal(a, b)
    batch.close()
    for s in (one, many, *sims):
        s.close()
