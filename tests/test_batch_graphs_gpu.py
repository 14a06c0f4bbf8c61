"""A batch builds its graph of ten steps once that is worth it: its creation costs
no more in the FP64 form than its other graphs, and its steps are the same before and after."""
import time
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest
import torch

from gasatt import _lib
from gasatt.dropin import Context
from gasatt.sim import Batch, Sim, births, config

pytestmark = pytest.mark.gpu

D = 5e-6
FORMS = {"fp64": (_lib.FP64, _lib.FP64), "fp32": (_lib.FP32_SPLIT, _lib.FP32_SPLIT), "both": (_lib.FP64, _lib.FP32_SPLIT)}


def make(precision, seed, ctx, ratio=1):
    nr, nz = 24, 40
    sim = Sim(config(nr, nz, D, 1e-14, 50.0, precision=precision, capacity=30000, seed=seed, sort_period=0,
                     fdtd_ratio=ratio), ctx=ctx)
    sim.load(*births(400, 8.0, nz * D, seed=seed, sigma_r=25e-6, Rp=0.98 * nr * D))
    return sim


def state(sim):
    st, d = sim.read(), sim.diag()
    a = st["r"] >= 0
    o = np.argsort(st["id"][a])
    return [st[k][a][o] for k in ("id", "r", "z", "ur", "ut", "uz")] + list(sim.fields()) + list(sim.current()) + \
        [np.array([d[k] for k in ("n_alive", "n_ionizations", "n_elastic", "steps")])]


@pytest.mark.parametrize("sort", [0, 24])
@pytest.mark.parametrize("forms,ratio", [("fp64", 1), ("fp32", 1), ("both", 1), ("both", 2)])
def test_same_steps_before_and_after(forms, ratio, sort):
    ctx = Context(0)
    sims = [make(p, 3 + k, ctx, ratio) for k, p in enumerate(FORMS[forms])]
    batch = Batch(sims, sort_period=sort)
    for n in (1, 64, 35, 1000, 40, 7):
        batch.step(n)
    for k, p in enumerate(FORMS[forms]):
        alone = make(p, 3 + k, ctx, ratio)
        alone.step(1147)
        for a, b in zip(state(sims[k]), state(alone)):
            np.testing.assert_array_equal(a, b)
        alone.close()
    batch.close()
    for s in sims:
        s.close()


def test_creation():
    """The FP64 form's forks make its graphs of one step cost twice the FP32 form's; graphs of ten
    would cost ten forks each."""
    t = []
    for precision in FORMS["both"]:
        ctx = Context(0)
        sims = [make(precision, k, ctx) for k in range(4)]
        each = []
        for _ in range(15):
            sims[0].synchronize()
            t0 = time.perf_counter()
            Batch(sims, sort_period=20).close()
            each.append(time.perf_counter() - t0)
        t.append(min(each))
        for s in sims:
            s.close()
    assert t[0] < 1.7 * t[1]


@pytest.mark.parametrize("precision,steps", [(_lib.FP64, 2000), (_lib.FP32_SPLIT, 100)])
def test_built_while_another_thread_captures(precision, steps):
    """The steps that build the graph neither fail because another thread of the program
    captures a graph of its own, in the mode that binds all threads, nor spoil that capture."""
    ctx = Context(0)
    sims = [make(precision, k, ctx) for k in (1, 2)]
    sims[0].bind_stream(torch.cuda.Stream())
    batch = Batch(sims, sort_period=0)
    batch.step(10)
    torch.cuda.synchronize()
    x, g = torch.zeros(8, device="cuda"), torch.cuda.CUDAGraph()
    with ThreadPoolExecutor(1) as other, torch.cuda.graph(g):
        x.add_(1)
        other.submit(batch.step, steps).result()
        x.add_(1)
    g.replay()
    torch.cuda.synchronize()
    assert x.tolist() == [2.0] * 8
    batch.close()
    for k, s in zip((1, 2), sims):
        alone = make(precision, k, ctx)
        alone.step(10 + steps)
        for a, b in zip(state(s), state(alone)):
            np.testing.assert_array_equal(a, b)
        alone.close()
        s.close()
