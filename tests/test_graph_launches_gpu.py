"""How many graph launches a run takes: ten steps each where no sort, ion push or odd
start falls between; the general field update (fdtd_ratio 2) in such graphs."""
import numpy as np
import pytest
from torch.profiler import ProfilerActivity, profile

from gasatt import _lib
from test_graph_steps_gpu import NR, NZ, D, make, state
from gasatt.dropin import Context
from gasatt.sim import Batch, Sim, births, config

pytestmark = pytest.mark.gpu


def graph_launches(f):
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as p:
        f()
    return sum(e.count for e in p.key_averages() if e.key == "cudaGraphLaunch")


# launches: graphs of ten + of one + sorts (the first step sorts too where there are any)
@pytest.mark.parametrize("precision", [_lib.FP64, _lib.FP32_SPLIT])
@pytest.mark.parametrize("sort,ions,calls,launches", [
    (0, 0, (10, 21), 3 + 1), (0, 0, (9,), 9), (10, 0, (31,), 3 + 1 + 4), (5, 0, (22,), 0 + 22 + 5),
    (12, 0, (9, 11, 12), 0 + 32 + 3), (20, 15, (45,), 3 + 15 + 3), (30, 10, (3, 37), 3 + 10 + 2)])
def test_cell(precision, sort, ions, calls, launches):
    sim = make(precision, sort, ions)
    assert graph_launches(lambda: [sim.step(n) for n in calls]) == launches
    sim.close()


@pytest.mark.parametrize("precision,worth", [(_lib.FP64, 360), (_lib.FP32_SPLIT, 40)])
def test_batch(precision, worth):
    ctx = Context(0)
    sims = [make(precision, 0, 0, ctx, seed) for seed in (3, 4)]
    batch = Batch(sims, sort_period=0)
    assert graph_launches(lambda: batch.step(30)) == 30
    batch.step(2 * worth)
    assert graph_launches(lambda: batch.step(45)) == 4 + 5
    batch.close()
    for s in sims:
        s.close()


@pytest.mark.parametrize("precision", [_lib.FP64, _lib.FP32_SPLIT])
@pytest.mark.parametrize("ratio", [2, 4])
def test_general_field_update(precision, ratio):
    """Ten steps a launch, whose kernels start early, against one a launch, whose kernels do not."""
    sims = []
    for _ in range(2):
        sim = Sim(config(NR, NZ, D, 1e-14, 200.0, precision=precision, capacity=20000, seed=3, sort_period=20,
                         fdtd_ratio=ratio))
        sim.load(*births(1500, 8.0, NZ * D, seed=3, sigma_r=30e-6, Rp=0.98 * NR * D))
        sims.append(sim)
    many, one = sims
    assert graph_launches(lambda: many.step(50)) == 5 + 3
    for _ in range(50):
        one.step(1)
    for a, b in zip(state(many), state(one)):
        np.testing.assert_array_equal(a, b)
    for s in sims:
        s.close()
