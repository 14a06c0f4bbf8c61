"""A gas map set between steps reaches every step graph (of one step and of ten, both
state buffers) and costs less than building them; only the graphs of one step are built
again when the timing is turned on or off."""
import time

import numpy as np
import pytest

from gasatt import _lib
from gasatt._lib import lib
from gasatt.sim import Sim, births, config

pytestmark = pytest.mark.gpu

NR, NZ, D = 32, 64, 5e-6


def make(precision, sort=0, ions=0):
    sim = Sim(config(NR, NZ, D, 1e-14, 200.0, precision=precision, capacity=20000, seed=3, sort_period=sort,
                     ion_capacity=ions))
    sim.load(*births(1500, 8.0, NZ * D, seed=3, sigma_r=30e-6, Rp=0.98 * NR * D))
    return sim


def state(sim):
    st, d, i = sim.read(), sim.diag(), sim.read_ions()
    a = st["r"] >= 0
    o, p = np.argsort(st["id"][a]), np.argsort(i["id"])
    return [st[k][a][o] for k in ("id", "r", "z", "ur", "ut", "uz")] + [i["ur"][p]] + list(sim.fields()) + \
        list(sim.current()) + [np.array([d[k] for k in ("n_alive", "n_ionizations", "n_elastic", "n_null")])]


def shortest(sim, f):
    t = []
    for _ in range(15):
        sim.synchronize()
        t0 = time.perf_counter()
        f()
        t.append(time.perf_counter() - t0)
    return min(t)


@pytest.mark.parametrize("precision", [_lib.FP64, _lib.FP32_SPLIT])
@pytest.mark.parametrize("sort", [0, 20])
def test_every_graph_takes_the_map(precision, sort):
    """Ten steps per launch against one, a map set, changed and taken away in between."""
    one, many = make(precision, sort, 20000), make(precision, sort, 20000)
    n = one.cfg.gas_density
    counts = []
    for density, hot in ((None, False), (2.0, True), (0.0, True), (0.5, False), (None, False)):
        for s in (one, many):
            if density is not None or counts:
                s.set_gas_density(None if density is None else np.full((NR, NZ), density * n))
                s.set_gas_temperature(np.full((NR, NZ), 3000.0) if hot else None)
        many.step(22)
        for _ in range(22):
            one.step(1)
        for a, b in zip(state(many), state(one)):
            np.testing.assert_array_equal(a, b)
        counts.append(one.diag()["n_elastic"])
    got = np.diff([0] + counts)
    assert got[2] == 0 and got[1] > got[0] > 0 and got[4] > got[3] > 0
    one.close()
    many.close()


@pytest.mark.parametrize("precision", [_lib.FP64, _lib.FP32_SPLIT])
def test_setting_a_map_does_not_build_graphs(precision):
    """Turning the timing on and off builds the graphs of one step twice: setting a map costs a
    fraction of that."""
    sim = make(precision)
    n = np.full((NR, NZ), sim.cfg.gas_density)
    build = shortest(sim, lambda: [lib.gasatt_sim_enable_timing(sim.h, on) for on in (1, 0)])
    assert shortest(sim, lambda: sim.set_gas_density(n)) < 0.4 * build
    sim.close()


def test_timing_on_and_off_builds_the_graphs_of_one_step():
    """The FP64 form's graphs of one step cost about twice the FP32 form's (their fork); its
    graphs of ten steps would cost as much again."""
    t = []
    for precision in (_lib.FP64, _lib.FP32_SPLIT):
        sim = make(precision, 20)
        t.append(shortest(sim, lambda: [lib.gasatt_sim_enable_timing(sim.h, on) for on in (1, 0)]))
        one = make(precision, 20)
        for k in range(3):                # with the timing on, off and on again the steps are the same
            lib.gasatt_sim_enable_timing(sim.h, (k + 1) & 1)
            sim.step(12)
            one.step(12)
        for a, b in zip(state(sim), state(one)):
            np.testing.assert_array_equal(a, b)
        sim.close()
        one.close()
    assert t[0] < 2.3 * t[1]
