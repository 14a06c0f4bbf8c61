"""The particle pass's deposit boxes where they can go wrong: grids narrower
and wider than a box, populations near the axis and over the whole radius,
population sizes around a block, a chunk and several chunks per block."""
import numpy as np
import pytest

import pyoracle as O
from _cases import close, grid_fields
from gasatt import _lib
from gasatt.sim import Sim, births, config

pytestmark = pytest.mark.gpu

D = 5e-6


def population(n, nr, nz, spread, seed):
    """n electrons: births near the axis, or the same moved to radii over the whole grid."""
    r, z, ur, ut, uz, ids = births((n + 1) // 2, 8.0, nz * D, seed=seed, sigma_r=12e-6, Rp=0.98 * nr * D)
    if spread:
        r = np.random.default_rng(seed).uniform(0, 0.98 * nr * D, r.size)
    return tuple(a[:n] for a in (r, z, ur, ut, uz, ids))


# n_r below, at and above the box's 256 columns; sizes 1, a block's edge, a
# chunk's edge for every block (444 x 256), several chunks per block
@pytest.mark.parametrize("nr,nz,n,spread", [
    (3, 5, 1, False), (31, 40, 257, True), (255, 12, 4609, True), (256, 12, 20_000, False),
    (257, 9, 20_001, True), (300, 8, 113_665, True), (600, 6, 120_000, False), (40, 700, 250_000, True)])
def test_fp64_pass_matches_oracle(tables, nr, nz, n, spread):
    parts = population(n, nr, nz, spread, seed=n)
    cfg = config(nr, nz, D, 1e-14, 100.0, precision=_lib.FP64, capacity=2 * n + 100, seed=3, sort_period=2)
    flds = grid_fields(nr, nz, np.random.default_rng(8), E0=3e6, H0=2e3)
    flds[0][:, 0] = 0; flds[0][:, -1] = 0; flds[1][-1, :] = 0
    sim = Sim(cfg, tables=tables)
    sim.load(*parts)
    sim.set_fields(*flds)
    sim.step(3)
    orc = O.Sim(cfg, tables, cap=cfg.capacity)
    orc.load(*parts)
    orc.Er[:], orc.Ez[:], orc.H[:] = flds
    orc.prologue()
    for _ in range(3):
        orc.step()
    got = sim.read()
    r, z, ur, ut, uz, ids, alive = orc.state_rz()
    a, g = alive.astype(bool), got["r"] >= 0
    want, have = np.argsort(ids[a]), np.argsort(got["id"][g])
    assert np.array_equal(ids[a][want], got["id"][g][have])
    # 1e-12 of each quantity's largest value: 64-bit rounding through three steps
    for k, w in (("r", r), ("z", z), ("ur", ur), ("ut", ut), ("uz", uz)):
        close(got[k][g][have], w[a][want], 1e-12, k)
    for f, w, k in zip(sim.fields() + sim.current(), (orc.Er, orc.Ez, orc.H, orc.jr, orc.jz),
                       ("Er", "Ez", "H", "jr", "jz")):
        close(f, w, 1e-12, k)
    d = sim.diag()
    assert (d["n_ionizations"], d["n_elastic"], d["n_excitation"], d["n_null"], d["n_lost_wall"]) == \
        tuple(int(c) for c in orc.counters[:5])
    sim.close()


# populations of one warp, around a block, around one chunk per block (592 x
# 256 and 592 x 1792 electrons) and between; at 100 Torr 2% of the electrons are
# collision candidates in each step, for idle and busy blocks alike
@pytest.mark.parametrize("nr,nz,n,spread", [
    (16, 20, 31, False), (16, 20, 257, False), (64, 64, 30_001, False), (64, 64, 151_553, False),
    (64, 300, 400_000, False), (64, 300, 1_060_865, False),
    # grids wider than a box: near its columns, one row per chunk, many rows per chunk
    (257, 9, 20_001, True), (600, 6, 120_000, False), (600, 60, 30_000, True), (1100, 20, 300_000, True)])
def test_fp32_chunk_choice_changes_no_bit(nr, nz, n, spread):
    """The chunk chosen from the population and fixed chunks give the same state, fields and counts."""
    parts = population(n, nr, nz, spread, seed=n)
    flds = grid_fields(nr, nz, np.random.default_rng(8), E0=3e6, H0=2e3)
    flds[0][:, 0] = 0; flds[0][:, -1] = 0; flds[1][-1, :] = 0
    ref = None
    for chunk in (0, 256, 1792):
        cfg = config(nr, nz, D, 1e-14, 100.0, precision=_lib.FP32_SPLIT, capacity=n + n // 4 + 100, seed=3,
                     sort_period=3)
        cfg.pass_chunk = chunk
        sim = Sim(cfg)
        sim.load(*parts)
        sim.set_fields(*flds)
        sim.step(7)
        d, st = sim.diag(), sim.read()
        a = st["r"] >= 0
        o = np.argsort(st["id"][a], kind="stable")
        got = [st[k][a][o] for k in ("id", "r", "z", "ur", "ut", "uz")] + list(sim.fields()) + list(sim.current())
        got.append(np.array([d[k] for k in ("n_alive", "n_ionizations", "n_elastic", "n_excitation", "n_null",
                                            "n_lost_wall", "collision_loss_ev")]))
        sim.close()
        if ref is None:
            ref = got
            assert d["n_alive"] > 0
        for x, y in zip(got, ref):
            np.testing.assert_array_equal(x, y)
