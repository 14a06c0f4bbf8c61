"""electricmagneticfield6 at the edges of what it takes: grids of millions of rows, currents
that are not finite, many turns into a narrow wedge."""
import math

import numpy as np
import pytest
import torch

import gasatt
import pyoracle as O
from _cases import close, grid_fields, wedge_particles
from gasatt import _lib

pytestmark = pytest.mark.gpu

NAMES = ("e_pos", "e_vel", "i1_pos", "i1_vel", "i2_pos", "i2_vel", "Er", "Ez", "Hphi", "kin")


def run(args, flags):
    return gasatt.electricmagneticfield6(*[torch.tensor(a) if isinstance(a, np.ndarray) else a for a in args], flags=flags)


@pytest.mark.parametrize("nr,nz", [(1, 53 * 65535 - 1), (1, 53 * 65535), (2, 53 * 65535 + 60)])
def test_more_rows_of_tiles_than_a_grid_dimension_holds(nr, nz):
    rng = np.random.default_rng(nz)
    d = 1e-4
    Er, Ez, H = grid_fields(nr, nz, rng, E0=3e5, H0=300.0)
    e = wedge_particles(300, nr * d, nz * d, 0.1, rng, vmag=4e7)
    i = wedge_particles(20, nr * d, nz * d, 0.1, rng, vmag=2e3)
    args = (*e, *i, *i, Er, Ez, H, d, 1e-13, nr * d, nz * d, 0.1, 1e4, 5)
    got = run(args, _lib.FAITHFUL | _lib.POS_IN_CYL)
    want = O.electricmagneticfield6(*args, _lib.FAITHFUL | _lib.POS_IN_CYL)
    for g, w, k in zip(got, want, NAMES):
        # 1e-12 of the largest value, as the drop-in's own test; a coordinate of 3.5 million cells holds its
        # place in a cell, and so the weights of the gather, to 3.5e6 x 2^-52 = 8e-10 only
        close(g.cpu().numpy(), w, 1e-12 if k[-3:] == "pos" else 1e-8, k)


@pytest.mark.parametrize("r,v", [(0.0, (0, 0, 3e7)), (2e-4, (0, 0, np.nan)), (2e-4, (0, 0, np.inf)), (2e-4, (0, 0, 1e10))])
@pytest.mark.parametrize("flags", [0, _lib.FAITHFUL])
def test_currents_that_are_not_finite(r, v, flags):
    """One electron moves, on the axis (whose azimuth atan(y / x) is none) or with an impossible
    velocity, among 4094 or 4095 that rest: its current is rounded by the same rules on both sides of
    the 4096 particles from which one FMA rounds (both in units of the same power of two)."""
    nr, nz, d = 12, 20, 1e-4
    out = []
    for n in (4095, 4096):
        pos = np.tile([3.3e-4, 0.05, 1e-3], (n, 1))
        vel = np.zeros((n, 3))
        pos[7], vel[7] = (r, 0.05, 4.4e-4), v
        no = np.zeros((0, 3))
        f = [np.zeros(s, order="F") for s in ((nr, nz + 1), (nr + 1, nz), (nr, nz))]
        out.append(run((pos, vel, no, no, no, no, *f, d, 1e-14, nr * d, nz * d, 0.1, 1e4, 5), flags | _lib.POS_IN_CYL))
    for k in (6, 7, 8):
        a, b = (o[k].cpu().numpy() for o in out)
        np.testing.assert_array_equal(a, b)
    if np.isfinite(v[2]):
        assert np.abs(a).max() > 0


@pytest.mark.parametrize("flags", [0, _lib.FAITHFUL])
@pytest.mark.parametrize("PHIp", [7e-4, 1e-3, 2.9e-3, 0.1, math.pi / 2])
def test_turns_into_the_wedge_keep_the_radius(PHIp, flags):
    """Electrons at rest at any azimuth, turned into the wedge up to 4500 times.  Two half drifts
    round the radius, its inverse, the sine, the cosine, their length and the coordinates: some
    twelve roundings of 1.1e-16 with the test's own."""
    rng = np.random.default_rng(5)
    nr, nz, d, n = 12, 20, 1e-4, 2000
    rr, phi = rng.uniform(0.1, 0.9, n) * nr * d, rng.uniform(-math.pi, math.pi, n)
    pos = np.stack([rr * np.cos(phi), rr * np.sin(phi), np.full(n, 1e-3)], 1)
    no = np.zeros((0, 3))
    f = [np.zeros(s, order="F") for s in ((nr, nz + 1), (nr + 1, nz), (nr, nz))]
    got = run((pos, np.zeros((n, 3)), no, no, no, no, *f, d, 1e-13, nr * d, nz * d, PHIp, 1e4, 5), flags)[0].cpu().numpy()
    was, now = (np.hypot(*p[:, :2].T.astype(np.longdouble)) for p in (pos, got))
    assert np.abs(now / was - 1).max() < 2e-15
    az = np.arctan2(got[:, 1], got[:, 0])
    assert az.min() > -1e-12 and az.max() < PHIp + 1e-12
