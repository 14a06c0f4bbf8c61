"""electricmagneticfield6 where its kernels branch: grids at the edges of the
field tiles (11 or 21 columns, 43 or 53 rows), one field launch and two per
step, odd and even step counts, both fixed-point roundings, every wedge."""
import math

import numpy as np
import pytest
import torch

import gasatt
import pyoracle as O
from _cases import close, grid_fields, wedge_particles
from gasatt import _lib

pytestmark = pytest.mark.gpu

FULL = 2 * math.pi


@pytest.mark.parametrize("nr,nz,n,steps,PHIp,flags", [
    (1, 2, 50, 1, 0.1, _lib.FAITHFUL), (10, 42, 500, 2, 0.1, _lib.FAITHFUL), (11, 43, 500, 3, 0.1, 0),
    (21, 86, 5000, 1, 0.1, _lib.FAITHFUL), (22, 53, 5000, 2, math.pi / 2, 0),
    (64, 1200, 6000, 2, 0.1, _lib.FAITHFUL), (64, 1200, 6000, 3, 0.1, 0),        # two launches per step
    (20, 50, 3000, 2, 2.0, _lib.FAITHFUL), (20, 50, 3000, 3, 2.0, 0), (20, 50, 3000, 2, FULL, 0),
    (20, 50, 3000, 2, 0.1, _lib.Q_ER_END_COPY | _lib.Q_EULER_KICK), (20, 50, 0, 3, 0.1, _lib.FAITHFUL),
    (20, 50, 700, 0, 0.1, _lib.FAITHFUL)])
def test_against_oracle(nr, nz, n, steps, PHIp, flags):
    rng = np.random.default_rng(nr + nz + n)
    d = 1e-4
    Er, Ez, H = grid_fields(nr, nz, rng, E0=3e5, H0=300.0)
    e = wedge_particles(n, nr * d, nz * d, PHIp, rng, vmag=4e7)
    i1 = wedge_particles(n // 3, nr * d, nz * d, PHIp, rng, vmag=2e3)
    i2 = wedge_particles(n // 7, nr * d, nz * d, PHIp, rng, vmag=2e3)
    e[0][:n // 40, 0] = nr * d * 0.995
    args = (*e, *i1, *i2, Er, Ez, H, d, 1e-13, nr * d, nz * d, PHIp, 1e4, 5 * steps)
    got = gasatt.electricmagneticfield6(*[torch.tensor(a) if isinstance(a, np.ndarray) else a for a in args],
                                        flags=flags | _lib.POS_IN_CYL)
    want = O.electricmagneticfield6(*args, flags | _lib.POS_IN_CYL)
    # 1e-12 of each quantity's largest value, as the drop-in's own test
    for g, w, k in zip(got, want, ("e_pos", "e_vel", "i1_pos", "i1_vel", "i2_pos", "i2_vel", "Er", "Ez", "Hphi", "kin")):
        close(g.cpu().numpy(), w, 1e-12, k)


@pytest.mark.parametrize("n,steps", [(68000, 9), (67742, 12), (67743, 10), (70000, 35)])
def test_sorted_particles(n, steps):
    """From 100,000 particles (n + n / 3 + n / 7) and ten steps on the particles
    are sorted by cell, and again after 25 steps: electrons that leave before
    and after a sort, order and energies as without it."""
    rng = np.random.default_rng(n + steps)
    d, nr, nz, PHIp = 1e-4, 24, 60, 0.1
    Er, Ez, H = grid_fields(nr, nz, rng, E0=3e5, H0=300.0)
    e = wedge_particles(n, nr * d, nz * d, PHIp, rng, vmag=4e7)
    i1 = wedge_particles(n // 3, nr * d, nz * d, PHIp, rng, vmag=2e3)
    i2 = wedge_particles(n // 7, nr * d, nz * d, PHIp, rng, vmag=2e3)
    args = (*e, *i1, *i2, Er, Ez, H, d, 1e-13, nr * d, nz * d, PHIp, 100.0, 5 * steps)
    flags = _lib.FAITHFUL | _lib.POS_IN_CYL
    got = gasatt.electricmagneticfield6(*[torch.tensor(a) if isinstance(a, np.ndarray) else a for a in args],
                                        flags=flags)
    want = O.electricmagneticfield6(*args, flags)
    # as above, times the number of steps: the rounding errors of a step add up
    for g, w, k in zip(got, want, ("e_pos", "e_vel", "i1_pos", "i1_vel", "i2_pos", "i2_vel", "Er", "Ez", "Hphi", "kin")):
        close(g.cpu().numpy(), w, 1e-12 * steps, k)
