"""electricmagneticfield6 at the edges of what it takes: grids of millions of rows."""
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
