"""A call whose device scratch cannot be allocated says so and leaves the context as good as new."""
import ctypes

import numpy as np
import pytest
import torch

import gasatt
from _cases import grid_fields, wedge_particles
from gasatt import _lib
from gasatt._lib import lib
from gasatt.dropin import default_context

pytestmark = pytest.mark.gpu


def small():
    rng = np.random.default_rng(1)
    nr, nz, d = 12, 30, 1e-4
    e = wedge_particles(500, nr * d, nz * d, 0.1, rng, vmag=4e7)
    i = wedge_particles(50, nr * d, nz * d, 0.1, rng, vmag=2e3)
    args = (*e, *i, *i, *grid_fields(nr, nz, rng), d, 1e-13, nr * d, nz * d, 0.1, 1e4, 10)
    out = gasatt.electricmagneticfield6(*[torch.tensor(a) if isinstance(a, np.ndarray) else a for a in args],
                                        flags=_lib.FAITHFUL | _lib.POS_IN_CYL)
    return [o.cpu().numpy() for o in out]


def test_after_a_scratch_that_does_not_fit():
    want = small()
    n, d = 65000, 1e-4                  # 4.2e9 cells: 236 GB of scratch, refused before any array is looked at
    outs = [ctypes.c_int64() for _ in range(3)]
    rc = lib.gasatt_electricmagneticfield6(default_context(0).handle, None, None, 0, None, None, 0, None, None, 0, None,
                                           None, None, n, n, d, 1e-13, n * d, n * d, 0.1, 1e4, 5, None,
                                           *[ctypes.byref(o) for o in outs], _lib.FAITHFUL)
    assert rc == _lib.E_CUDA
    for _ in range(2):
        for g, w in zip(small(), want):
            np.testing.assert_array_equal(g, w)
