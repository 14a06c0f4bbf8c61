"""The field update's patches of 16, 32 and 64 rows (knob 12, 16, 20): grids that
end at, before and past a tile (10, 26, 58 rows) and put the conducting end in the
first and last row of a warp's segment (4 or 8 rows); against the oracle, all
shapes and the automatic choice bit-identical, FP32 quads equal to fields."""
import numpy as np
import pytest

import pyoracle as O
from _cases import close
from gasatt import abi
from test_field_update_gpu import STEPS, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flags", [0, abi.Q_ER_END_COPY])
@pytest.mark.parametrize("nz", [2, 25, 26, 57, 58, 60, 61, 64, 65, 121])
def test_tile_edges(tables, nz, flags):
    nr = 53
    ref = None
    for rows in (0, 12, 16, 20):
        (f64, st), cfg, parts, flds = run(nr, nz, flags, abi.FP64, rows)
        assert st == 0
        if ref is None:
            ref = f64
            orc = O.Sim(cfg, tables, cap=cfg.capacity)
            orc.load(*parts)
            orc.Er[:], orc.Ez[:], orc.H[:] = flds
            orc.prologue()
            for _ in range(STEPS):
                orc.step()
            for g, w, k in zip(f64, (orc.Er, orc.Ez, orc.H), ("Er", "Ez", "H")):
                close(g, w, 1e-12, k)              # as the field update's own test
        for a, b in zip(ref, f64):
            np.testing.assert_array_equal(a, b)
    f32 = [run(nr, nz, flags, abi.FP32_SPLIT, rows, gather)[0][0]
           for rows in (12, 16, 20) for gather in (abi.GATHER_QUADS, abi.GATHER_FIELDS)]
    for f in f32[1:]:
        for a, b in zip(f, f32[0]):
            np.testing.assert_array_equal(a, b)
