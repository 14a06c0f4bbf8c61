"""electron_collision where its kernels branch: no electron, one, counts around
a warp and a group of elastic collisions, with few and with almost all
electrons colliding, in both angle inversions."""
import numpy as np
import pytest
import torch

import gasatt
import pyoracle as O
from _cases import close
from gasatt import _lib
from test_dropin_gpu import collision_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flags", [_lib.FAITHFUL & ~_lib.Q_EXC_POWF, 0, _lib.Q_CDF_NEXTBIN, _lib.FAITHFUL & ~_lib.Q_CDF_NEXTBIN])
@pytest.mark.parametrize("n,dt", [(0, 2e-10), (1, 1e-6), (31, 1e-6), (33, 2e-10), (300, 1e-6), (20_000, 1e-12)])
def test_against_oracle(tables, n, dt, flags):
    cs = collision_inputs(n + 1, n=n)
    se, si, sx = (np.nan_to_num(a, nan=0.0) for a in O.find_cs0(tables, cs["kin"], _lib.FAITHFUL))
    common = (tables["t_el"], tables["t_sel_1"], tables["t_del"], tables["t_sdel"], tables["t_exc"])
    cells = (cs["sum_cell"], cs["cellnumxy"], cs["density"], cs["temperature"], cs["PHIp"], cs["phimax"], cs["dr"], cs["dz"])
    T = lambda a: torch.tensor(a) if isinstance(a, np.ndarray) else a  # noqa: E731
    got = gasatt.electron_collision(*map(T, (cs["pos"], cs["vel"], cs["ion_pos"], cs["ion_vel"])), *common, T(cs["kin"]),
                                    cs["sum_cell"], cs["cellnumxy"], T(cs["density"]), T(cs["temperature"]), cs["PHIp"],
                                    cs["phimax"], cs["dr"], cs["dz"], T(se), T(si), T(sx), dt, draws=T(cs["draws"]), flags=flags)
    want = O.electron_collision(cs["pos"], cs["vel"], cs["ion_pos"], cs["ion_vel"], tables, cs["kin"], *cells, se, si, sx,
                                dt, cs["draws"], flags)
    # as the drop-in's own test: 1e-12 of the largest value, 1e-6 with the single-precision powers
    rtol = 1e-6 if flags & _lib.Q_EXC_POWF else 1e-12
    for g, w, k in zip(got, want, ("e_pos", "e_vel", "i_pos", "i_vel")):
        close(g.cpu().numpy(), w, rtol, k)
