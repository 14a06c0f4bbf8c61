"""find_CS0's excitation powers at energies where their base is 0, infinite, negative or no number."""
import numpy as np
import pytest
import torch

import gasatt
import pyoracle as O
from gasatt import _lib
from gasatt.tables import N2Tables

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flags", [0, _lib.FAITHFUL])
@pytest.mark.parametrize("om", [0.75, 1.0, 3.0, 2.5])
@pytest.mark.parametrize("nu", [0.75, 1.0, 3.0])
@pytest.mark.parametrize("ga", [0.75, 1.0, 3.0])
def test_powers(om, nu, ga, flags):
    tab = N2Tables(t_exc=np.array([[10.0, 0.3, om, nu, ga]]))
    E = np.array([0.0, -0.0, 1e-300, 1e-3, 0.01, 0.02, 0.5, 30.0, 1e300, -0.02, np.inf, -np.inf, np.nan])
    got = gasatt.find_CS0(*(tab[k] for k in ("t_el", "t_sel", "t_ion", "t_exc")), torch.tensor(E), flags=flags)[2].cpu().numpy()
    want = O.find_cs0(tab, E, flags)[2]
    # a few roundings of the powers
    np.testing.assert_allclose(got, want, rtol=1e-14, atol=0)
