"""The packaged tables are read again when their file has changed, and each object has its own copy."""
import os

import numpy as np

from gasatt import tables
from gasatt.tables import N2Tables


def test_a_new_file_is_read(tmp_path, monkeypatch):
    was = N2Tables()
    path = str(tmp_path / "n2_tables.npz")
    monkeypatch.setattr(tables, "DATA", path)
    for factor in (1.0, 2.0, 3.0):
        new = str(tmp_path / "new.npz")
        np.savez(new, **{k: factor * was[k] for k in N2Tables.NAMES})
        os.replace(new, path)
        for _ in range(2):
            t = N2Tables(path)
            np.testing.assert_array_equal(t["t_exc"], factor * was["t_exc"])
            t["t_exc"][:] = 0                # its own copy
    monkeypatch.undo()
    np.testing.assert_array_equal(N2Tables()["t_exc"], was["t_exc"])
