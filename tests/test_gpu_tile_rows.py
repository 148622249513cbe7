"""Tile plans of a structure that is not tuned: the height that the rule gives
by its plan, and the plan that launches of several vectors take (another one
in the larger of these structures), against the oracle."""
import numpy as np
import pytest

import h2eri_gb300 as hg
from conftest import relerr

pytestmark = pytest.mark.gpu


def oracle_y(orc, h, x):
    y = np.zeros_like(x)
    orc.oracle_matvec(h.handle, x.ctypes.data, y.ctypes.data)
    return y


@pytest.mark.parametrize("name,rows", [("alkane:2", 0), ("alkane:8", 0), ("alkane:10", 128)])
def test_default_plans(oracle_lib, tmp_path, name, rows):
    """C2H6 fills 0.1 waves, C8H18 4 and C10H22 15 (QR 1e-6); FP64 mode."""
    path = str(tmp_path / "m.mol")
    hg.molecules.write_alkane(path, int(name.split(":")[1]))
    h = hg.H2ERI.from_mol(path, qr_tol=1e-6)
    try:
        x = np.random.default_rng(31).standard_normal((3, h.krnl_mat_size))
        for n in (1, 2, 3):
            y = np.atleast_2d(h.matvec(x[:n] if n > 1 else x[0]))
            for i in range(n):
                assert relerr(y[i], oracle_y(oracle_lib, h, x[i])) < 1e-12
        assert h.report()["tile_rows"] == rows
        h.autotune(1)
        y = h.matvec(x)
        assert max(relerr(y[i], oracle_y(oracle_lib, h, x[i])) for i in range(3)) < 1e-12
    finally:
        h.destroy()
