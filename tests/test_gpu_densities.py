"""Several densities per launch (tensor-core kernel) at the edges of its passes
of 16 and of its halves of 8, and the tile heights that a structure gets by its
size."""
import os

import numpy as np
import pytest

import h2eri_gb300 as hg
from conftest import GOLDEN, relerr

pytestmark = pytest.mark.gpu


def oracle_J(orc, h, D):
    J = np.zeros_like(D)
    orc.oracle_build_Coulomb(h.handle, np.ascontiguousarray(D).ctypes.data, J.ctypes.data)
    return J


@pytest.mark.parametrize("name", ["CH4", "C2H6", "C4H10"])
@pytest.mark.parametrize("n", [2, 8, 9, 16, 17, 26])
def test_density_counts(small_mols, name, n):
    """A density's J does not depend on the others of its launch: the digits
    are its own, the products exact. What differs is the order of the FP64
    additions, which can move the last digit (2^-40) of an entry."""
    h = small_mols[name]
    D = np.stack([hg.molecules.seeded_density(h.num_bf, 3, 40 + i) for i in range(n)])
    D[n // 2] *= 1e-6          # a scale of its own per density
    h.set_precision(hg.MIXED)
    try:
        J = h.build_coulomb(D)
        for i in sorted({0, 1, n // 2, n - 1}):
            pair = h.build_coulomb(np.stack([D[i], D[0]]))
            assert relerr(J[i], pair[0]) < 1e-11, i
    finally:
        h.set_precision(hg.FP64)


@pytest.mark.parametrize("rows", ["0", "128", "256", "512"])
def test_default_tile_rows(alk26, oracle_lib, monkeypatch, rows):
    """A structure that is not tuned gives the J of every explicit tile height
    (FP64 sums of exact tile products: equal to rounding)."""
    D = hg.molecules.seeded_density(alk26.num_bf, 33, 55)
    J = alk26.build_coulomb(D)
    assert alk26.report()["tile_rows"] in (0, 128, 256, 512)
    assert relerr(J, oracle_J(oracle_lib, alk26, D)) < 1e-12
    monkeypatch.setenv("H2G_TILE_ROWS", rows)
    h = hg.H2ERI.from_mol(os.path.join(GOLDEN, "alk26_ccpvdz.mol"), qr_tol=1e-6)
    try:
        assert relerr(h.build_coulomb(D), J) < 1e-12
        assert h.report()["tile_rows"] == int(rows)
    finally:
        h.destroy()
