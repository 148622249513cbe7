"""FP64 exchange products on the tensor cores (k_gemm_z) and the FP64 near field
(k_near64) against the oracle where their tilings can go wrong: no far field,
few rows, one and many ranges of n (short runs of columns), inner products
longer than a tile's 64, densities with a wide spread of magnitudes, and a
density entry that is not finite."""
import numpy as np
import pytest

import h2eri_gb300 as hg
from conftest import relerr
from h2eri_gb300 import molecules

pytestmark = pytest.mark.gpu
# digit products are exact to 2^-62 of a row's largest, sums rounded once per
# tile; K's FP64 atomics dominate (C5H12: 0.8e-15 against 80-bit arithmetic)
TOL = 1e-12


def oracle_K(orc, h, D):
    K = np.zeros_like(D)
    orc.oracle_build_exchange(h.handle, D.ctypes.data, K.ctypes.data)
    return K


def density(h, seed):
    return molecules.seeded_density(h.num_bf, max(1, h.num_bf // 6), seed)


@pytest.mark.parametrize("name", ["CH4", "C2H6", "C4H10"])
def test_small(small_mols, oracle_lib, name):
    h = small_mols[name]
    D = density(h, 5)
    assert relerr(h.build_exchange(D), oracle_K(oracle_lib, h, D)) < TOL


@pytest.mark.parametrize("bytes_", [3e8, 2e7, 2e6])
def test_ranges(alk26, oracle_lib, bytes_):
    D = density(alk26, 6)
    assert hg.lib().H2ERI_gpu_set_exchange_memory(alk26.handle, bytes_) == 0
    K = alk26.build_exchange(D)
    n = alk26.exchange_report()["n_ranges"]
    assert hg.lib().H2ERI_gpu_set_exchange_memory(alk26.handle, 0.0) == 0
    assert n > 1
    assert relerr(K, oracle_K(oracle_lib, alk26, D)) < TOL


@pytest.mark.parametrize("spread", ["graded", "spike", "tiny"])
def test_density_magnitudes(alk26, oracle_lib, spread):
    D = density(alk26, 7)
    if spread == "graded":
        s = 10.0 ** -np.random.default_rng(1).uniform(0, 4, D.shape[0])
        D = np.ascontiguousarray(s[:, None] * D * s[None, :])
    elif spread == "spike":
        D *= 1e-7
        D[11, 90] = D[90, 11] = 1.0
    else:
        D *= 1e-8
    assert relerr(alk26.build_exchange(D), oracle_K(oracle_lib, alk26, D)) < TOL


def test_non_finite_density(alk26):
    """Rows with an infinity take FP64 arithmetic: K is non-finite in some rows
    and the rest is that of the density without them."""
    D = density(alk26, 8)
    K = alk26.build_exchange(D)
    E = D.copy()
    E[3, 50] = E[50, 3] = np.inf
    KE = alk26.build_exchange(E)
    bad = ~np.isfinite(KE)
    assert bad.any() and not bad.all()
    E[3, 50] = E[50, 3] = 0.0
    assert relerr(KE[~bad], alk26.build_exchange(E)[~bad]) < 1e-12
    assert relerr(alk26.build_exchange(D), K) < 1e-13
