"""FP64-mode tile kernel (fixed-point products, h2g_tile64.cuh) against the
oracle at its edges: vectors per CTA (1 and 2, with a remainder), inputs whose
exponents spread over a tile or lie far from 1, zero and non-finite inputs."""
import numpy as np
import pytest

from conftest import relerr

pytestmark = pytest.mark.gpu
# sums exact but for roundings to 2^-58 of a tile's largest product (a tile has
# at most 512 x 128 products); the FP64 oracle itself is good to about 1e-15
TOL = 1e-12


def oracle_y(orc, h, x):
    y = np.zeros_like(x)
    orc.oracle_matvec(h.handle, x.ctypes.data, y.ctypes.data)
    return y


@pytest.mark.parametrize("name", ["CH4", "C2H6", "C4H10"])
@pytest.mark.parametrize("nvec", [1, 2, 3, 5])
def test_vectors_per_cta(small_mols, oracle_lib, name, nvec):
    h = small_mols[name]
    x = np.random.default_rng(10 * nvec).standard_normal((nvec, h.krnl_mat_size))
    y = h.matvec(x)
    for i in range(nvec):
        assert relerr(y[i], oracle_y(oracle_lib, h, x[i])) < TOL


@pytest.mark.parametrize("spread", ["graded", "tiny", "huge", "spike", "zero"])
def test_input_exponents(alk32, oracle_lib, spread):
    rng = np.random.default_rng(3)
    x = rng.standard_normal(alk32.krnl_mat_size)
    if spread == "graded":
        x *= 10.0 ** -rng.uniform(0, 12, x.size)
    elif spread == "tiny":
        x *= 2.0 ** -500
    elif spread == "huge":
        x *= 2.0 ** 500
    elif spread == "spike":
        x *= 1e-9
        x[x.size // 3] = 1.0
    else:
        x[:] = 0.0
    y, ref = alk32.matvec(x), oracle_y(oracle_lib, alk32, x)
    if spread == "zero":
        assert not y.any()
        return
    s = np.abs(ref).max()
    assert relerr(y / s, ref / s) < TOL


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_non_finite_inputs(alk32, oracle_lib, value):
    """The tiles that read the entry give what FP64 arithmetic gives: non-finite
    where the oracle is, the other outputs unchanged."""
    x = np.random.default_rng(4).standard_normal((2, alk32.krnl_mat_size))
    x[1, 17] = value
    y = alk32.matvec(x)
    ref = oracle_y(oracle_lib, alk32, x[1])
    assert relerr(y[0], oracle_y(oracle_lib, alk32, x[0])) < TOL
    fine = np.isfinite(ref)
    assert np.array_equal(fine, np.isfinite(y[1]))
    if fine.any():
        assert relerr(y[1][fine], ref[fine]) < TOL
