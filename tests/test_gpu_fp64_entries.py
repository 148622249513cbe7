"""FP64 mode, entry by entry: |y - y_oracle| <= c 2^-53 (|A| |x|), where |A| |x|
comes from the oracle on the blocks' magnitudes. An arithmetic that is accurate
only beside the largest entry of a tile passes a norm and fails here, with inputs
that are small or zero where the matrix is large.

An output is a sum over at most eight stages of the tree (up, across, down, near
field, two factors of a low-rank block), in chains of up to 512 terms, on both
sides of the comparison: c = 8 * 512 * 2."""
import contextlib
import ctypes

import numpy as np
import pytest

import h2eri_gb300 as hg

pytestmark = pytest.mark.gpu
BOUND = 8 * 512 * 2 * 2.0 ** -53


@contextlib.contextmanager
def magnitudes(h):
    """The structure's host blocks replaced by their magnitudes (the device
    copies stay as they were uploaded)."""
    h.upload()
    saved = []
    for name, n in (("U", h.s.n_node), ("c_B_blks", h.s.n_B), ("c_D_blks", h.s.n_D)):
        mats = ctypes.cast(getattr(h.s, name), ctypes.POINTER(ctypes.POINTER(hg.DenseMat)))
        for i in range(n):
            m = mats[i].contents
            size = (m.nrow + m.ncol) * -m.ld if m.ld < 0 else m.nrow * m.ld
            if m.nrow == 0 or m.ncol == 0 or size == 0:
                continue
            a = np.ctypeslib.as_array(m.data, (size,))
            saved.append((a, a.copy()))
            np.abs(a, out=a)
    try:
        yield
    finally:
        for a, old in saved:
            a[:] = old


def inputs(kind, n):
    rng = np.random.default_rng(21)
    x = rng.standard_normal(n)
    if kind == "graded":
        x *= 10.0 ** -rng.uniform(0, 20, n)
    elif kind == "spike":
        x *= 1e-15
        x[n // 3] = 1.0
    elif kind == "unit":
        x[:] = 0.0
        x[2 * n // 3] = 1.0
    elif kind == "sparse":
        x[rng.random(n) < 0.97] = 0.0
        x *= 10.0 ** -rng.uniform(0, 30, n)
    return x


@pytest.mark.parametrize("nvec", [1, 2])
@pytest.mark.parametrize("kind", ["normal", "graded", "spike", "unit", "sparse"])
def test_matvec_entries(alk32, oracle_lib, kind, nvec):
    x = inputs(kind, alk32.krnl_mat_size)
    xs = np.stack([x, inputs("normal", x.size)])[:nvec]
    y = alk32.matvec(xs if nvec > 1 else x)
    y = y[0] if nvec > 1 else y
    ref, size, ax = np.zeros_like(x), np.zeros_like(x), np.abs(x)
    oracle_lib.oracle_matvec(alk32.handle, x.ctypes.data, ref.ctypes.data)
    with magnitudes(alk32):
        oracle_lib.oracle_matvec(alk32.handle, ax.ctypes.data, size.ctypes.data)
    off = np.abs(y - ref)
    assert (off <= BOUND * size).all(), (off[size > 0] / size[size > 0]).max()


def density(kind, h):
    D = hg.molecules.seeded_density(h.num_bf, max(1, h.num_bf // 6), 9)
    rng = np.random.default_rng(22)
    if kind == "graded":
        s = 10.0 ** -rng.uniform(0, 6, D.shape[0])
        D = s[:, None] * D * s[None, :]
    elif kind == "spike":
        D = 1e-10 * D
        D[7, 19] = D[19, 7] = 1.0
    elif kind == "constant":     # rows whose digits are all 127, in sums of any length
        D = np.full_like(D, 127.0 / 255.0)
    return np.ascontiguousarray(D)


@pytest.mark.parametrize("kind", ["normal", "graded", "spike", "constant"])
def test_exchange_entries(alk26, oracle_lib, kind):
    """K's terms (basis, block and density entries, up to 512 per chain) likewise."""
    D = density(kind, alk26)
    K = alk26.build_exchange(D)
    ref, size, aD = np.zeros_like(D), np.zeros_like(D), np.abs(D)
    oracle_lib.oracle_build_exchange(alk26.handle, D.ctypes.data, ref.ctypes.data)
    with magnitudes(alk26):
        oracle_lib.oracle_build_exchange(alk26.handle, aD.ctypes.data, size.ctypes.data)
    off = np.abs(K - ref)
    assert (off <= BOUND * size).all(), (off[size > 0] / size[size > 0]).max()


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_exchange_non_finite_entries(alk26, oracle_lib, value):
    """K is non-finite in the entries where the oracle's is, and in no other."""
    D = density("normal", alk26)
    D[3, 50] = D[50, 3] = value
    K, ref = alk26.build_exchange(D), np.zeros_like(D)
    oracle_lib.oracle_build_exchange(alk26.handle, D.ctypes.data, ref.ctypes.data)
    fine = np.isfinite(ref)
    assert np.array_equal(np.isfinite(K), fine)
    assert np.abs(K - ref)[fine].max() <= 1e-12 * np.abs(ref[fine]).max()
