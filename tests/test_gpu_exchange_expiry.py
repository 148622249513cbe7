"""An expired wait in the expansion of the low-rank blocks (made once, when the
exchange is set up) is an error of that call: no damaged blocks are kept, and
the next build sets the exchange up anew. The error word is set before the
launch; no kernel waits for anything that does not come."""
import numpy as np
import pytest

import h2eri_gb300 as hg
from conftest import relerr

pytestmark = pytest.mark.gpu


def test_expansion_expiry_is_an_error(library, alk26, oracle_lib):
    D = hg.molecules.seeded_density(alk26.num_bf, 20, 77)
    assert library.H2ERI_gpu_selftest_exchange_expiry(alk26.handle) == 1
    assert b"expansion" in library.H2ERI_gpu_last_error()
    assert library.H2ERI_gpu_check(alk26.handle) == 0        # reported once, by the failing call
    K = alk26.build_exchange(D)
    Ko = np.zeros_like(D)
    oracle_lib.oracle_build_exchange(alk26.handle, D.ctypes.data, Ko.ctypes.data)
    assert relerr(K, Ko) < 1e-12


def test_pending_report_survives_the_set_up(library, alk26):
    """A report of an earlier asynchronous call that was not read yet is not
    taken for the expansion's, and is not lost to it."""
    assert library.H2ERI_gpu_selftest_wait_timeout_async(alk26.handle, 100_000, None) == 0
    assert library.H2ERI_gpu_set_exchange_memory(alk26.handle, 0.0) == 0     # drops the exchange state
    assert alk26.exchange_report()["n_ranges"] >= 1                         # sets it up
    assert library.H2ERI_gpu_check(alk26.handle) == 11
    assert library.H2ERI_gpu_check(alk26.handle) == 0
