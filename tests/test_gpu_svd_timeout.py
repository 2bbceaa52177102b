"""A bounded wait that expires between the two factorisations of the
QR-preconditioned SVD (csrc/svd_qr.cu).

``TNAD_TEST_FAULT=qr_timeout`` sets the error word of the context's next such
decomposition as a wait of the second factorisation would: its column order is
then never written, and the kernels after it must not store through it.  The
host reports TNAD_ERR_TIMEOUT, and the context works normally afterwards.

23 columns: no FP32 sweeps, so that the host reads the status at the end only;
24 and more: it reads the rank, and the status, after the FP32 sweeps.  Rank
deficient matrices take the second factorisation, full-rank ones skip it.
"""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rank", ["full", "deficient"])
@pytest.mark.parametrize("n", [9, 23, 24, 70, 200])
def test_expired_wait_is_an_error_and_nothing_else(tn, n, rank):
    rng = np.random.default_rng(n)
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    lam = np.where(np.arange(n) < (n if rank == "full" else n // 2), 2.0 ** (-np.arange(n) / 8.0), 0.0)
    A = np.asfortranarray((Q * lam) @ Q.T)
    A = np.asfortranarray(0.5 * (A + A.T))
    os.environ["TNAD_TEST_FAULT"] = "qr_timeout"
    try:
        c = tn._lib.Context(0)
    finally:
        del os.environ["TNAD_TEST_FAULT"]
    try:
        U, S, V = tn.fzeros((n, n)), tn.fzeros((n,)), tn.fzeros((n, n))
        args = (c.h, tn._lib.PREC_FP64, tn.ptr(A), n, tn.ptr(U), tn.ptr(S), tn.ptr(V))
        assert c.lib.tnad_svd_sym(*args) == -8, c.lib.tnad_last_error(c.h)  # TNAD_ERR_TIMEOUT
        assert b"wait expired" in c.lib.tnad_last_error(c.h)
        assert c.lib.tnad_svd_sym(*args) == 0, c.lib.tnad_last_error(c.h)
        assert np.max(np.abs(S - lam)) <= 10 * n * np.finfo(float).eps
        assert np.max(np.abs(A @ V - U * S)) <= 10 * n * np.finfo(float).eps
    finally:
        c.close()


def test_expired_wait_in_a_pair_of_splits(tn):
    """Both splits of a TRG step (general matrices, both factors accumulated)."""
    import ctypes as C

    os.environ["TNAD_TEST_FAULT"] = "qr_timeout"
    try:
        c = tn._lib.Context(0)
    finally:
        del os.environ["TNAD_TEST_FAULT"]
    try:
        a = tn.farr(tn.model_tensor(tn.Ising(), 0.4))
        z = C.c_double()
        args = (c.h, tn.ptr(a), 2, 7, 4, 1e-16, C.byref(z), None)
        assert c.lib.tnad_trg(*args) == -8, c.lib.tnad_last_error(c.h)
        assert c.lib.tnad_trg(*args) == 0, c.lib.tnad_last_error(c.h)
        assert abs(z.value - tn.trg(a, 7, 4)) <= 1e-13 * abs(z.value)
    finally:
        c.close()
