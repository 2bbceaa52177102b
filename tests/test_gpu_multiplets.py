"""Symmetric SVD (csrc/svd_qr.cu) where eigenvalues of both signs share their size:
a singular subspace of dimension k does not say which vectors are eigenvectors.

Multiplets of 2 to 6 of alternating sign at sizes from 1e-2 to 1e-12 of the
largest eigenvalue; spectra of nothing but exact pairs, near pairs (relative
distance 1e-3 to 1e-11) or quartets; one reflection (all sizes equal) and a permutation.

Bounds as for the other spectra (test_gpu_svd_qr.py): 8√n·ε for orthogonality of both
factors, 10·n·ε·‖A‖ for values and residual; U is ±V to the bit.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


def _sym(lam, rng):
    Q, _ = np.linalg.qr(rng.standard_normal((len(lam), len(lam))))
    A = (Q * lam) @ Q.T
    return 0.5 * (A + A.T)


def _check(tn, A):
    n = A.shape[0]
    U, S, V = tn.svd_symmetric(A)
    scale = np.linalg.norm(A, 2)
    ref = np.sort(np.abs(np.linalg.eigvalsh(A)))[::-1]
    orth = 8 * np.sqrt(max(n, 16)) * EPS
    assert np.all(np.diff(S) <= 0.0)
    assert np.max(np.abs(S - ref)) <= 10 * n * EPS * scale
    assert np.max(np.abs(V.T @ V - np.eye(n))) <= orth
    assert np.max(np.abs(U.T @ U - np.eye(n))) <= orth
    assert np.max(np.abs(A @ V - U * S)) <= 10 * n * EPS * scale
    assert np.array_equal(np.abs(U), np.abs(V))


def _alternating(n):
    return np.where(np.arange(n) % 2 == 0, 1.0, -1.0)


@pytest.mark.parametrize("n", [9, 24, 64, 65, 130, 300])
@pytest.mark.parametrize("mult", [2, 3, 4, 6])
def test_one_multiplet(tn, n, mult):
    rng = np.random.default_rng(10 * n + mult)
    for size in (1e-2, 1e-5, 1e-7, 1e-9, 1e-12):
        lam = 10.0 ** rng.uniform(-9.0, 0.0, n) * rng.choice([-1.0, 1.0], n)
        lam[0] = 1.0
        lam[1:1 + mult] = size * _alternating(mult)
        _check(tn, _sym(lam, rng))


@pytest.mark.parametrize("n", [16, 40, 90, 200, 300])
@pytest.mark.parametrize("kind", ["pairs", "near", "quartets", "reflection", "uniform"])
def test_whole_spectra(tn, n, kind):
    rng = np.random.default_rng(n)
    spectra = {
        "pairs": [10.0 ** (-14.0 * (np.arange(n) // 2) / (n / 2)) * _alternating(n)],
        "near": [10.0 ** (-7.0 * (np.arange(n) // 2) / (n / 2)) * np.where(np.arange(n) % 2 == 0, 1.0, -1.0 - gap)
                 for gap in (1e-3, 1e-5, 1e-7, 1e-9, 1e-11)],
        "quartets": [10.0 ** (-14.0 * (np.arange(n) // 4) / (n / 4)) * _alternating(n)],
        "reflection": [_alternating(n)],
        "uniform": [rng.uniform(-1.0, 1.0, n)],
    }
    for lam in spectra[kind]:
        _check(tn, _sym(lam, rng))


def test_permutation_and_scaled_quartets(tn):
    _check(tn, np.eye(40)[::-1].copy())
    rng = np.random.default_rng(3)
    A = _sym(10.0 ** (-6.0 * (np.arange(32) // 4) / 8) * _alternating(32), rng)
    S = tn.svd_symmetric(A)[1]
    for e in (-900, 900):
        U2, S2, V2 = tn.svd_symmetric(np.ldexp(A, e))
        assert np.max(np.abs(np.ldexp(S2, -e) - S)) <= 10 * 32 * EPS * S[0]
        assert np.max(np.abs(np.ldexp(np.ldexp(A, e) @ V2 - U2 * S2, -e))) <= 10 * 32 * EPS * S[0]
