"""QR-preconditioned Jacobi SVD (csrc/svd_qr.cu) on the GPU against LAPACK: the
symmetric decomposition below the size where the product refinement starts and
where that gives up, and the general one through TRG's splits.

Sizes sit at the edges of its variants: one and two columns a block, the last
cluster-sized and the first grid-sized factorisation (64/65 columns), the first
with FP32 sweeps (24), 32-row chunks, 512/513 and beyond.

Tolerances (‖A‖₂ = 1): singular values and residuals n·ε times a constant of 10
for the accumulation over ~10 sweeps; |VᵀV − I| the stop rule 2√n·ε plus the
rounding of an n-term product, together below 8√n·ε.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


def _spectrum(kind, n, rng):
    sign = rng.choice([-1.0, 1.0], n)
    if kind == "graded":  # down to the rounding floor, as the corners of uniform tensors
        return 10.0 ** (-16.0 * np.arange(n) / n) * sign
    if kind == "mild":
        return 10.0 ** (-3.0 * np.arange(n) / n) * sign
    if kind == "rank":  # zero-padded first environments
        return np.where(np.arange(n) < max(1, n // 3), 0.5 ** (np.arange(n) / 4.0), 0.0) * sign
    lam = 10.0 ** (-6.0 * np.arange(n // 2) / n)  # ±λ pairs
    return np.concatenate([lam, -lam, np.zeros(n % 2)])


def _check(A, U, S, V):
    n = A.shape[0]
    scale = np.linalg.norm(A, 2)
    ref = np.sort(np.abs(np.linalg.eigvalsh(A)))[::-1]
    assert np.all(np.diff(S) <= 0.0)
    assert np.max(np.abs(S - ref)) <= 10 * n * EPS * scale
    assert np.max(np.abs(V.T @ V - np.eye(n))) <= 8 * np.sqrt(max(n, 16)) * EPS
    assert np.max(np.abs(U.T @ U - np.eye(n))) <= 8 * np.sqrt(max(n, 16)) * EPS
    assert np.max(np.abs(A @ V - U * S)) <= 10 * n * EPS * scale


@pytest.mark.parametrize("kind", ["graded", "mild", "rank", "pairs"])
@pytest.mark.parametrize("n", [2, 3, 7, 23, 24, 31, 32, 33, 64, 65, 100, 128, 129, 255])
def test_symmetric_matches_lapack(tn, n, kind):
    rng = np.random.default_rng(100 * n + len(kind))
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    A = (Q * _spectrum(kind, n, rng)) @ Q.T
    A = 0.5 * (A + A.T)
    _check(A, *tn.svd_symmetric(A))


@pytest.mark.parametrize("n", [300, 512, 513, 777])
def test_graded_beyond_the_refinement(tn, n):
    """Graded spectra where the product refinement starts (n ≥ 256): it hands them
    over to the QR-preconditioned sweeps, or resolves their small eigenvalues as
    one large group."""
    rng = np.random.default_rng(n)
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    A = (Q * _spectrum("graded", n, rng)) @ Q.T
    A = 0.5 * (A + A.T)
    r0, f0 = tn.solver_stats()
    out = tn.svd_symmetric(A)
    r1, f1 = tn.solver_stats()
    assert r1 - r0 + f1 - f0 == 1
    _check(A, *out)


def test_zero_and_extreme_scales(tn):
    U, S, V = tn.svd_symmetric(np.zeros((40, 40)))
    assert np.all(S == 0.0) and np.allclose(V.T @ V, np.eye(40)) and np.allclose(U.T @ U, np.eye(40))
    rng = np.random.default_rng(1)
    Q, _ = np.linalg.qr(rng.standard_normal((50, 50)))
    A = (Q * _spectrum("mild", 50, rng)) @ Q.T
    A = 0.5 * (A + A.T)
    S1 = tn.svd_symmetric(A)[1]
    for e in (-900, 900):  # powers of two: the same bits up to the exponent
        assert np.array_equal(tn.svd_symmetric(np.ldexp(A, e))[1], np.ldexp(S1, e))


def test_nonfinite_input_gives_nonfinite_values(tn):
    A = np.eye(40)
    A[3, 4] = A[4, 3] = np.nan
    assert not np.any(np.isfinite(tn.svd_symmetric(A)[1]))


@pytest.mark.parametrize("beta,chi,niter", [(0.44, 7, 5), (0.35, 13, 5), (0.44, 23, 5)])
def test_trg_splits_match_the_oracle(tn, orc, beta, chi, niter):
    """General decomposition with both factors accumulated, two at a time: odd
    bond dimensions, and 529×529 splits (the variant beyond 512 rows)."""
    lnZ, g = tn.trg_beta(beta, chi, niter)
    z_ref, g_ref = orc.trg_dbeta(beta, chi, niter)
    assert abs(lnZ - z_ref) < 1e-12 * abs(z_ref)
    assert abs(g - g_ref) < 1e-10 * abs(g_ref)
