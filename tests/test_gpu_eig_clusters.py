"""Symmetric SVD of corners whose small eigenvalues lie closer together than the
FP32 start resolves (csrc/eig_refine.cu, large groups; csrc/svd_qr.cu, FP32
sweeps with the eigenvalue rule): 60% of the spectrum dense in ±1e-3, sizes on
both sides of the sweeps' variants (384/385, 512/513 columns) and the largest.

Tolerances as for the refinement's other spectra: 1e-12 of ‖A‖ for values and
residuals (2e-12 with tensor-core products), ten times that for orthogonality.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def dense_cluster(n, seed):
    rng = np.random.default_rng(seed)
    k = int(0.4 * n)
    lam = np.concatenate([10.0 ** rng.uniform(-2.0, 0.0, k) * rng.choice([-1.0, 1.0], k),
                          rng.uniform(-1e-3, 1e-3, n - k)])
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    A = (Q * lam) @ Q.T
    return 0.5 * (A + A.T)


@pytest.mark.parametrize("tc", [False, True])
@pytest.mark.parametrize("n", [300, 384, 385, 512, 513, 1000, 1024])
def test_dense_small_eigenvalues(tn, n, tc):
    A = dense_cluster(n, n)
    r0, f0 = tn.solver_stats()
    U, S, V = tn.svd_symmetric(A, tensor_cores=tc)
    r1, f1 = tn.solver_stats()
    assert (r1 - r0) + (f1 - f0) == 1
    tol = 2e-12 if tc else 1e-12
    nA = np.linalg.norm(A, 2)
    ref = np.sort(np.abs(np.linalg.eigvalsh(A)))[::-1]
    assert np.max(np.abs(S - ref)) <= tol * nA
    assert np.max(np.abs(V.T @ V - np.eye(n))) <= 10 * tol
    assert np.max(np.abs(U.T @ U - np.eye(n))) <= 10 * tol
    assert np.max(np.abs(A @ V - U * S)) <= tol * nA
