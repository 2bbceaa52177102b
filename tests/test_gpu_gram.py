"""Symmetric products as half of their tiles (the last measurement of the corner
refinement): eigenpairs of symmetric matrices whose size ends inside, at and just
beyond a tile, against their definition.

Tolerance: the refinement stops with |XᵀAX − Λ| ≤ 1e-10·‖A‖_F before its last
correction, which squares it; what is left is rounding of n-term DFMA sums,
n·ε·‖A‖ for the residual and n·ε for the orthogonality.  A tile that was skipped
or mirrored wrongly shows as an error of order one.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [256, 257, 271, 272, 300, 511, 512, 513, 640])
def test_refined_symmetric_svd(tn, n):
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n))
    A = np.asfortranarray((A + A.T) / 2)
    U, S, V = tn.svd_symmetric(A)
    eps, nrm = np.finfo(float).eps, np.linalg.norm(A, 2)
    assert np.linalg.norm(A @ V - U * S, 2) <= n * eps * nrm
    assert np.linalg.norm(V.T @ V - np.eye(n), 2) <= n * eps
    assert np.linalg.norm(U.T @ U - np.eye(n), 2) <= n * eps
    assert np.max(np.abs(S - np.sort(np.abs(np.linalg.eigvalsh(A)))[::-1])) <= n * eps * nrm
