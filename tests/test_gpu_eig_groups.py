"""Corners with 65 to 130 clustered eigenvalues: the smallest groups that the
refinement solves as one (csrc/eig_refine.cu), flat or graded inside, in matrices
of 256 to 640 columns with both signs outside.

Every one is refined, none handed over.  Bounds as for the refinement's other
spectra: 1e-12 of ‖A‖ for values and residual, ten times that for orthogonality.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [256, 300, 400, 640])
@pytest.mark.parametrize("k", [65, 66, 80, 96, 130])
def test_groups_are_refined_to_the_bound(tn, n, k):
    for width, grades in ((1e-5, 0), (1e-4, 1), (1e-3, 1), (1e-3, 2)):
        for seed in range(2):
            rng = np.random.default_rng(1000 * n + 10 * k + seed)
            inner = rng.uniform(-width, width, k) * 10.0 ** (-grades * rng.random(k))
            lam = np.concatenate([10.0 ** rng.uniform(-1.0, 0.0, n - k) * rng.choice([-1.0, 1.0], n - k), inner])
            Q, R = np.linalg.qr(rng.standard_normal((n, n)))
            Q = Q * np.sign(np.diag(R))
            A = (Q * lam) @ Q.T
            A = 0.5 * (A + A.T)
            r0, f0 = tn.solver_stats()
            U, S, V = tn.svd_symmetric(A)
            assert tuple(b - a for a, b in zip((r0, f0), tn.solver_stats())) == (1, 0)
            nA = np.linalg.norm(A, 2)
            assert np.max(np.abs(S - np.sort(np.abs(np.linalg.eigvalsh(A)))[::-1])) <= 1e-12 * nA
            assert np.max(np.abs(V.T @ V - np.eye(n))) <= 1e-11
            assert np.max(np.abs(A @ V - U * S)) <= 1e-12 * nA
