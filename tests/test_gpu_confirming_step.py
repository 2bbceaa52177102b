"""The mixed path's gradient after its confirming step (csrc/ctmrg_mixed.cu).

The stop rule compares Ritz values, which converge with the square of the
environment's error; the implicit adjoint feels the error itself.  A run that is
differentiated therefore takes one step more than the same run without a gradient.

D = 3, χ = 36 uniform tensors, tol 1e-12: the gradient within 5e-9 of the plain
path's at tol 1e-13 (the worst of 60 tensors was 4.0e-9; 1e-9 is exceeded by 2 of
them, by 5 without the step), the median of six within 1e-11, and the energy is the
one without a gradient to 1e-13.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_a_differentiated_run_takes_one_step_more(tn):
    h = tn.hamiltonian(tn.Heisenberg())
    errors = []
    for seed in range(6):
        p = tn.SquareIPEPS(np.asfortranarray(np.random.default_rng(seed).random((3, 3, 3, 3, 2))))
        _, g_ref = tn.energy_and_gradient(h, p, 36, 1e-13, 200)
        stats = {}
        E, g = tn.energy_and_gradient(h, p, 36, 1e-12, 200, opts=tn.mixed_opts(fp_tol=1e-11), stats=stats)
        alone = tn._energy(h, p, 36, 1e-12, 200, opts=tn.mixed_opts(fp_tol=1e-11))
        assert stats["steps"] == alone.steps + 1
        assert abs(E - alone.E) <= 1e-13 * abs(E)
        errors.append(np.max(np.abs(g - g_ref)) / np.max(np.abs(g_ref)))
    assert max(errors) <= 5e-9 and np.median(errors) <= 1e-11
