"""TRG on tensors whose splits have full rank (csrc/svd_qr.cu with both factors
accumulated), ln Z and its gradient against the CPU oracle (FP64, LAPACK).

* Random positive tensors with bond dimension 25 to 32: splits of 625 to 1024
  columns, of full rank at the third step: the variants of 640, 768, 1024 rows, a pair in one
  batch up to 608 columns and one after the other beyond.  (Ising splits of these
  sizes have rank ~250, which the third group reaches.)
* Graded tensors: every leg weighted by 10^-(g·index), so that the kept singular
  values reach 1e-5 to 1e-11 of the largest one, and √s of them is differentiated.
  The solver is accurate to ε·s₁ there, as LAPACK is.

Bounds: 1e-12 relative for ln Z; the gradient's conditioning is the distance of the
kept from the cut values (a few percent here), 1e-10 of its largest entry.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _oracle(orc, a, chi, niter):
    import torch

    t = torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, requires_grad=True)
    z = orc.trg(t, chi, niter)
    (g,) = torch.autograd.grad(z, t)
    return float(z.detach()), g.numpy()


def _compare(tn, orc, a, chi, niter):
    z, g = tn.trg_gradient(np.asfortranarray(a), chi, niter)
    z_ref, g_ref = _oracle(orc, a, chi, niter)
    assert abs(z - z_ref) <= 1e-12 * abs(z_ref)
    assert np.max(np.abs(g - g_ref)) <= 1e-10 * np.max(np.abs(g_ref))


@pytest.mark.parametrize("d,chi", [(5, 24), (5, 25), (6, 27), (6, 29), (6, 32)])
def test_full_rank_splits(tn, orc, d, chi):
    a = np.random.default_rng(10 * d + chi).random((d, d, d, d)) + 0.1
    _compare(tn, orc, a, chi, 3)


@pytest.mark.parametrize("beta,chi", [(0.35, 25), (0.44, 29), (0.6, 32)])
def test_rank_deficient_splits(tn, orc, beta, chi):
    lnZ, g = tn.trg_beta(beta, chi, 7)
    z_ref, g_ref = orc.trg_dbeta(beta, chi, 7)
    assert abs(lnZ - z_ref) < 1e-12 * abs(z_ref)
    assert abs(g - g_ref) < 1e-10 * abs(g_ref)


@pytest.mark.parametrize("d,grade,chi", [(3, 1.0, 7), (4, 1.0, 12), (3, 2.0, 8), (4, 1.5, 10), (4, 1.8, 16)])
def test_small_kept_values_are_differentiated(tn, orc, d, grade, chi):
    rng = np.random.default_rng(int(10 * grade) + d)
    w = 10.0 ** (-grade * np.arange(d) / 2.0)
    a = (rng.random((d, d, d, d)) + 0.1) * np.einsum("i,j,k,l->ijkl", w, w, w, w)
    _compare(tn, orc, a, chi, 2)
