"""The subspace solver's small dense kernels (csrc/dense_small.cu) at the edges of
their tiles, through the mixed-path energy against plain CTMRG (the CPU oracle's, or the GPU's
full decompositions where the oracle's LAPACK gives up).

The block width is p = min(4χ, χ + max(16, χ/2)) here (D = 2): one and several
panels of the Cholesky cluster with and without a remainder (p = 8, 12, 20, 22,
33, 49), 32-row chunks of the FP32 eigensolver (p = 32, 33, 64, 96, 97, 128, 129)
and its largest size (160); the gauge alignment's polar factor takes χ, whose
4×4 tiles end inside or at the matrix.  Uniform tensors have rank-deficient
blocks (the pivot floor, a full second factorisation), N(0,1) ones have not (a
second Gram matrix near the identity, which is not factored).

Tolerance: both runs stop at 1e-10 on their spectra; the energy's error is of
that order, 1e-9 allowed.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chi", [2, 3, 5, 6, 16, 17, 33, 43, 64, 65, 85, 86, 107])
@pytest.mark.parametrize("recipe", ["uniform", "normal_maxabs"])
def test_mixed_energy_at_block_width_edges(tn, orc, chi, recipe):
    h = tn.hamiltonian(tn.Heisenberg())
    A = tn.site_tensor(recipe, 2, 2, 0)
    E = tn.energy(h, tn.SquareIPEPS(A), chi, 1e-10, 300, opts=tn.mixed_opts())
    if chi <= 43:
        E_ref = float(orc.energy(h, torch.as_tensor(np.ascontiguousarray(A)), chi, 1e-11, 300))
    else:  # corners rank-deficient beyond what every LAPACK's SVD takes: the plain GPU path
        E_ref = tn.energy(h, tn.SquareIPEPS(A), chi, 1e-11, 300)
    assert abs(E - E_ref) < 1e-9
