"""Contractions of a matrix with a vector (csrc/contract.cu) on both sides of the
rule that chooses between the matrix-vector kernels and the DFMA tiles: rows from
64 per SM on, up to 32 columns of at least 16384 values, either operand first,
label orders that are not a matrix, and a dot product.

Bound: K-term FP64 sums of standard normals, 1e-13·√K of the largest result.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [("ij,j->i", dict(i=9727, j=5)), ("ij,j->i", dict(i=9728, j=5)), ("ij,j->i", dict(i=20001, j=33)),
         ("ji,j->i", dict(i=32, j=16383)), ("ji,j->i", dict(i=32, j=16384)), ("ji,j->i", dict(i=33, j=16384)),
         ("ji,j->i", dict(i=1, j=40001)), ("j,ji->i", dict(i=7, j=20003)), ("j,ij->i", dict(i=9999, j=3)),
         ("ijk,k->ij", dict(i=101, j=99, k=7)), ("ikj,k->ji", dict(i=101, j=99, k=7)),
         ("abi,ab->i", dict(a=130, b=130, i=9)), ("i,i->", dict(i=70001)), ("i,j->ij", dict(i=9800, j=1))]


@pytest.mark.parametrize("spec,ext", CASES)
def test_matrix_vector(tn, spec, ext):
    rng = np.random.default_rng(sum(ext.values()))
    la, rest = spec.split(",")
    lb, _ = rest.split("->")
    A = rng.standard_normal(tuple(ext[ch] for ch in la))
    B = rng.standard_normal(tuple(ext[ch] for ch in lb))
    K = np.prod([ext[ch] for ch in set(la) & set(lb)])
    got, ref = tn.contract(spec, A, B), np.einsum(spec, A, B)
    assert got.shape == ref.shape
    assert np.max(np.abs(got - ref)) <= 1e-13 * np.sqrt(K) * max(1.0, np.max(np.abs(ref)))
