"""The DFMA GEMM (csrc/gemm_f64.cu) against NumPy at the edges of its tiles and
splits, and pairwise contractions whose labels it reads and writes in place.

Tolerance: an entry of a K-term FP64 sum is within K·ε of the sum of the terms'
magnitudes (|A|·|B|); the split sums add their number of parts (at most 64).
"""
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


@pytest.mark.parametrize("K", [1, 15, 16, 17, 33, 64, 700])
@pytest.mark.parametrize("M,N", [(1, 2), (15, 16), (16, 17), (33, 31), (64, 65), (130, 7), (257, 300)])
def test_gemm_edges(tn, M, N, K):
    rng = np.random.default_rng(M * 10007 + N * 101 + K)
    for ta, tb in itertools.product("NT", "NT"):
        A = rng.standard_normal((K, M) if ta == "T" else (M, K))
        B = rng.standard_normal((N, K) if tb == "T" else (K, N))
        C = rng.standard_normal((M, N))
        opA, opB = (A.T if ta == "T" else A), (B.T if tb == "T" else B)
        bound = (K + 64) * EPS * (np.abs(opA) @ np.abs(opB)) + 4 * EPS * np.abs(C)
        assert np.all(np.abs(tn.gemm(A, B, ta, tb) - opA @ opB) <= bound)
        got = tn.gemm(A, B, ta, tb, alpha=-0.5, beta=1.5, Cin=C)
        assert np.all(np.abs(got - (1.5 * C - 0.5 * (opA @ opB))) <= 2 * bound + 8 * EPS * np.abs(C))


def test_split_products_leave_their_counters_at_zero(tn):
    """Many split products in a row on one context give the same bits."""
    rng = np.random.default_rng(3)
    A, B = rng.standard_normal((20, 900)), rng.standard_normal((900, 20))
    first = tn.gemm(A, B)
    for _ in range(20):
        tn.gemm(A[:, :300], B[:300])
        assert np.array_equal(tn.gemm(A, B), first)


@pytest.mark.parametrize("spec", ["ab,bc->ac", "ab,bc->ca", "abc,cbd->ad", "abc,cbd->da", "abcd,bedf->aecf",
                                  "abcd,dbe->cea", "abc,dbe->eadc", "abcde,cfag->gbfde", "ab,ab->", "ab,cd->cadb",
                                  "abcdef,bdgf->gaec", "abcdefgh,hfdb->geca"])
def test_contractions_in_any_label_order(tn, spec):
    rng = np.random.default_rng(len(spec))
    lhs, _ = spec.split("->")
    la, lb = lhs.split(",")
    for ext in (dict(zip("abcdefgh", (3, 1, 5, 2, 4, 3, 2, 3))), dict(zip("abcdefgh", (2, 7, 3, 4, 1, 5, 6, 2)))):
        A, B = rng.standard_normal([ext[x] for x in la]), rng.standard_normal([ext[x] for x in lb])
        K = int(np.prod([ext[x] for x in la if x in lb]))
        ref = np.einsum(spec, A, B)
        bound = (K + 64) * EPS * np.einsum(spec, np.abs(A), np.abs(B))
        assert np.all(np.abs(tn.contract(spec, A, B).reshape(ref.shape, order="F") - ref) <= bound)
