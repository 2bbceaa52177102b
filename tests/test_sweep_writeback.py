"""Write-back decision of the FP64 Jacobi sweeps (csrc/svd_qr.cu, k_svd_sweeps).

A CTA rotates two disjoint column pairs with two groups of 64 threads and then
stores its four columns, each thread its own share, if the round rotated
anything: `nrot`, a shared counter, against the value read earlier (`rot0`).
All threads have to come to the same answer, or a column is stored in part.

The GPU gives no control over the order of two groups, so the orders are
enumerated here: the place of the read relative to the CTA barriers is taken
from the source, and every order that those barriers allow is tried.  The GPU
test runs matrices whose late rounds rotate a single pair.
"""
import itertools
import re
from pathlib import Path

import numpy as np
import pytest

SRC = Path(__file__).resolve().parent.parent / "tensornetworkad.jl_gb300" / "csrc" / "svd_qr.cu"


def _round_source():
    text = SRC.read_text()
    body = text[text.index("k_svd_sweeps(SvdArgs a)"):]
    body = body[body.index("cp.async.wait_all"):]
    return re.sub(r"//[^\n]*", "", body[:body.index("if (nrot != rot0")])


def _decisions(read_before_barrier, rotates):
    """The answers that threads of the two groups can reach: each thread's read and
    each group's count are events of the phase between two barriers."""
    seen = set()
    events = [("read", 0), ("read", 1)] + [("count", g) for g in (0, 1) if rotates[g]]
    for order in itertools.permutations(events):
        if any(order.index(("count", g)) < order.index(("read", g)) for g in (0, 1) if rotates[g]):
            continue  # a thread counts after its own read
        nrot, rot0 = 0, {}
        if read_before_barrier:
            rot0 = {0: 0, 1: 0}
        for kind, g in order:
            if kind == "count":
                nrot += 1
            elif not read_before_barrier:
                rot0[g] = nrot
        seen.add((nrot != rot0[0], nrot != rot0[1]))
    return seen


@pytest.mark.parametrize("rotates", [(False, False), (True, False), (False, True), (True, True)])
def test_both_groups_agree_on_the_write_back(rotates):
    src = _round_source()
    read = src.index("rot0 = nrot")
    before = read < src.index("__syncthreads()")
    assert "process(" not in src[:read]
    for a, b in _decisions(before, rotates):
        assert a == b == any(rotates)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [40, 96, 200])
def test_rounds_with_a_single_rotation(tn, n):
    """Diagonal but for a few coupled pairs: almost every round rotates one pair or
    none.  Values and factors to the bound of the other decompositions."""
    rng = np.random.default_rng(n)
    eps = np.finfo(float).eps
    for seed in range(6):
        lam = np.linspace(1.0, 2.0, n) * rng.choice([-1.0, 1.0], n)
        A = np.diag(lam)
        for i, j in rng.choice(n, (4, 2), replace=False):
            A[i, j] = A[j, i] = 10.0 ** rng.uniform(-9.0, -1.0)
        U, S, V = tn.svd_symmetric(A)
        ref = np.sort(np.abs(np.linalg.eigvalsh(A)))[::-1]
        assert np.max(np.abs(S - ref)) <= 10 * n * eps * ref[0]
        assert np.max(np.abs(V.T @ V - np.eye(n))) <= 8 * np.sqrt(n) * eps
        assert np.max(np.abs(U.T @ U - np.eye(n))) <= 8 * np.sqrt(n) * eps
        assert np.max(np.abs(A @ V - U * S)) <= 10 * n * eps * ref[0]
