"""Stop rule of the FP32 eigenvalue sweeps (csrc/sweep_rule.h) on groups of clustered
eigenvalues, from the smallest that is solved by them (65 columns).

The sweeps are restated in NumPy: one-sided, FP32, the circle method's rounds,
rotations where |v_p·A·v_q| > 2ε₃₂·‖A‖_F.  Stopped by the rule, VᵀAV has to be
diagonal to what their result is documented to have, ~1e-6·‖A‖_F; the bound is 2e-6
(the threshold itself is 2.4e-7).  The rule is compiled by the host compiler.
"""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parent.parent / "tensornetworkad.jl_gb300" / "csrc"


@pytest.fixture(scope="module")
def last_rotations(tmp_path_factory):
    cxx = shutil.which("g++") or pytest.skip("no host C++ compiler")
    d = tmp_path_factory.mktemp("rule")
    (d / "m.cpp").write_text('#include "sweep_rule.h"\nextern "C" int rule(int n) { return tnad::eig_sweep_last(n); }\n')
    subprocess.run([cxx, "-std=c++17", "-shared", "-fPIC", f"-I{CSRC}", "-o", str(d / "m.so"), str(d / "m.cpp")], check=True)
    return C.CDLL(str(d / "m.so")).rule


def _rounds(n):
    N = n + (n & 1)
    for r in range(N - 1):
        pairs = [(N - 1, r)] + [((r + k) % (N - 1), (r - k + N - 1) % (N - 1)) for k in range(1, N // 2)]
        P, Q = np.array([sorted(p) for p in pairs]).T
        yield P[Q < n], Q[Q < n]


def _offdiagonal_after(A, last):
    """max |off-diagonal of VᵀAV|/‖A‖_F once a sweep made at most `last` rotations."""
    n = len(A)
    W, V = A.astype(np.float32), np.eye(n, dtype=np.float32)
    thr = np.float32(2 * np.finfo(np.float32).eps * np.linalg.norm(A))
    for _ in range(30):
        rotations = 0
        for P, Q in _rounds(n):
            a, b = (V[:, P] * W[:, P]).sum(0), (V[:, Q] * W[:, Q]).sum(0)
            g2 = (V[:, P] * W[:, Q]).sum(0) + (V[:, Q] * W[:, P]).sum(0)
            on = np.abs(g2) > 2 * thr
            P, Q, a, b, g2 = P[on], Q[on], a[on], b[on], g2[on]
            rotations += len(P)
            tau = (b - a) / g2
            t = np.copysign(1, tau) / (np.abs(tau) + np.sqrt(1 + tau * tau))
            c = 1 / np.sqrt(1 + t * t)
            for M in (W, V):
                x, y = M[:, P].copy(), M[:, Q].copy()
                M[:, P], M[:, Q] = c * x - c * t * y, c * t * x + c * y
        if rotations <= last:
            break
    X, _ = np.linalg.qr(V.astype(float))
    B = X.T @ A @ X
    return np.max(np.abs(B - np.diag(np.diag(B)))) / np.linalg.norm(A)


@pytest.mark.parametrize("n", [65, 80, 100, 130])
@pytest.mark.parametrize("graded", [False, True])
def test_groups_reach_the_documented_accuracy(last_rotations, n, graded):
    rng = np.random.default_rng(n)
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    lam = rng.uniform(-1, 1, n) * (10.0 ** (-3 * rng.random(n)) if graded else 1.0)
    A = (Q * lam) @ Q.T
    assert _offdiagonal_after(0.5 * (A + A.T), last_rotations(n)) <= 2e-6


def test_large_matrices_keep_their_rule(last_rotations):
    assert [last_rotations(n) for n in (257, 384, 1024)] == [16 * 257, 16 * 384, 16 * 1024]
