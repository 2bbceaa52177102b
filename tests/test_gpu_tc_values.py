"""Value ranges of the tensor-core products: the packing, slicing and epilogue
conversions are integer operations, which must agree with the conversion
instructions where an argument or a result is zero, subnormal or not finite.
A product with the identity (or with a power of two on its diagonal) shows each
stored element by itself."""
from __future__ import annotations

import ctypes as C
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

M, N = 200, 168  # neither a multiple of a tile; M·N·N above the tensor-core threshold


def _rel(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / np.linalg.norm(b))


def _entries(seed, lo, hi):
    rng = np.random.default_rng(seed)
    X = np.ldexp(rng.uniform(0.5, 1.0, (M, N)), rng.integers(lo, hi, (M, N))) * rng.choice([-1.0, 1.0], (M, N))
    X[3, :] = 0.0
    X[:, 5] = 0.0
    return np.asfortranarray(X)


@pytest.mark.parametrize("alpha,beta", [(1.0, 0.0), (-0.5, 0.0), (1.0, 1.0)])
@pytest.mark.parametrize("lo,hi", [(-40, 40), (-125, -60), (60, 126)])
def test_tf32x3_times_identity(tn, lo, hi, alpha, beta):
    X = _entries(1, lo, hi)
    C0 = _entries(2, lo, hi)
    got = tn.gemm(X, np.eye(N), alpha=alpha, beta=beta, Cin=C0, prec=tn._lib.PREC_TF32X3)
    # x − hi − lo: 11 bits each, 2^-22·|x|; FP32 accumulation of the two, another
    # 2^-22 with truncation; lo and sums below the FP32 normal range may be flushed
    tol = 2.0 ** -20 * (np.abs(X) + abs(beta) * 2.0 ** -30 * np.abs(C0)) + 2.0 ** -124
    assert np.all(np.abs(got - (alpha * X + beta * C0)) <= tol)


def test_tf32x3_keeps_non_finite_rows_apart(tn):
    X = _entries(3, -10, 10)
    X[7, 11] = np.nan
    X[9, 2] = np.inf
    X[11, 4] = 1e300  # above the FP32 range: the plane holds an infinity
    got = tn.gemm(X, np.eye(N), prec=tn._lib.PREC_TF32X3)
    bad = np.zeros(M, bool)
    bad[[7, 9, 11]] = True
    assert np.all(np.isfinite(got[~bad]))
    assert not np.any(np.isfinite(got[bad]).all(axis=1))


@pytest.mark.parametrize("alpha,beta", [(1.0, 0.0), (-0.5, 0.0), (1.0, 1.0)])
@pytest.mark.parametrize("K", [N, 680])
@pytest.mark.parametrize("row,col", [(0, 0), (500, 480), (-500, -560), (-1000, 0), (-700, 700)])
def test_fp64_tc_over_the_exponent_range(tn, K, row, col, alpha, beta):
    # rows near 2^row, columns near 2^col: results up to 2^980, down to subnormal
    rng = np.random.default_rng(4)
    A = np.asfortranarray(np.ldexp(rng.standard_normal((M, K)), row))
    A[3, :] = 0.0
    B = np.zeros((K, N), order="F")
    B[np.arange(N), np.arange(N)] = np.ldexp(1.0, col)
    C0 = np.asfortranarray(np.ldexp(rng.standard_normal((M, N)), row + col)) if row + col > -1000 else np.zeros((M, N))
    got = tn.gemm(A, B, alpha=alpha, beta=beta, Cin=C0, prec=tn._lib.PREC_FP64_TC)
    ref = alpha * np.ldexp(A[:, :N], col) + beta * C0
    # 2^-47 of the row and column scales, each a power of two up to twice the
    # largest entry (2^-45), once more for the digits' carries; FP64 roundings of C;
    # a subnormal result is rounded to its spacing, twice with alpha
    scale = np.ldexp(np.abs(A).max(axis=1, keepdims=True), col)
    tol = 2.0 ** -44 * (np.minimum(scale, 1e300) + 2.0 ** -5 * np.abs(C0)) + 2 * 5e-324
    assert np.all(np.abs(got - ref) <= tol)
    assert np.all(got[3] == (beta * C0)[3])


@pytest.mark.parametrize("ta,tb", [("N", "N"), ("T", "T")])
@pytest.mark.parametrize("M_,N_,K_", [(70, 130, 700), (1300, 70, 1500), (2500, 90, 600), (5000, 40, 65), (70, 40, 4000)])
def test_fp64_tc_slicing_blocks(tn, M_, N_, K_, ta, tb):
    """4, 8, 16 and 32 rows a block of the one-pass slicing, and the two-kernel form
    for an inner dimension that does not fit; rows over many binades."""
    rng = np.random.default_rng(K_)
    A = rng.standard_normal((M_, K_)) * np.ldexp(1.0, rng.integers(-60, 60, (M_, 1)))
    B = rng.standard_normal((K_, N_)) * np.ldexp(1.0, rng.integers(-60, 60, (1, N_)))
    A[7], B[:, 3] = 0.0, 0.0
    got = tn.gemm(np.asfortranarray(A.T if ta == "T" else A), np.asfortranarray(B.T if tb == "T" else B), ta, tb,
                  prec=tn._lib.PREC_FP64_TC)
    # each of the K products is off by 2^-47 of scales up to twice the largest entries
    tol = K_ * 2.0 ** -45 * np.abs(A).max(axis=1, keepdims=True) * np.abs(B).max(axis=0, keepdims=True)
    assert np.all(np.abs(got - A @ B) <= tol)
    assert not got[7].any() and not got[:, 3].any()


@pytest.mark.parametrize("batch,n_in,width,n_out", [(1, 7, 40, 33), (31, 32, 64, 129), (33, 81, 65, 64),
                                                    (130, 20, 600, 70)])
def test_network_gradient_edges(tn, batch, n_in, width, n_out):
    """Bias, ReLU and mask applied while a product is stored, with and without a
    split inner dimension, and bias gradients over batches around a warp."""
    from oracle import mlp_oracle as mo
    wl = importlib.import_module(tn.__name__ + ".learned")
    c, h = wl.ctx(), wl.L.VP()
    c.check(c.lib.tnad_mlp_create(c.h, n_in, width, n_out, 5, C.byref(h)))
    net = wl.WarmStartNet.__new__(wl.WarmStartNet)
    net.c, net.h, net.n_in, net.n_out, net.width = c, h, n_in, n_out, width
    net.n_params = int(c.lib.tnad_mlp_param_count(h))
    rng = np.random.default_rng(batch)
    rows, offs, _ = mo.layout(n_in, width, n_out)
    P = net.get_params().copy()
    for l in range(3):
        P[offs[l][1]:offs[l][1] + rows[l + 1]] = 0.1 * rng.standard_normal(rows[l + 1])
    net.set_params(P)
    X = np.asfortranarray(rng.standard_normal((n_in, batch)).astype(np.float32))
    Y = np.asfortranarray(rng.standard_normal((n_out, batch)).astype(np.float32))
    # the same BF16 roundings in the oracle: what differs are FP32 sums, and
    # through them single BF16 roundings (2^-9) and masks of activations near 0
    assert _rel(net.forward(X), mo.mlp_forward(P, X, n_in, width, n_out)[2]) <= 2e-3
    loss, G = net.gradient(X, Y)
    lo, Go = mo.mlp_gradient(P, X, Y, n_in, width, n_out)
    assert abs(loss - lo) <= 1e-4 * lo
    for l, (ow, ob) in enumerate(offs):
        nw = rows[l + 1] * rows[l]
        assert _rel(G[ow:ow + nw], Go[ow:ow + nw]) <= 5e-3
        assert _rel(G[ob:ob + rows[l + 1]], Go[ob:ob + rows[l + 1]]) <= 5e-3
    c.lib.tnad_mlp_free(h)
    net.h = wl.L.VP()
