"""Decompositions and TRG from eight threads at once, a context each: their
grid-wide barriers, counters and workspaces are the context's own.  The results are
the bits of the same calls made alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _matrix(n):
    rng = np.random.default_rng(n)
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    A = (Q * (10.0 ** (-6.0 * np.arange(n) / n) * np.where(np.arange(n) % 3, 1.0, -1.0))) @ Q.T
    return 0.5 * (A + A.T)


def test_eight_contexts_give_the_bits_of_one(tn):
    rng = np.random.default_rng(0)
    mats = {n: _matrix(n) for n in (20, 33, 65, 130, 255, 300)}
    X, Y = rng.standard_normal((64, 4096)), rng.standard_normal((4096, 32))

    def results():
        out = {n: tn.svd_symmetric(A) for n, A in mats.items()}
        out["trg"] = [np.array(tn.trg_beta(0.44, chi, 4)) for chi in (5, 9, 16)]
        out["gemm"] = [tn.gemm(X, Y)]
        return out

    ref, wrong = results(), []

    def work():
        try:
            for _ in range(3):
                for key, arrays in results().items():
                    if not all(np.array_equal(a, b) for a, b in zip(arrays, ref[key])):
                        wrong.append(key)
        except Exception as e:  # noqa: BLE001 - reported by the assertion
            wrong.append(repr(e))

    threads = [threading.Thread(target=work) for _ in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
