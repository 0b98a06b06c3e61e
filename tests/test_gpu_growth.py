"""Tiles whose inverses grow: up to the records' limit the product with the inverse is no
further from the exact solution than the row-by-row kernels, past it those run."""
import numpy as np
import pytest

import oracle
import spike_pstrsv_b200 as spk
from cases import rel_err
from spike_pstrsv_b200 import synth

pytestmark = pytest.mark.gpu
TOL = 1e-12  # the repository's bound on x against the substitution
LIMIT = 4.0


def _inverse(T):
    W = np.eye(16)
    for i in range(1, 16):
        for p in range(i - 1, -1, -1):
            W[p, i] = -(T[p, i] + T[p, p + 1:i] @ W[p + 1:i, i])
    return W


def _blocks(m, growth, seed):
    """m / 16 random unit upper triangles of 16 rows, each scaled so that the largest absolute row
    sum of its inverse is `growth`, their rows scaled by random diagonals."""
    rng = np.random.default_rng(seed)
    ia, ja, a = [0], [], []
    for j in range(0, m, 16):
        T = np.triu(rng.standard_normal((16, 16)), 1) * (rng.random((16, 16)) < rng.choice([0.25, 0.5, 1.0]))
        lo, hi = 0.0, 8.0
        while hi - lo > 1e-13:
            mid = (lo + hi) / 2
            lo, hi = (mid, hi) if np.abs(_inverse(mid * T)).sum(1).max() < growth else (lo, mid)
        for i in range(16):
            d = rng.uniform(0.5, 2.0)
            cols = np.flatnonzero(T[i])
            ja += [j + i] + (j + cols).tolist()
            a += [d] + (lo * T[i, cols] * d).tolist()
            ia.append(len(ja))
    return synth.CSR(m, np.array(ia, np.int32), np.array(ja, np.int32), np.array(a))


def _exact(A, b):
    x = b.astype(np.longdouble)
    for i in range(A.m - 1, -1, -1):
        e0, e1 = A.ia[i], A.ia[i + 1]
        x[i] = (x[i] - A.a[e0 + 1:e1].astype(np.longdouble) @ x[A.ja[e0 + 1:e1]]) / np.longdouble(A.a[e0])
    return x


def _solved(A, B, k):
    import torch

    S = spk.System().preproc(A.a, A.ia, A.ja, A.m, 4, "U")
    dB = torch.from_numpy(B[:k]).cuda()
    dX = torch.zeros_like(dB)
    S.solve_batch(dB, dX, mode=0)
    return S.scalar("sweep"), dX.cpu().numpy(), S.solve(B[0])


@pytest.mark.parametrize("growth", [2.0, 3.9])
def test_errors_below_the_limit(growth, monkeypatch):
    m, k = 8192, 4
    A = _blocks(m, growth, 1)
    _, B = synth.make_rhs(A, seed=2, nrhs=k)
    ref = np.stack([_exact(A, b) for b in B])
    on, X, x = _solved(A, B, k)
    monkeypatch.setenv("SPK_DISABLE_SWEEP", "1")
    off, Y, y = _solved(A, B, k)
    assert (on, off) == (1, 0)

    def mean(v, r):  # each block's largest error, relative to its largest value, over all blocks
        e = np.abs(v - r).astype(float).reshape(-1, 16).max(1)
        return (e / np.abs(r).astype(float).reshape(-1, 16).max(1)).mean()

    # the same recurrences in numpy: the product's mean error is 0.5 to 0.7 of the substitution's here
    assert mean(X, ref) <= mean(Y, ref)
    assert mean(x, ref[0]) <= mean(y, ref[0])


@pytest.mark.parametrize("growth,want", [(LIMIT - 0.1, 1), (LIMIT + 0.1, 0), (12.0, 0)])
def test_both_sides_of_the_limit(growth, want):
    m, k = 2048, 9
    A = _blocks(m, growth, 3)
    _, B = synth.make_rhs(A, seed=4, nrhs=k)
    on, X, x = _solved(A, B, k)
    assert on == want
    xs = [oracle.sequential_solve(A, b, "U") for b in B]
    assert rel_err(x, xs[0]) <= TOL
    assert max(rel_err(u, v) for u, v in zip(X, xs)) <= TOL
