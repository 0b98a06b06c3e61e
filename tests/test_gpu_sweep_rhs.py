"""Batched solves on 16-row records: every shape of the columns (1 to 32) on the chain
path (one launch) and the partition path (cut tiles, reduced system, kept rows),
rows with more off-diagonals than the common groups, bands below a tile's 16 rows
and beyond 128, after compaction, FP64 against the sequential substitution of every
column and FP32 + refinement to the repository's residual bound."""
import numpy as np
import pytest

import oracle
import spike_pstrsv_b200 as spk
from cases import rel_err
from spike_pstrsv_b200 import synth
from test_gpu_sweep import _with

pytestmark = pytest.mark.gpu
TOL = 1e-12  # the repository's bound on x against the substitution


def _check(A, P, uplo, ks, exact=False, path=None, compact=False):
    import torch

    S = spk.System()
    if exact:
        S.set_truncation(-1.0)
    S.preproc(A.a, A.ia, A.ja, A.m, P, uplo)
    assert S.scalar("sweep") == 1
    if compact:
        S.compact()
    if path is not None and S.scalar("chain"):
        S.tune("batch_path", path)
    _, B = synth.make_rhs(A, seed=9, nrhs=max(ks))
    xs = np.stack([oracle.sequential_solve(A, b, uplo) for b in B])
    for k in ks:
        dB = torch.from_numpy(B[:k].copy()).cuda()
        dX = torch.full_like(dB, float("nan"))
        S.solve_batch(dB, dX, mode=0)
        X = dX.cpu().numpy()
        assert max(rel_err(X[i], xs[i]) for i in range(k)) <= TOL, (k, "fp64")
        dX.fill_(float("nan"))
        _, r = S.solve_batch(dB, dX, mode=1, tol=1e-12, maxit=8)
        assert r <= TOL, (k, "fp32")
        assert max(rel_err(dX.cpu().numpy()[i], xs[i]) for i in range(k)) <= TOL, (k, "fp32")


@pytest.mark.parametrize("m,per_row,band", [(40013, 16, 64), (30001, 3, 7), (20011, 25, 128)])
@pytest.mark.parametrize("uplo", ["L", "U"])
def test_chain_path(m, per_row, band, uplo):
    L = synth.banded_lower(m, per_row=per_row, band=band, seed=m)
    _check(L if uplo == "L" else synth.transpose(L), 9, uplo, (1, 2, 8, 9, 16, 17, 32, 35), path=1)


@pytest.mark.parametrize("m,per_row,band,P", [(65, 5, 24, 7), (1000, 1, 1, 13), (9013, 8, 100, 11), (20011, 8, 250, 23)])
@pytest.mark.parametrize("uplo", ["L", "U"])
@pytest.mark.parametrize("exact", [False, True])
def test_partition_path(m, per_row, band, P, uplo, exact, monkeypatch):
    monkeypatch.setenv("SPK_CHAIN_BATCH", "0")
    L = synth.banded_lower(m, per_row=per_row, band=band, seed=m)
    _check(L if uplo == "L" else synth.transpose(L), P, uplo, (2, 7, 13, 32), exact=exact)


def test_long_rows_and_compaction():
    m = 20011
    rng = np.random.default_rng(1)
    base = synth.banded_lower(m, per_row=3, band=30, seed=2)
    extra = [(r, int(c), float(rng.standard_normal() / 16)) for r in (200, 9999, 10000, 19990)
             for c in rng.choice(np.arange(r - 120, r), size=rng.integers(20, 90), replace=False)]
    A = _with(m, extra, base)
    _check(A, 9, "L", (3, 12, 32), path=1)
    _check(synth.transpose(A), 9, "U", (5, 20), path=1, compact=True)


def test_wide_window():
    """Columns 1,000 rows away: the window of 8 columns fits, that of 32 does not."""
    m = 9001
    base = synth.banded_lower(m, per_row=2, band=16, seed=3)
    _check(_with(m, [(r, r - 1000, 0.25) for r in range(1000, m, 7)], base), 3, "L", (2, 8, 16, 32))
