"""The reduced solve on a cluster of CTAs: dense and CSR coefficients, one to many
levels, column blocks of 8/4/2/1 and their remainders, FP64 and FP32 work
columns, against the sequential substitution.  Nothing truncated, so every
reduced row is kept."""
import numpy as np
import pytest

import oracle
import spike_pstrsv_b200 as spk
from cases import rel_err
from spike_pstrsv_b200 import synth

pytestmark = pytest.mark.gpu
TOL = 1e-12  # the repository's bound on x against the substitution


def _check(A, P, uplo, ks):
    import torch

    S = spk.System()
    S.set_truncation(-1.0)
    S.preproc(A.a, A.ia, A.ja, A.m, P, uplo)
    Xt, B = synth.make_rhs(A, seed=5, nrhs=max(ks))
    xs = np.stack([oracle.sequential_solve(A, b, uplo) for b in B])
    assert rel_err(S.solve(B[0]), xs[0]) <= TOL
    for k in ks:
        dB = torch.from_numpy(B[:k].copy()).cuda()
        dX = torch.zeros_like(dB)
        S.solve_batch(dB, dX, mode=0)
        X = dX.cpu().numpy()
        assert max(rel_err(X[i], xs[i]) for i in range(k)) <= TOL, k
        dX.zero_()
        _, r = S.solve_batch(dB, dX, mode=1, tol=1e-12, maxit=8)
        assert r <= TOL, k


# partitions: one level, two, many; bands: levels of 1 row up to more rows than a
# cluster has warps, columns below and above what is loaded ahead (256)
@pytest.mark.parametrize("m,per_row,band,P", [(4001, 1, 1, 3), (4003, 3, 8, 4), (20011, 16, 64, 40),
                                              (30011, 8, 250, 30), (30011, 40, 300, 8)])
@pytest.mark.parametrize("uplo", ["L", "U"])
def test_banded_levels(m, per_row, band, P, uplo):
    L = synth.banded_lower(m, per_row=per_row, band=band, seed=m)
    _check(L if uplo == "L" else synth.transpose(L), P, uplo, (1, 2, 3, 7, 8, 16, 19, 32))


def test_many_partitions_fill_the_wide_batch():
    """Enough partitions for the one-pass solve of 17 to 32 columns (a partial
    last block of eight)."""
    _check(synth.banded_lower(120011, seed=3), 320, "L", (17, 24, 31))


@pytest.mark.parametrize("n,P", [(12, 4), (20, 8)])
def test_sparse_levels(n, P):
    """A 3-D factor: levels of n^2 rows whose spikes are mostly zero (CSR
    coefficients), rings up to 4,096 unknowns."""
    L = synth.ic0_laplace3d_lower(n)
    _check(L, P, "L", (1, 4, 8, 13))
    _check(synth.transpose(L), P, "U", (1, 2, 16))
