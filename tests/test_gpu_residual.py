"""The blocked FP64 residual of 2 to 32 columns: every column count's layout, sizes
around its 128-row blocks, bands within and past its rows in shared memory, 'L' and
'U', through the scaled residual that a batch reports: the batch's own solution (at
rounding level) and, for the value, an FP32 solution without corrections against
numpy."""
import numpy as np
import pytest

import spike_pstrsv_b200 as spk
from spike_pstrsv_b200 import synth

pytestmark = pytest.mark.gpu


def _scaled(A, X, B):
    rows = np.repeat(np.arange(A.m), np.diff(A.ia))
    anorm = np.bincount(rows, weights=np.abs(A.a), minlength=A.m).max()
    return max(np.abs(b - synth.spmv(A, x)).max() / (anorm * np.abs(x).max() + np.abs(b).max()) for x, b in zip(X, B))


@pytest.mark.parametrize("m,per_row,band", [(1, 1, 1), (127, 4, 20), (128, 16, 64), (129, 3, 7), (5003, 8, 120), (9001, 8, 700)])
@pytest.mark.parametrize("uplo", ["L", "U"])
def test_scaled_residual_of_batches(m, per_row, band, uplo):
    import torch

    L = synth.banded_lower(m, per_row=per_row, band=band, seed=m)
    A = L if uplo == "L" else synth.transpose(L)
    S = spk.System().preproc(A.a, A.ia, A.ja, m, min(4, m), uplo)
    for k in (2, 8, 9, 16, 17, 31, 32):
        _, B = synth.make_rhs(A, seed=k, nrhs=k)
        dB = torch.from_numpy(B).cuda()
        dX = torch.zeros_like(dB)
        _, r = S.solve_batch(dB, dX, mode=0)
        assert r <= 1e-15, k
        _, r = S.solve_batch(dB, dX, mode=1, tol=-1.0, maxit=0)  # FP32: a residual of about 1e-8
        want = _scaled(A, dX.cpu().numpy(), B)
        # both FP64, differing by summation order: 1e-16 of the terms, against 1e-8 of them
        assert r == pytest.approx(want, rel=1e-6, abs=1e-15), k
