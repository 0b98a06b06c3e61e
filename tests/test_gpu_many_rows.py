"""A batch of more rows than 2^32 / 2,185 tiles of 16: its records' offsets still fit 32 bits."""
import numpy as np
import pytest

import oracle
import spike_pstrsv_b200 as spk
from cases import rel_err
from spike_pstrsv_b200 import synth

pytestmark = pytest.mark.gpu
TOL = 1e-12  # the repository's bound on x against the substitution


def test_records_of_many_rows():
    import torch

    m, k = 31_500_011, 2
    ia = np.minimum(2 * np.arange(m + 1, dtype=np.int64), 2 * m - 1).astype(np.int32)  # row r: r, r + 1
    ja = (np.arange(2 * m - 1) // 2 + np.arange(2 * m - 1) % 2).astype(np.int32)
    a = np.where(np.arange(2 * m - 1) % 2 == 0, 2.0, 0.5)
    A = synth.CSR(m, ia, ja, a)
    S = spk.System().preproc(A.a, A.ia, A.ja, m, 1024, "U")
    assert S.scalar("chain") == 1 and S.scalar("sweep") == 1
    B = np.random.default_rng(0).uniform(-1, 1, (k, m))
    dB = torch.from_numpy(B).cuda()
    dX = torch.zeros_like(dB)
    before = S.scalar("launches")
    S.solve_batch(dB, dX, mode=0, tol=-1.0, maxit=0, want_resid=False)
    assert S.scalar("launches") - before == 1  # one launch on records
    X = dX.cpu().numpy()
    assert max(rel_err(x, oracle.sequential_solve(A, b, "U")) for x, b in zip(X, B)) <= TOL
    S.close()
