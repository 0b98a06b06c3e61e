"""Forms of the reduced solve: systems of two halves that do not read each other, one of
them with a NaN in its right-hand side (a dense level holds both)."""
import numpy as np
import pytest

import oracle
import spike_pstrsv_b200 as spk
from cases import rel_err
from spike_pstrsv_b200 import synth

pytestmark = pytest.mark.gpu
TOL = 1e-12  # the repository's bound on x against the substitution


def _two_halves(m):
    """Upper CSR: rows of even 32-row tiles read even tiles only, odd ones odd; each row reads
    the row after it in its tile, and the first row and its own place of the tile two up."""
    rows = []
    for r in range(m):
        t = r - r % 32 + 64
        rows.append(sorted({c for c in (r + 1 if (r + 1) % 32 else m, t, r + 64) if c < m}))
    ia = np.cumsum([0] + [1 + len(c) for c in rows]).astype(np.int32)
    ja = np.array([c for r in range(m) for c in [r] + rows[r]], dtype=np.int32)
    return synth.CSR(m, ia, ja, np.where(ja == np.repeat(np.arange(m), np.diff(ia)), 2.0, 0.5))


@pytest.mark.parametrize("k,mode", [(1, 0), (3, 0), (8, 0), (20, 0), (8, 1)])
def test_a_nan_stays_in_its_half(k, mode):
    import torch

    m, P = 2048, 8
    A = _two_halves(m)
    S = spk.System().set_truncation(-1.0).preproc(A.a, A.ia, A.ja, m, P, "U")
    _, B = synth.make_rhs(A, seed=6, nrhs=k)
    xs = np.stack([oracle.sequential_solve(A, b, "U") for b in B])
    B[:, m - 40] = np.nan  # in an even tile of the last block
    even = (np.arange(m) // 32) % 2 == ((m - 40) // 32) % 2
    dB = torch.from_numpy(B).cuda()
    dX = torch.zeros_like(dB)
    S.solve_batch(dB, dX, mode=mode, tol=-1.0, maxit=3, want_resid=False)
    X = dX.cpu().numpy()
    assert max(rel_err(x[~even], y[~even]) for x, y in zip(X, xs)) <= TOL
