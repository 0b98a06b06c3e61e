"""Rows without a column outside their 16-row tile keep what they do not depend on out:
work columns that phase 1 never writes (nothing depends on a block's first rows) filled
with NaN, and right-hand sides with an infinity or a NaN in a few rows of a factor
whose couplings end inside small blocks."""
import numpy as np
import pytest

import oracle
import spike_pstrsv_b200 as spk
from cases import rel_err
from spike_pstrsv_b200 import synth

pytestmark = pytest.mark.gpu
TOL = 1e-12  # the repository's bound on x against the substitution


def _upper(m, cols):
    """Upper CSR with diagonal 2 and 1/4 at the columns cols(r) of each row."""
    rows = [sorted(c for c in cols(r) if r < c < m) for r in range(m)]
    ia = np.cumsum([0] + [1 + len(c) for c in rows]).astype(np.int32)
    ja = np.array([c for r in range(m) for c in [r] + rows[r]], dtype=np.int32)
    return synth.CSR(m, ia, ja, np.where(ja == np.repeat(np.arange(m), np.diff(ia)), 2.0, 0.25))


def _unread_block_starts(m, block):
    """Chains i -> i + 1 inside each block, and one row near a block's end that reads row 30 of
    the next: nothing reads its first 30, and the other rows just below the bound have no
    column outside their tile."""
    return _upper(m, lambda r: ([r + 1] if (r + 1) % block else []) + ([r + 36] if r % block == block - 6 else []))


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("k", [1, 4, 13, 32])
def test_unwritten_work_rows(k, mode):
    import torch

    m, P = 1024, 4
    A = _unread_block_starts(m, m // P)
    S = spk.System().set_truncation(-1.0).preproc(A.a, A.ia, A.ja, m, P, "U")
    assert S.scalar("sweep") == 1 and S.scalar("chain") == 0
    _, B = synth.make_rhs(A, seed=3, nrhs=k)
    xs = [oracle.sequential_solve(A, b, "U") for b in B]
    ws = torch.full((S.workspace_bytes(mode=mode),), 255, dtype=torch.uint8, device="cuda")  # NaN in FP32 and FP64
    S.set_workspace(ws)
    X = torch.zeros(k, m, dtype=torch.float64, device="cuda")
    S.solve_batch(torch.from_numpy(B).cuda(), X, mode=mode, tol=-1.0, maxit=3, want_resid=False)
    assert max(rel_err(x, y) for x, y in zip(X.cpu().numpy(), xs)) <= TOL


def _blocks_of_eight(m):
    """Blocks of eight coupled rows; the last 200 rows couple 40 apart, so that the window is
    wider than a tile."""
    return _upper(m, lambda r: [c for c in (r + 1, r + 3) if c // 8 == r // 8] + ([r + 40] if r >= m - 200 else []))


@pytest.mark.parametrize("uplo", ["L", "U"])
@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("k,mode", [(0, 0), (5, 0), (12, 0), (32, 0), (5, 1), (32, 1)])  # 0: the plain solve
def test_non_finite_stay_in_their_tile(uplo, exact, k, mode):
    import torch

    m = 20000  # whole 32-row tiles: blocks lie inside tiles in either order
    A = _blocks_of_eight(m)
    if uplo == "L":
        A = synth.transpose(A)
    S = spk.System()
    if exact:
        S.set_truncation(-1.0)
    S.preproc(A.a, A.ia, A.ja, m, 7, uplo)
    assert S.scalar("sweep") == 1
    _, B = synth.make_rhs(A, seed=4, nrhs=max(k, 1))
    xs = np.stack([oracle.sequential_solve(A, b, uplo) for b in B])
    far = np.ones(m, bool)
    for r, v in ((5003, np.inf), (9000, np.nan), (15007, -np.inf)):
        B[:, r] = v
        far[max(0, r - 31):r + 32] = False  # rows that may share a tile with it
    dB = torch.from_numpy(B).cuda()
    dX = torch.zeros_like(dB)
    if k:
        S.solve_batch(dB, dX, mode=mode, tol=-1.0, maxit=3, want_resid=False)
    else:
        S.solve_device(dB.data_ptr(), dX.data_ptr(), torch.cuda.current_stream().cuda_stream)
    X = dX.cpu().numpy()
    assert max(rel_err(x[far], y[far]) for x, y in zip(X, xs)) <= TOL
