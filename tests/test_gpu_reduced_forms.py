"""Forms of the reduced solve: systems of two halves that do not read each other, one of
them with a NaN in its right-hand side (a dense level holds both), and the one-CTA solve of
systems whose levels span more unknowns than shared memory holds; levels whose kept rows
are mostly zeros while the dropped ones are full."""
import numpy as np
import pytest

import oracle
import spike_pstrsv_b200 as spk
from cases import rel_err
from spike_pstrsv_b200 import group, synth
from test_gpu_sweep import _with

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


@pytest.mark.parametrize("m,per_row,band,P", [(4003, 3, 8, 4), (20011, 16, 64, 40)])
@pytest.mark.parametrize("uplo", ["L", "U"])
@pytest.mark.parametrize("records", [True, False])
def test_one_cta(m, per_row, band, P, uplo, records, monkeypatch):
    """Forced, on either kind of phase kernels; FP64 and FP32 columns, powers of two and others."""
    import torch

    monkeypatch.setenv("SPK_DISABLE_RING", "1")
    if not records:
        monkeypatch.setenv("SPK_DISABLE_SWEEP", "1")
    L = synth.banded_lower(m, per_row=per_row, band=band, seed=m)
    A = L if uplo == "L" else synth.transpose(L)
    S = spk.System().set_truncation(-1.0).preproc(A.a, A.ia, A.ja, m, P, uplo)
    assert S.scalar("reduced_ring") == 0 and S.scalar("kept_reduced_rows") > 0
    _, B = synth.make_rhs(A, seed=5, nrhs=32)
    xs = np.stack([oracle.sequential_solve(A, b, uplo) for b in B])
    assert rel_err(S.solve(B[0]), xs[0]) <= TOL
    for k in (1, 2, 3, 4, 8, 13, 16, 31, 32):
        dB = torch.from_numpy(B[:k]).cuda()
        for mode in (0, 1):
            dX = torch.zeros_like(dB)
            S.solve_batch(dB, dX, mode=mode, tol=-1.0, maxit=3, want_resid=False)
            assert max(rel_err(x, y) for x, y in zip(dX.cpu().numpy(), xs)) <= TOL, (k, mode)


def test_levels_wider_than_shared_memory():
    """300 partitions with 64 dependents each, and a row near the end that reads one near the
    start: its level spans more unknowns than a column's ring (16,384) holds."""
    import torch

    m, P = 40011, 300
    A = _with(m, [(m - 200, 5, 0.25)], synth.banded_lower(m, seed=3))
    S = spk.System().set_truncation(-1.0).preproc(A.a, A.ia, A.ja, m, P, "L")
    assert S.scalar("reduced_ring") == 0 and S.scalar("kept_reduced_rows") > 16384
    _, B = synth.make_rhs(A, seed=8, nrhs=5)
    xs = np.stack([oracle.sequential_solve(A, b, "L") for b in B])
    assert rel_err(S.solve(B[0]), xs[0]) <= TOL
    dB = torch.from_numpy(B).cuda()
    for mode in (0, 1):
        dX = torch.zeros_like(dB)
        S.solve_batch(dB, dX, mode=mode, tol=-1.0, maxit=3, want_resid=False)
        assert max(rel_err(x, y) for x, y in zip(dX.cpu().numpy(), xs)) <= TOL, mode


def _sparse_kept_full_dropped(m, block):
    """Upper CSR, blocks of 256 rows.  Even rows of the first 64 read their own place a block up
    (one column each, 1/2); odd ones read a chain through the rest of the block that ends in every
    odd row of the next (32 columns each, 1/4 a step: below 2^-60 after 30)."""
    ia, ja, a = [0], [], []
    for r in range(m):
        o, up = r % block, r - r % block + block
        if o < 64 and o % 2 == 0:
            cols, v = [r + block], 0.5
        elif o < 64:
            cols, v = [up - block + 64], 0.25
        elif o < block - 1:
            cols, v = [r + 1], 0.25
        else:
            cols, v = list(range(up + 1, up + 64, 2)), 0.25 / 32
        cols = [c for c in cols if c < m]
        ja += [r] + cols
        a += [1.0] + [v] * len(cols)
        ia.append(len(ja))
    return synth.CSR(m, np.array(ia, np.int32), np.array(ja, np.int32), np.array(a))


@pytest.mark.parametrize("k", [1, 8])
def test_dropped_rows_do_not_make_a_level_dense(k):
    import torch

    m, block = 2560, 256
    A = _sparse_kept_full_dropped(m, block)
    S = spk.System().preproc(A.a, A.ia, A.ja, m, m // block, "U")
    # 32 kept rows a level of one nonzero each, over 63 columns; the dropped ones have 32 each
    assert S.scalar("chain") == 0 and S.scalar("reduced_ring") > 0
    assert 0 < S.scalar("kept_reduced_rows") <= 32 * (m // block - 2)
    assert S.scalar("reduced_dense") == 0
    _, B = synth.make_rhs(A, seed=12, nrhs=k)
    dB = torch.from_numpy(B).cuda()
    dX = torch.zeros_like(dB)
    S.solve_batch(dB, dX, mode=0, tol=-1.0, maxit=0, want_resid=False)
    assert max(rel_err(x, oracle.sequential_solve(A, b, "U")) for x, b in zip(dX.cpu().numpy(), B)) <= TOL


@pytest.mark.parametrize("k", [1, 4])
def test_group_of_small_and_large_rings(k):
    """One launch for a member with many CTAs on a small ring and one with a ring that fills shared memory."""
    import torch

    mats = [(synth.banded_lower(20011, per_row=16, band=250, seed=1), 30),
            (synth.banded_lower(9001, per_row=60, band=1500, seed=2), 4)]
    systems = [spk.System().set_truncation(-1.0).preproc(A.a, A.ia, A.ja, A.m, P, "L") for A, P in mats]
    assert 256 < systems[0].scalar("reduced_ring") < 1024 and systems[1].scalar("reduced_ring") > 2048
    rhs = [synth.make_rhs(A, seed=3, nrhs=k)[1] for A, _ in mats]
    B = [torch.from_numpy(b).cuda() for b in rhs]
    X = [torch.zeros_like(b) for b in B]
    st = torch.cuda.Stream()
    g = group.Group(systems, B, X, mode=0, iters=0, stream=st.cuda_stream)
    g.solve()
    st.synchronize()
    for (A, _), b, x in zip(mats, rhs, X):
        assert max(rel_err(u, oracle.sequential_solve(A, v, "L")) for u, v in zip(x.cpu().numpy(), b)) <= TOL
    g.close()
