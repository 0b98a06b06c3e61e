"""One-right-hand-side solves on 16-row records: tiles cut by partition bounds and
by the matrix's end, rows with more off-diagonals than the common slots, columns
beyond 128 rows (two-byte offsets) up to the window's limit and past it, and
matrices whose tile inverses grow too much for the records, on the chain path,
the partition path and in exact mode, against the sequential substitution and
the row-by-row kernels."""
import numpy as np
import pytest

import oracle
import spike_pstrsv_b200 as spk
from cases import rel_err
from spike_pstrsv_b200 import synth

pytestmark = pytest.mark.gpu
TOL = 1e-12  # the repository's bound on x against the substitution


def _solve(A, P, uplo, b, exact):
    S = spk.System()
    if exact:
        S.set_truncation(-1.0)
    S.preproc(A.a, A.ia, A.ja, A.m, P, uplo)
    return S, S.solve(b)


def _check(L, P, want=1, monkeypatch=None):
    for uplo, A in (("L", L), ("U", synth.transpose(L))):
        _, b = synth.make_rhs(A, seed=7)
        xs = oracle.sequential_solve(A, b, uplo)
        for exact in (False, True):
            S, x = _solve(A, P, uplo, b, exact)
            assert S.scalar("sweep") == want, (uplo, exact)
            assert rel_err(x, xs) <= TOL, (uplo, exact)
            if monkeypatch is not None:
                monkeypatch.setenv("SPK_DISABLE_SWEEP", "1")
                T, y = _solve(A, P, uplo, b, exact)
                monkeypatch.delenv("SPK_DISABLE_SWEEP")
                assert T.scalar("sweep") == 0
                assert rel_err(x, y) <= 1e-14, (uplo, exact)  # a few roundings of either order


def _with(m, entries, base):
    """base plus off-diagonals (row, col, value) below the diagonal."""
    rows = [dict(zip(base.ja[base.ia[i]:base.ia[i + 1]].tolist(), base.a[base.ia[i]:base.ia[i + 1]].tolist()))
            for i in range(m)]
    for r, c, v in entries:
        rows[r][c] = v
        rows[r][r] += abs(v)
    ia = np.cumsum([0] + [len(r) for r in rows]).astype(np.int32)
    ja = np.array([c for r in rows for c in sorted(r)], dtype=np.int32)
    a = np.array([r[c] for r in rows for c in sorted(r)])
    return synth.CSR(m, ia, ja, a)


@pytest.mark.parametrize("m,P", [(1, 1), (15, 1), (16, 2), (17, 2), (63, 3), (64, 4), (65, 7), (1000, 13), (4099, 37)])
def test_cut_tiles(m, P, monkeypatch):
    """Sizes around a tile and partitions that cut tiles everywhere."""
    _check(synth.banded_lower(m, per_row=5, band=24, seed=m), P, monkeypatch=monkeypatch)


@pytest.mark.parametrize("per_row,band", [(1, 1), (4, 8), (9, 40), (16, 64), (30, 100), (41, 128)])
def test_slot_classes(per_row, band, monkeypatch):
    _check(synth.banded_lower(9013, per_row=per_row, band=band, seed=band), 11, monkeypatch=monkeypatch)


def test_long_rows_take_extra_slots(monkeypatch):
    """A few rows with many more off-diagonals than the rest, and one with none."""
    m = 6007
    rng = np.random.default_rng(1)
    base = synth.banded_lower(m, per_row=3, band=30, seed=2)
    extra = [(r, int(c), float(rng.standard_normal() / 16)) for r in (200, 2999, 3000, 5990)
             for c in rng.choice(np.arange(r - 120, r), size=rng.integers(20, 90), replace=False)]
    _check(_with(m, extra, base), 9, monkeypatch=monkeypatch)


@pytest.mark.parametrize("reach,want", [(127, 1), (128, 1), (129, 1), (1000, 1), (8176, 1), (8177, 0)])
def test_reach(reach, want):
    """The widest column distance: one-byte offsets, two-byte offsets, past the window."""
    m = 3 * reach + 1001
    base = synth.banded_lower(m, per_row=2, band=16, seed=3)
    _check(_with(m, [(r, r - reach, 0.25) for r in range(reach, m, 97)], base), 3, want)


def test_growing_inverses_keep_the_row_kernels():
    """Off-diagonals of size 1 beside unit diagonals: the tiles' inverses grow like 2^15."""
    m = 2000
    A = synth.banded_lower(m, per_row=8, band=16, seed=4)
    a = A.a.copy()
    a[A.ia[1:] - 1] = 1.0
    off = np.ones(len(a), bool)
    off[A.ia[1:] - 1] = False
    a[off] = -0.9
    A = synth.CSR(m, A.ia, A.ja, a)
    S = spk.System().preproc(A.a, A.ia, A.ja, m, 4, "L")
    assert S.scalar("sweep") == 0
