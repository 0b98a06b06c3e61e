"""The chains' spikes: every chain's first significant row against scipy's triangular
solves, over one, two and four warps a chain, the ring full and not, few and many slots a
row, chains that end with the matrix."""
import numpy as np
import pytest

import spike_pstrsv_b200 as spk
from chain_ref import chain_plan, upper
from spike_pstrsv_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_row,band", [(1, 1), (3, 7), (8, 31), (8, 32), (12, 33), (16, 64), (40, 64), (8, 65), (17, 127),
                                          (30, 128), (63, 128)])
@pytest.mark.parametrize("uplo", ["L", "U"])
def test_first_significant_rows(per_row, band, uplo):
    m = 3 * 1024 + 77
    L = synth.banded_lower(m, per_row=per_row, band=band, seed=per_row * 1000 + band)
    a = L.a.copy()
    a[L.ia[1:] - 1] *= 32  # spikes that decay within a chain also where rows are long
    L = synth.CSR(m, L.ia, L.ja, a)
    A = L if uplo == "L" else synth.transpose(L)
    S = spk.System().preproc(A.a, A.ia, A.ja, m, 4, uplo)
    if np.diff(A.ia).max() > 65:  # more than 64 off-diagonals in a row (a column of L): no chains
        assert S.scalar("chain") == 0
        return
    assert S.scalar("chain") == 1
    want, reach = chain_plan(upper(A, uplo)[0], S.scalar("chain_rows"))
    assert S.scalar("chain_reach") == reach
    got = S.array("chain_tasks1").reshape(-1, 4)
    want = want.reshape(-1, 4)
    assert np.array_equal(got[:, :3], want[:, :3])
    # a row whose sum rounds to either side of 2^-60 would move f by one
    assert np.abs(got[:, 3] - want[:, 3]).max() <= 1


@pytest.mark.parametrize("m,per_row,band", [(2544, 16, 64), (5003, 8, 48), (9013, 24, 33)])
@pytest.mark.parametrize("uplo", ["L", "U"])
def test_starts_of_the_one_launch_tasks(m, per_row, band, uplo):
    """Every task's start is low enough: the spike of the rows walked before its own is negligible
    in the first `reach` of them."""
    import scipy.sparse.linalg as sla

    L = synth.banded_lower(m, per_row=per_row, band=band, seed=m)
    A = L if uplo == "L" else synth.transpose(L)
    S = spk.System().preproc(A.a, A.ia, A.ja, m, 4, uplo)
    assert S.scalar("launches_per_solve") == 1
    n, rows, walked, reach = m, S.scalar("rows"), S.scalar("chain_solve_rows"), S.scalar("chain_reach")
    tops = [min(a + rows, n) for a in range(0, n, rows)]
    warm = [w for w in range(0, n, 32) if sum(min(q + w, n) - a for a, q in zip(range(0, n, rows), tops)) == walked]
    assert len(warm) == 1
    U = upper(A, uplo)[0]
    for q in tops:
        h = q + warm[0]
        if h >= n:
            break
        R = U[q:h, h:]
        cols = np.unique(R.nonzero()[1])
        X = sla.spsolve_triangular(U[q:h, q:h].tocsr(), R[:, cols].toarray(), lower=False)
        assert np.abs(X[:reach]).sum(axis=1).max() <= 2.0 ** -60 * (1 + 1e-9)
