"""Solves whose x is the array of b: one column and many, on tasks short and long, chain
plans, partitions and compacted systems, several times each, against the sequential
substitution.  A task that read rows another one has stored would depend on timing and
mostly come out right, so the launches are counted too: one launch alone holds such tasks."""
import numpy as np
import pytest

import oracle
import spike_pstrsv_b200 as spk
from cases import rel_err
from spike_pstrsv_b200 import synth

pytestmark = pytest.mark.gpu
TOL = 1e-12  # the repository's bound on x against the substitution
TIMES = 10


@pytest.mark.parametrize("m,per_row,band,P", [(1201, 6, 24, 3), (5003, 8, 48, 4), (262147, 16, 64, 64)])
@pytest.mark.parametrize("uplo", ["L", "U"])
@pytest.mark.parametrize("compact", [False, True])
def test_same_array(m, per_row, band, P, uplo, compact):
    import torch

    L = synth.banded_lower(m, per_row=per_row, band=band, seed=m)
    A = L if uplo == "L" else synth.transpose(L)
    S = spk.System().preproc(A.a, A.ia, A.ja, m, P, uplo)
    if compact:
        if not S.scalar("chain"):
            pytest.skip("only chain-solved systems are compacted")
        S.compact()
    k = 32 if m < 10000 else 18
    _, B = synth.make_rhs(A, seed=11, nrhs=k)
    xs = np.stack([oracle.sequential_solve(A, b, uplo) for b in B])
    dB = torch.from_numpy(B).cuda()
    st = torch.cuda.current_stream().cuda_stream

    def launched(call, *args, **kw):
        before = S.scalar("launches")
        call(*args, **kw)
        return S.scalar("launches") - before

    for _ in range(TIMES):
        v = dB[0].clone()
        assert launched(S.solve_device, v.data_ptr(), v.data_ptr(), st) >= 2
        assert rel_err(v.cpu().numpy(), xs[0]) <= TOL
    for cols in (2, 9, k):
        for _ in range(TIMES):
            V = dB[:cols].clone()
            assert launched(S.solve_batch, V, V, mode=0, tol=-1.0, maxit=0, want_resid=False) >= 2
            assert max(rel_err(x, y) for x, y in zip(V.cpu().numpy(), xs)) <= TOL, cols
    # FP32 without corrections (those need b): 1e-5 covers FP32 roundings over a decay length
    V = dB.clone()
    S.solve_batch(V, V, mode=1, tol=-1.0, maxit=0, want_resid=False)
    assert max(rel_err(x, y) for x, y in zip(V.cpu().numpy(), xs)) <= 1e-5
    v = B[0].copy()  # host arrays
    S.solve(v, v)
    assert rel_err(v, xs[0]) <= TOL


def test_columns_between_each_other():
    """B and X as alternate columns of one array: no column is shared."""
    import torch

    m, k = 5003, 8
    A = synth.banded_lower(m, per_row=8, band=48, seed=m)
    S = spk.System().preproc(A.a, A.ia, A.ja, m, 4, "L")
    _, B = synth.make_rhs(A, seed=2, nrhs=k)
    both = torch.zeros(k, 2, m, dtype=torch.float64, device="cuda")
    both[:, 0] = torch.from_numpy(B).cuda()
    S.solve_batch(both[:, 0], both[:, 1], mode=0)
    X = both[:, 1].cpu().numpy()
    assert max(rel_err(x, oracle.sequential_solve(A, b, "L")) for x, b in zip(X, B)) <= TOL
    assert np.array_equal(both[:, 0].cpu().numpy(), B)
