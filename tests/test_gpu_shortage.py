"""A batch without memory for what it prepares on first use (its plan, its records) fails as
such, and the next one, with memory again, runs as if nothing had been; an FP32 group on
records keeps no copies that only the row-by-row kernels read."""
import pytest

import oracle
import spike_pstrsv_b200 as spk
from cases import rel_err
from spike_pstrsv_b200 import group, synth

pytestmark = pytest.mark.gpu
TOL = 1e-12  # the repository's bound on x against the substitution


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("m,chain", [(40013, 1), (4003, 0)])  # 4,003 rows in exact mode: the partitions
def test_first_batch_without_memory(m, chain, mode):
    import torch

    k = 8
    A = synth.banded_lower(m, seed=5)
    S = spk.System().set_truncation(2.0 ** -60 if chain else -1.0).preproc(A.a, A.ia, A.ja, m, 8, "L")
    assert S.scalar("chain") == chain and S.scalar("sweep") == 1
    _, B = synth.make_rhs(A, seed=1, nrhs=k)
    dB = torch.from_numpy(B).cuda()
    dX = torch.zeros_like(dB)
    rows = S.scalar("chain_batch_rows")

    def solve():
        before = S.scalar("launches")
        S.solve_batch(dB, dX, mode=mode, tol=-1.0, maxit=2, want_resid=False)
        return S.scalar("launches") - before

    for _ in range(2 if chain else 1):  # the plan (chains), then the records
        S.debug_set("fail_allocs", 1)
        with pytest.raises(spk.SpkError) as e:
            solve()
        assert e.value.code == -3  # SPK_ERR_NOMEM
    launches = solve()
    if chain:
        assert launches == 1 + 2 * mode  # one launch a solve
        assert S.scalar("chain_batch_rows") == rows
    assert max(rel_err(x, oracle.sequential_solve(A, b, "L")) for x, b in zip(dX.cpu().numpy(), B)) <= TOL


def test_fp32_group_on_records_keeps_no_other_copies():
    import torch

    m, k = 20011, 8
    A = synth.banded_lower(m, seed=6)
    S = spk.System().set_truncation(-1.0).preproc(A.a, A.ia, A.ja, m, 8, "L")
    assert S.scalar("sweep") == 1
    _, B = synth.make_rhs(A, seed=1, nrhs=k)
    dB = torch.from_numpy(B).cuda()
    dX = torch.zeros_like(dB)
    st = torch.cuda.Stream()
    before = S.scalar("device_bytes")
    g = group.Group([S], [dB], [dX], mode=1, iters=1, stream=st.cuda_stream)
    # records and the diagonal; the sliced-ELL copy in FP32 would be 80 bytes a row more
    assert S.scalar("device_bytes") - before <= m * (190 + 8) + (1 << 16)
    g.solve()
    st.synchronize()
    assert max(rel_err(x, oracle.sequential_solve(A, b, "L")) for x, b in zip(dX.cpu().numpy(), B)) <= 1e-11
    g.close()
