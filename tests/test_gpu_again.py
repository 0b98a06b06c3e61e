"""A system preprocessed again and again: sizes that keep the memory of the records and of the
reduced solve's tables and sizes that do not, with and without each, solved against the
substitution."""
import pytest

import oracle
import spike_pstrsv_b200 as spk
from cases import rel_err
from spike_pstrsv_b200 import synth

pytestmark = pytest.mark.gpu
TOL = 1e-12  # the repository's bound on x against the substitution


@pytest.mark.parametrize("exact", [False, True])
def test_preprocessed_again(exact, monkeypatch):
    import torch

    S = spk.System()
    if exact:  # every reduced row kept
        S.set_truncation(-1.0)
    for m, records in ((20011, 1), (19003, 1), (20011, 1), (5003, 1), (19003, 1), (19003, 0), (19007, 1), (30011, 1)):
        monkeypatch.setenv("SPK_DISABLE_SWEEP", str(1 - records))
        monkeypatch.setenv("SPK_DISABLE_RING", str(1 - records))
        A = synth.banded_lower(m, seed=m + records)
        S.preproc(A.a, A.ia, A.ja, m, 9, "L")
        assert S.scalar("sweep") == records
        if exact or not records:  # else a small system's levels may be kept or not
            assert (S.scalar("reduced_ring") > 0) == (records == 1)
        _, B = synth.make_rhs(A, seed=1, nrhs=5)
        xs = [oracle.sequential_solve(A, b, "L") for b in B]
        assert rel_err(S.solve(B[0]), xs[0]) <= TOL
        dB = torch.from_numpy(B).cuda()
        for mode in (0, 1):
            dX = torch.zeros_like(dB)
            S.solve_batch(dB, dX, mode=mode, tol=-1.0, maxit=3, want_resid=False)
            assert max(rel_err(x, y) for x, y in zip(dX.cpu().numpy(), xs)) <= TOL, (m, mode)
