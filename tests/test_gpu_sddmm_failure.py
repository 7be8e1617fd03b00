"""The SDDMM block kernel's bounded wait: with the stall test on it waits on a
barrier that nothing arrives on and gives up after the poll limit.  The run
returns, the error flag is set, the scores of the block tiles are zeros (not
what the buffer held), those of the 1D tiles are right, and the next default
run is correct."""
import numpy as np
import pytest
import torch

import oracle.semantics as S
from stile_gb300 import device as D
from stile_gb300 import synthetic as syn
from stile_gb300.ops import DeviceSddmmPlan
from stile_gb300.planner import search_sddmm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nnz", [(300, 3000), (30_000, 600_000)])
@pytest.mark.parametrize("bf16", [False, True], ids=["fp32", "bf16"])
def test_scores_of_a_wait_that_runs_out_are_zeros(n, nnz, bf16):
    A = syn.sddmm_mask(n=n, target_nnz=nnz, seed=9)
    F = 72
    dev = D.build_sddmm_device(search_sddmm(A, F, max_bucket_size=32).tiles, A.shape, A.nnz)
    assert len(dev.blk_out)
    p = DeviceSddmmPlan(dev)
    g = torch.Generator("cuda").manual_seed(3)
    X, Y = (torch.randn(n, F, device="cuda", generator=g) for _ in range(2))
    if bf16:
        X, Y = X.to(torch.bfloat16), Y.to(torch.bfloat16)
    ref = S.sddmm_fp64(A, X.float().cpu().numpy(), Y.float().cpu().numpy())
    p.set_wait_policy(polls=1000, stall_test=True)
    one_d, blocks = np.setdiff1d(dev.remap, dev.blk_out), np.setdiff1d(dev.blk_out, dev.remap)
    assert len(blocks) and len(one_d)
    for given in (False, True):
        junk = torch.full((A.nnz,), 7.0, device="cuda")
        if not given:
            del junk        # the buffer that the run allocates holds it
        out = p.run(X, Y, junk if given else None)
        assert p.error_flag() != 0
        got = out.cpu().numpy()
        assert not got[blocks].any()
        assert S.rel_fro(got[one_d], ref[one_d]) <= 1e-5
    p.set_wait_policy()
    out = p.run(X, Y)
    assert p.error_flag() == 0
    assert S.rel_fro(out.cpu().numpy(), ref) <= 1e-5
