"""The operator's backward sets the row runs whatever value-gradient mode its
plans had."""
import numpy as np
import pytest
import torch

from stile_gb300 import _lib
from stile_gb300 import synthetic as syn
from stile_gb300.api import PlanConfig, plan_spmm

pytestmark = pytest.mark.gpu


def _operands(A, N):
    rng = np.random.default_rng(17)
    B = rng.standard_normal((A.shape[1], N)).astype(np.float32)
    dC = rng.standard_normal((A.shape[0], N)).astype(np.float32)
    return torch.as_tensor(B, device="cuda"), torch.as_tensor(dC, device="cuda")


@pytest.mark.parametrize("backward", ["fused", "separate"])
def test_operator_backward_sets_the_row_runs(backward):
    """A mode set at the C entry point between two backwards."""
    A = syn.community_graph(n=2048, target_nnz=30000, seed=15, max_deg=256)
    op = plan_spmm(A, 64, PlanConfig(backward=backward))
    Bt, dCt = _operands(A, 64)
    _, want = op.backward(dCt, Bt)
    for h in (op.handle, op.transposed[0].handle):
        _lib.check(h.lib.stile_spmm_plan_set_dvals_mode(h.handle, 1), "stile_spmm_plan_set_dvals_mode")
    _, got = op.backward(dCt, Bt)
    assert torch.equal(got, want)
