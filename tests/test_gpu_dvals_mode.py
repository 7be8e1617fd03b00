"""Value gradients of the tensor-tile nonzeros on the tensor cores
(stile_spmm_plan_set_dvals_mode 1) in the fused backward, and the operator's
backward, which sets the row runs whatever the plan's mode was."""
import numpy as np
import pytest
import torch

import oracle.semantics as S
from stile_gb300 import _lib
from stile_gb300 import device as D
from stile_gb300 import synthetic as syn
from stile_gb300.api import PlanConfig, plan_spmm

pytestmark = pytest.mark.gpu


def _operands(A, N):
    rng = np.random.default_rng(17)
    B = rng.standard_normal((A.shape[1], N)).astype(np.float32)
    dC = rng.standard_normal((A.shape[0], N)).astype(np.float32)
    return B, dC, torch.as_tensor(B, device="cuda"), torch.as_tensor(dC, device="cuda")


@pytest.mark.parametrize("N", [33, 64, 128, 129, 200])
@pytest.mark.parametrize("mode", [D.TC_BF16, D.TC_SPLIT_BF16], ids=["bf16", "split"])
@pytest.mark.parametrize("pattern", ["graph", "rect"])
def test_fused_backward_with_tensor_core_value_gradients(pattern, mode, N):
    """The transposed plan's backward with mode 1: hi + lo bf16 products for
    its tensor tiles' gradients (within 1e-5), both where one feature pass
    gives dB and the row tiles' gradients and where the width takes two."""
    A = (syn.community_graph(n=2048, target_nnz=30000, seed=15, max_deg=256) if pattern == "graph"
         else syn.power_law_rows(3000, 2200, min_len=2, max_len=300, seed=16))
    op = plan_spmm(A, N, PlanConfig(tc_mode=mode))
    opT, _ = op.transposed
    assert opT.handle.has_tensor_tiles
    B, dC, Bt, dCt = _operands(A, N)
    opT.handle.set_dvals_mode(2)
    _, runs = opT.handle.backward(dCt, Bt)
    opT.handle.set_dvals_mode(1)
    dB, dv = opT.handle.backward(dCt, Bt)
    assert opT.handle.error_flag() == 0
    assert not torch.equal(dv, runs)      # the tensor cores' products, not the row runs'
    assert S.rel_fro(dv.cpu().numpy(), S.sddmm_fp64(A, dC, B)) <= 1e-5
    assert S.rel_fro(dB.cpu().numpy(), S.spmm_fp64(op.A.T.tocsr(), dC)) <= (1e-2 if mode == D.TC_BF16 else 1e-5)


@pytest.mark.parametrize("backward", ["fused", "separate"])
def test_operator_backward_sets_the_row_runs(backward):
    """A mode set at the C entry point between two backwards."""
    A = syn.community_graph(n=2048, target_nnz=30000, seed=15, max_deg=256)
    op = plan_spmm(A, 64, PlanConfig(backward=backward))
    _, _, Bt, dCt = _operands(A, 64)
    _, want = op.backward(dCt, Bt)
    for h in (op.handle, op.transposed[0].handle):
        _lib.check(h.lib.stile_spmm_plan_set_dvals_mode(h.handle, 1), "stile_spmm_plan_set_dvals_mode")
    _, got = op.backward(dCt, Bt)
    assert torch.equal(got, want)
