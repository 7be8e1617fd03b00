"""What an operator remembers of the values it loaded last: the transposed
operator's copy under a replayed graph, and values of another shape."""
import numpy as np
import pytest
import torch

import oracle.semantics as S
from stile_gb300 import device as D
from stile_gb300 import synthetic as syn
from stile_gb300.api import PlanConfig, SpmmOperator
from stile_gb300.ops import launch_count

pytestmark = pytest.mark.gpu


def test_transposed_values_follow_a_replayed_graph():
    A = syn.power_law_rows(300, 200, min_len=2, max_len=40, seed=5)
    op = SpmmOperator(A, 32, PlanConfig())
    opT, perm = op.transposed
    vals = torch.ones(A.nnz, device="cuda")
    op.set_values(vals)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        op.set_values(vals)
    for scale in (2.0, 3.0):
        vals.copy_(torch.arange(A.nnz, device="cuda") * scale)
        graph.replay()
        assert torch.equal(opT._vals, vals[perm])
        assert torch.equal(op._vals, vals)


@pytest.mark.parametrize("shape", [(1, -1), (-1, 1)], ids=["row", "column"])
def test_values_of_another_shape(shape):
    A = syn.power_law_rows(300, 200, min_len=2, max_len=40, seed=5)
    op = SpmmOperator(A, 32, PlanConfig())
    opT, perm = op.transposed
    vals = torch.arange(A.nnz, dtype=torch.float32, device="cuda")
    op.set_values(vals.reshape(shape))
    assert torch.equal(op._vals, vals) and torch.equal(opT._vals, vals[perm])


@pytest.mark.parametrize("kw", [{}, {"only_ELL": True}, {"only_TC": True}], ids=["mixed", "rows", "tensor"])
def test_values_without_a_transposed_plan_come_in_one_launch(kw):
    A = syn.power_law_rows(300, 200, min_len=2, max_len=40, seed=5)
    op = SpmmOperator(A, 32, PlanConfig(tc_mode=D.TC_SPLIT_BF16, **kw))
    vals = torch.randn(A.nnz, device="cuda")
    before = launch_count()
    op.set_values(vals)
    assert launch_count() == before + 1
    assert torch.equal(op._vals, vals) and op._vals.data_ptr() != vals.data_ptr()
    B = torch.randn(A.shape[1], 32, device="cuda")
    Av = A.copy()
    Av.data = vals.cpu().numpy().astype(np.float64)
    assert S.rel_fro(op(B).cpu().numpy(), S.spmm_fp64(Av, B.cpu().numpy())) <= 1e-5
