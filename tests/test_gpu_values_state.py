"""What an operator remembers of the values it loaded last: the transposed
operator's copy under a replayed graph, and values of another shape."""
import pytest
import torch

from stile_gb300 import synthetic as syn
from stile_gb300.api import PlanConfig, SpmmOperator

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
