"""Ragged dense operands whose bytes are not their values: a view with torch's
lazy negation (the imaginary part of a conjugate is one)."""
import pytest
import torch

from stile_gb300.ops import dense_operand, dense_operand_bf16

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("take,dtype", [(dense_operand, torch.float32), (dense_operand_bf16, torch.bfloat16)])
def test_negated_view_is_padded_with_its_values(take, dtype):
    x = torch.randn(9, 41, device="cuda").to(dtype)
    y, _ = take(torch._neg_view(x))
    assert torch.equal(y, -x)
