"""Split-bf16 tensor tiles on operands that are not exact in bf16, where each of
the three products counts: the edges of stages, units and feature slices, and
sums of one sign, which show the tensor cores' accumulation.

An accumulation there truncates: it loses half a unit in the last place on
average, 0.5 * 0.72 * 2^-23 of the partial sum (0.72: the mean of unit over value
within a binade).  A sum that grows evenly over c accumulations therefore loses
c / 2 * 0.5 * 0.72 * 2^-23 of itself.  Drained into fp32 registers (which round
both ways) every 4 k-steps of 3 products, c = 12: 2.6e-7."""
import numpy as np
import pytest
import scipy.sparse as sp
import torch

import oracle.semantics as S
from stile_gb300 import device as D
from stile_gb300.api import PlanConfig, SpmmOperator
from test_gpu_tc_kernel import _matrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [1, 31, 33, 63, 64, 65, 127, 128, 129, 200])
@pytest.mark.parametrize("kind", ["short", "long", "one"])
def test_products_of_operands_with_low_parts(kind, N):
    A = _matrix(kind)
    rng = np.random.default_rng(41)
    A.data = rng.standard_normal(A.nnz)
    op = SpmmOperator(A, N, PlanConfig(tc_mode=D.TC_SPLIT_BF16, only_TC=True))
    B = rng.standard_normal((A.shape[1], N)).astype(np.float32)
    C = op(torch.as_tensor(B, device="cuda")).cpu().numpy()
    assert op.handle.error_flag() == 0
    A.data = A.data.astype(np.float32).astype(np.float64)
    # each product drops lo * lo, at most 2^-16 of it (a missing hi * lo: 2^-9)
    assert S.rel_fro(C, S.spmm_fp64(A, B)) <= 1e-5


@pytest.mark.parametrize("N", [64, 128])
@pytest.mark.parametrize("k", [700, 3000])
def test_sums_of_one_sign_lose_no_more_than_a_short_chain(k, N):
    rng = np.random.default_rng(42)
    A = sp.csr_matrix(rng.uniform(0.5, 1.5, (64, k)).astype(np.float32).astype(np.float64))
    op = SpmmOperator(A, N, PlanConfig(tc_mode=D.TC_SPLIT_BF16, only_TC=True))
    B = rng.uniform(0.5, 1.5, (k, N)).astype(np.float32)
    C = op(torch.as_tensor(B, device="cuda")).cpu().numpy()
    ref = S.spmm_fp64(A, B)
    assert abs(np.mean((C - ref) / ref)) <= 2.6e-7
