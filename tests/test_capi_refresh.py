"""Refusals of the row-padding and paired value-refresh entry points.  Those of
stile_pad_rows and the null arguments come before any device call (aligned
dummies, never read); the pair's need uploaded plans."""
import numpy as np
import pytest
import torch

from stile_gb300 import _lib
from stile_gb300 import device as D
from stile_gb300 import synthetic as syn

INVALID, UNSUPPORTED = -1, -4
FAKE = 1 << 20


@pytest.mark.parametrize("args,code,msg", [
    ((FAKE, -1, 8, 8, 4, FAKE, 8), INVALID, "bad shape"),
    ((FAKE, 8, -1, 8, 4, FAKE, 8), INVALID, "bad shape"),
    ((FAKE, 8, 8, 8, 8, FAKE, 8), UNSUPPORTED, "2 or 4 bytes"),
    ((FAKE, 8, 8, 8, 1, FAKE, 16), UNSUPPORTED, "2 or 4 bytes"),
    ((None, 8, 8, 8, 4, FAKE, 8), INVALID, "null argument"),
    ((FAKE, 8, 8, 8, 4, None, 8), INVALID, "null argument"),
    ((FAKE, 8, 9, 9, 4, FAKE, 8), INVALID, "16-byte"),          # dst rows shorter than cols
    ((FAKE, 8, 6, 6, 4, FAKE, 6), INVALID, "16-byte"),          # 24-byte dst rows
    ((FAKE, 8, 12, 12, 2, FAKE, 12), INVALID, "16-byte"),
    ((FAKE, 8, 8, 8, 4, FAKE + 8, 8), INVALID, "16-byte"),
    ((FAKE + 2, 8, 8, 8, 4, FAKE, 8), INVALID, "misaligned"),
    ((FAKE + 1, 8, 8, 8, 2, FAKE, 8), INVALID, "misaligned"),
    ((FAKE, (1 << 37) + 1, 8, 8, 4, FAKE, 8), UNSUPPORTED, "more rows"),
    ((FAKE, 2, 41, 41, 4, FAKE, 1 << 31), UNSUPPORTED, "2^31 elements"),
    ((FAKE, 2, 41, 41, 2, FAKE, 1 << 40), UNSUPPORTED, "2^31 elements"),
])
def test_pad_rows_refuses(args, code, msg):
    lib = _lib.load()
    assert lib.stile_pad_rows(*args, None) == code
    assert msg in _lib.last_error(), _lib.last_error()


@pytest.mark.parametrize("rows,cols", [(0, 5), (5, 0), (0, 0)])
def test_pad_rows_of_nothing(rows, cols):
    assert _lib.load().stile_pad_rows(None, rows, cols, 5, 4, None, 8, None) == 0


def test_refresh_and_policy_refuse_null_plans():
    lib = _lib.load()
    assert lib.stile_spmm_plan_set_values_pair(None, None, FAKE, None, None) == INVALID
    assert "null argument" in _lib.last_error()
    assert lib.stile_sddmm_plan_set_wait_policy(None, 10, 1) == INVALID
    assert "null plan" in _lib.last_error()


@pytest.mark.gpu
def test_paired_refresh_refuses_plans_that_do_not_belong_together():
    from stile_gb300.api import PlanConfig, SddmmOperator, SpmmOperator
    lib = _lib.load()
    A = syn.power_law_rows(300, 200, min_len=4, max_len=60, seed=5)
    op = SpmmOperator(A, 32, PlanConfig(only_TC=True))
    opT, _ = op.transposed
    pair = lib.stile_spmm_plan_set_values_pair
    vals = torch.ones(A.nnz, device="cuda")
    args = (vals.data_ptr(), None, None)
    assert pair(op.handle.handle, opT.handle.handle, None, None, None) == INVALID
    fresh = SpmmOperator(A.T.tocsr(), 32, PlanConfig(only_TC=True))
    assert pair(op.handle.handle, fresh.handle.handle, *args) == INVALID
    assert "set_transpose_ids" in _lib.last_error()
    split = SpmmOperator(A.T.tocsr(), 32, PlanConfig(only_TC=True, tc_mode=D.TC_SPLIT_BF16))
    split.handle.set_transpose_ids(op.transposed[1])
    assert pair(op.handle.handle, split.handle.handle, *args) == UNSUPPORTED
    assert "same tensor-tile mode" in _lib.last_error()
    other = SpmmOperator(syn.power_law_rows(200, 300, min_len=3, max_len=20, seed=6), 32, PlanConfig(only_TC=True))
    assert other.nnz != op.nnz
    assert pair(op.handle.handle, other.handle.handle, *args) == INVALID
    assert "same nonzeros" in _lib.last_error()
    fp8 = SpmmOperator(A, 32, PlanConfig(only_TC=True, tc_mode=D.TC_FP8))
    assert pair(fp8.handle.handle, None, *args) == UNSUPPORTED
    # refused calls changed nothing
    B = np.ones((A.shape[1], 32), np.float32)
    assert torch.isfinite(op(torch.as_tensor(B, device="cuda"))).all()
    sop = SddmmOperator(syn.sddmm_mask(n=300, target_nnz=3000, seed=9), 32)
    assert lib.stile_sddmm_plan_set_wait_policy(sop.handle.handle, 0, 1) == INVALID
    assert "needs a poll limit" in _lib.last_error()
