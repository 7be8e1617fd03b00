"""Row padding of dense operands, and the SDDMM's split between 1D and block
tiles: plans whose tiles share no entry run the 1D kernel first."""
import numpy as np
import pytest
import torch

import oracle.semantics as S
from stile_gb300 import device as D
from stile_gb300 import synthetic as syn
from stile_gb300.api import PlanConfig, SpmmOperator
from stile_gb300.ops import DeviceSddmmPlan, dense_operand, dense_operand_bf16
from stile_gb300.planner import search_sddmm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,cols,ld,off", [(1, 1, 1, 0), (7, 41, 41, 0), (300, 3, 3, 0), (33, 129, 131, 1),
                                              (1000, 8, 9, 3), (5, 64, 64, 1), (2, 1023, 1030, 0)])
def test_padded_operand_holds_the_rows_and_zeros(rows, cols, ld, off, dtype):
    base = torch.randn(rows * ld + off, device="cuda").to(dtype)
    x = torch.as_strided(base, (rows, cols), (ld, 1), off)
    y, got = (dense_operand if dtype == torch.float32 else dense_operand_bf16)(x)
    step = 4 if dtype == torch.float32 else 8
    assert got % step == 0 and y.data_ptr() % 16 == 0 and y.stride() == (got, 1) and y.shape == x.shape
    assert torch.equal(y, x)
    if y.data_ptr() != x.data_ptr():
        assert not torch.as_strided(y, (rows, got), (got, 1), 0)[:, cols:].any()


@pytest.mark.parametrize("F,bf16", [(64, False), (100, False), (33, True), (192, True)])
@pytest.mark.parametrize("shared", [False, True], ids=["disjoint", "shared"])
def test_scores_of_disjoint_and_overlapping_tiles(shared, F, bf16):
    """The bound of the two kernels' fp32 / split-bf16 products; an entry in
    both kinds of tile keeps the 1D result (bf16 operands: the same value)."""
    A = syn.sddmm_mask(n=2500, target_nnz=40_000, seed=9)
    dev = D.build_sddmm_device(search_sddmm(A, F, max_bucket_size=32).tiles, A.shape, A.nnz)
    assert len(dev.blk_out) and len(dev.mid_idx)
    if shared:
        rows = np.repeat(np.arange(A.shape[0]), np.diff(A.indptr)).astype(np.int32)
        extra = dev.blk_out[:5]
        for name, new in (("mid_idx", rows[extra]), ("j_idx", A.indices[extra].astype(np.int32)), ("remap", extra)):
            setattr(dev, name, np.concatenate([getattr(dev, name), new]))
    p = DeviceSddmmPlan(dev)
    g = torch.Generator("cuda").manual_seed(3)
    X, Y = (torch.randn(n, F, device="cuda", generator=g) for n in A.shape)
    if bf16:
        X, Y = X.to(torch.bfloat16), Y.to(torch.bfloat16)
    out = p.run(X, Y)
    assert p.error_flag() == 0
    ref = S.sddmm_fp64(A, X.float().cpu().numpy(), Y.float().cpu().numpy())
    assert S.rel_fro(out.cpu().numpy(), ref) <= 1e-5
    if shared and not bf16:     # the 1D kernel's fp32 sums, not the block kernel's split products
        e = dev.blk_out[:5]
        assert np.allclose(out.cpu().numpy()[e], ref[e], rtol=1e-6, atol=F * 1e-7)


@pytest.mark.parametrize("N,dtype", [(128, torch.float32), (41, torch.float32), (200, torch.float32),
                                     (256, torch.bfloat16), (72, torch.bfloat16)])
def test_product_of_rows_far_apart(N, dtype):
    """A view whose row stride makes every row offset exceed 31 bits of
    elements gives what the packed rows give (the same sums in the same
    order, but for atomic adds)."""
    A = syn.community_graph(n=640, target_nnz=9000, seed=4, max_deg=200)
    op = SpmmOperator(A, N, PlanConfig())
    B = torch.randn(A.shape[1], N, device="cuda").to(dtype)
    ld = (1 << 31) // 600 // 8 * 8          # 640 rows of 3.58M elements: 2.29e9 elements
    far = torch.empty(A.shape[1] * ld, dtype=dtype, device="cuda").as_strided((A.shape[1], N), (ld, 1))
    far.copy_(B)
    assert torch.allclose(op(far), op(B), rtol=1e-5, atol=1e-5)
