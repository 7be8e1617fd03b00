"""Rows of 4 GB and more (row strides past 32 bits of bytes): the 64-bit
variants of the tensor-core and row-tile kernels and the bf16 run kernel's
general form.  A few rows are enough; each case holds 43 GB at most."""
import numpy as np
import pytest
import scipy.sparse as sp
import torch

import oracle.semantics as S
from stile_gb300 import device as D
from stile_gb300.api import PlanConfig, SddmmOperator, SpmmOperator

pytestmark = pytest.mark.gpu

ROW = 1 << 32      # bytes


def _matrix(m, k):
    """no empty row (C needs no zeroing), not every entry there"""
    rng = np.random.default_rng(3)
    keep = rng.random((m, k)) < 0.8
    keep[:, 0] = True
    A = sp.csr_matrix(np.where(keep, rng.standard_normal((m, k)), 0.0))
    A.sort_indices()
    return A


def _far(rows, cols, dtype=torch.float32):
    size = torch.empty(0, dtype=dtype).element_size()
    ld = ROW // size
    return torch.empty((rows - 1) * ld + (cols + 15) // 16 * 16, dtype=dtype, device="cuda").as_strided((rows, cols), (ld, 1))


def _spread(x):
    y = _far(*x.shape, x.dtype)
    y.copy_(x)
    return y


@pytest.fixture(autouse=True)
def _free():
    yield
    torch.cuda.empty_cache()


@pytest.mark.parametrize("N", [20, 64, 128, 150, 300])
@pytest.mark.parametrize("mode,dtype", [(D.TC_BF16, torch.float32), (D.TC_F16, torch.float32),
                                        (D.TC_SPLIT_BF16, torch.float32), (D.TC_BF16, torch.bfloat16)],
                         ids=["bf16", "f16", "split", "bf16-B"])
@pytest.mark.parametrize("kind", ["rows", "tensor"])
@pytest.mark.parametrize("far", ["B", "C"])
def test_product(far, kind, mode, dtype, N):
    A = _matrix(40, 3) if far == "B" else _matrix(6, 6)
    op = SpmmOperator(A, N, PlanConfig(tc_mode=mode, only_ELL=kind == "rows", only_TC=kind == "tensor"))
    B = torch.randn(A.shape[1], N, device="cuda", generator=torch.Generator("cuda").manual_seed(N)).to(dtype)
    if far == "B":
        C = op(_spread(B))
    else:
        C = op(B, out=_far(6, N))
    assert op.handle.error_flag() == 0
    tol = 1e-2 if kind == "tensor" and mode != D.TC_SPLIT_BF16 else 1e-5
    assert S.rel_fro(C.cpu().numpy(), S.spmm_fp64(A, B.float().cpu().numpy())) <= tol
    assert torch.allclose(C, op(B), rtol=1e-5, atol=1e-5)      # as packed rows, but for the order of atomic adds


@pytest.mark.parametrize("kind", ["rows", "tensor"])
@pytest.mark.parametrize("N", [41, 128, 200])
def test_backward(N, kind):
    A = _matrix(6, 6)
    op = SpmmOperator(A, N, PlanConfig(tc_mode=D.TC_SPLIT_BF16, backward="fused", only_ELL=kind == "rows",
                                       only_TC=kind == "tensor"))
    g = torch.Generator("cuda").manual_seed(N)
    B, dC = (torch.randn(6, N, device="cuda", generator=g) for _ in range(2))
    dB, dv = op.backward(_spread(dC), _spread(B))
    assert S.rel_fro(dB.cpu().numpy(), S.spmm_fp64(A.T.tocsr(), dC.cpu().numpy())) <= 1e-5
    assert S.rel_fro(dv.cpu().numpy(), S.sddmm_fp64(A, dC.cpu().numpy(), B.cpu().numpy())) <= 1e-5
    Bb = B.to(torch.bfloat16)
    dv = op.handle.dvals(dC, _spread(Bb))
    assert S.rel_fro(dv.cpu().numpy(), S.sddmm_fp64(A, dC.cpu().numpy(), Bb.float().cpu().numpy())) <= 1e-5


@pytest.mark.parametrize("F", [30, 64, 128, 200])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16], ids=["fp32", "bf16"])
def test_scores(dtype, F):
    A = _matrix(3, 3)
    op = SddmmOperator(A, F)
    g = torch.Generator("cuda").manual_seed(F)
    X, Y = (torch.randn(3, F, device="cuda", generator=g).to(dtype) for _ in range(2))
    out = op(_spread(X), _spread(Y))
    assert S.rel_fro(out.cpu().numpy(), S.sddmm_fp64(A, X.float().cpu().numpy(), Y.float().cpu().numpy())) <= 1e-5
