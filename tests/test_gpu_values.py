"""Value refresh of a plan: the transposed plan's values from the forward's
(no permuted copy) equal to loading the permuted values, and batched sets
whose row-tile values are not a multiple of 4 entries."""
import numpy as np
import pytest
import scipy.sparse as sp
import torch

import oracle.semantics as S
from stile_gb300 import device as D
from stile_gb300 import synthetic as syn
from stile_gb300.api import PlanConfig, SpmmOperator

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [D.TC_BF16, D.TC_F16, D.TC_SPLIT_BF16], ids=["bf16", "f16", "split"])
@pytest.mark.parametrize("kind", ["mixed", "tensor", "rows", "one"])
def test_forward_numbered_values_equal_permuted_values(kind, mode):
    A = {"mixed": lambda: syn.power_law_rows(700, 523, min_len=6, max_len=300, seed=3),
         "tensor": lambda: syn.pruned_weight(64, 96, sparsity=0.5, seed=4),
         "rows": lambda: syn.power_law_rows(333, 333, min_len=1, max_len=9, seed=5),
         "one": lambda: sp.csr_matrix(([2.0], ([5], [7])), shape=(10, 9))}[kind]()
    cfg = PlanConfig(tc_mode=mode, only_ELL=kind == "rows", only_TC=kind == "tensor")
    op = SpmmOperator(A, 36, cfg)
    opT, perm = op.transposed
    vals = torch.randn(A.nnz, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    X = torch.randn(A.shape[0], 36, device="cuda", generator=torch.Generator("cuda").manual_seed(2))
    opT.handle.set_values(vals[perm])
    want = opT(X).clone()
    opT.handle.set_values(torch.zeros_like(vals))
    op.set_values(vals)
    assert torch.allclose(opT(X), want, rtol=1e-5, atol=1e-5)  # equal but for the order of atomic sums
    assert torch.equal(opT._vals, vals[perm])
    Av = A.copy()
    Av.data = vals.cpu().numpy().astype(np.float64)
    ref = S.spmm_fp64(Av.T.tocsr(), X.cpu().numpy())
    assert S.rel_fro(opT(X).cpu().numpy(), ref) <= (1e-5 if mode == D.TC_SPLIT_BF16 else 1e-2)


@pytest.mark.parametrize("heads", [1, 3])
def test_batched_values_of_an_odd_entry_count(heads):
    A = syn.power_law_rows(97, 203, min_len=1, max_len=64, seed=7)
    while A.nnz % 4 == 0:
        A.data[0] = 0.0
        A.eliminate_zeros()
    op = SpmmOperator(A, 20, PlanConfig(only_ELL=True))
    g = torch.Generator("cuda").manual_seed(8)
    vals = torch.randn(heads, A.nnz, device="cuda", generator=g)
    B = torch.randn(heads, A.shape[1], 20, device="cuda", generator=g)
    C = op.batched(vals, B).cpu().numpy()
    for h in range(heads):
        Ah = A.copy()
        Ah.data = vals[h].cpu().numpy().astype(np.float64)
        assert S.rel_fro(C[h], S.spmm_fp64(Ah, B[h].cpu().numpy())) <= 1e-6
