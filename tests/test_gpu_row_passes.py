"""Row tiles alone at 129 to 1000 features, over too few entries to fill the
device with passes of 128 features (each pass a block of its own) and over
more (passes of 256)."""
import numpy as np
import pytest
import torch

import oracle.semantics as S
from stile_gb300 import synthetic as syn
from stile_gb300.api import PlanConfig, SpmmOperator

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [129, 150, 255, 300, 500, 1000])
@pytest.mark.parametrize("m,shortest", [(40, 1), (500, 2), (2000, 3), (4096, 8), (6000, 20)])
def test_wide_rows_of_few_and_many_entries(m, shortest, N):
    A = syn.power_law_rows(m, m, min_len=shortest, max_len=min(m, 300), seed=3)
    op = SpmmOperator(A, 128, PlanConfig(only_ELL=True))
    B = np.random.default_rng(4).standard_normal((m, N)).astype(np.float32)
    C = op(torch.as_tensor(B, device="cuda")).cpu().numpy()
    assert S.rel_fro(C, S.spmm_fp64(A, B)) <= 1e-6      # fp32 sums of at most 300 products
