"""Row runs of several feature passes: short and long groups, few and more than
the device keeps resident (2 or 4 gathered rows in flight)."""
import numpy as np
import pytest
import scipy.sparse as sp
import torch

import oracle.semantics as S
from stile_gb300.ops import plain_sddmm_plan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("F", [129, 192, 256, 500])
@pytest.mark.parametrize("bf16", [False, True], ids=["fp32", "bf16"])
@pytest.mark.parametrize("rows,length", [(50, 1), (50, 5), (40, 30), (20_000, 2), (20_000, 5), (20_000, 11), (3_000, 40)])
def test_scores(rows, length, bf16, F):
    rng = np.random.default_rng(length)
    k = 700
    cols = np.sort(np.stack([rng.choice(k, size=length, replace=False) for _ in range(rows)]), axis=1)
    A = sp.csr_matrix((np.ones(cols.size), cols.reshape(-1), np.arange(0, cols.size + 1, length)), shape=(rows, k))
    g = torch.Generator("cuda").manual_seed(F)
    X, Y = (torch.randn(n, F, device="cuda", generator=g) for n in (rows, k))
    if bf16:
        X, Y = X.to(torch.bfloat16), Y.to(torch.bfloat16)
    out = plain_sddmm_plan(A).run(X, Y).cpu().numpy()
    assert S.rel_fro(out, S.sddmm_fp64(A, X.float().cpu().numpy(), Y.float().cpu().numpy())) <= 1e-6   # fp32 sums
