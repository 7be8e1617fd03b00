"""The tensor-core SpMM kernel at the edges of its stages, units and feature
slices: row widths around 32, 64 and 128 features, items of one k-step next to
items longer than a chunk, k-step counts that fill no stage of 2 or 4, B in
fp32 and bf16, every 16-bit mode, and C rows that are added to or stored.
Values and B are exact in bf16 (and in fp16), so the products are exact and
only the fp32 sums round: rows hold at most 700 entries, and 700 roundings of
2^-24 stay below 1e-5 even if they all fell the same way relative to the
row's norm."""
import numpy as np
import pytest
import scipy.sparse as sp
import torch

import oracle.semantics as S
from stile_gb300 import device as D
from stile_gb300.api import PlanConfig, SpmmOperator

pytestmark = pytest.mark.gpu


def _matrix(kind):
    """only tensor tiles: short items (1 to 3 k-steps), long ones, one item."""
    rng = np.random.default_rng(31)
    if kind == "short":      # 16-row bands with 5, 17 or 40 columns each
        parts = []
        for b in range(37):
            cols = rng.choice(300, size=(5, 17, 40)[b % 3], replace=False)
            r = np.repeat(np.arange(16), len(cols)) + 16 * b
            parts.append((r, np.tile(cols, 16)))
        r, c = (np.concatenate(x) for x in zip(*parts))
        shape = (37 * 16 - 5, 300)
        keep = r < shape[0]
        r, c = r[keep], c[keep]
    elif kind == "long":     # 700 columns in some bands: more than a chunk of 32 k-steps
        shape = (70, 900)
        dense = rng.random(shape) < 0.02
        dense[:16, :700] |= rng.random((16, 700)) < 0.9
        dense[33:40, 100:650] = True
        r, c = np.nonzero(dense)
    else:                    # one k-step in all
        shape = (16, 16)
        r, c = np.nonzero(rng.random(shape) < 0.6)
    v = rng.integers(-32, 33, len(r)) / 16.0
    v[v == 0] = 1.0
    A = sp.csr_matrix((v, (r, c)), shape=shape)
    A.sort_indices()
    return A


MODES = {"bf16": D.TC_BF16, "f16": D.TC_F16, "split": D.TC_SPLIT_BF16}


@pytest.mark.parametrize("N", [1, 12, 31, 32, 33, 63, 64, 65, 127, 128, 129, 200, 320])
@pytest.mark.parametrize("kind", ["short", "long", "one"])
@pytest.mark.parametrize("mode,operand", [("bf16", "fp32"), ("f16", "fp32"), ("split", "fp32"), ("bf16", "bf16")])
def test_products_of_exact_operands(kind, N, mode, operand):
    A = _matrix(kind)
    op = SpmmOperator(A, N, PlanConfig(tc_mode=MODES[mode], only_TC=True))
    assert op.device_layout.stats()["ell_rows"] == 0 and op.device_layout.stats()["tc_ksteps"] > 0
    B = np.random.default_rng(32).integers(-16, 17, (A.shape[1], N)).astype(np.float32) / 8
    Bt = torch.as_tensor(B, device="cuda")
    if operand == "bf16":
        Bt = Bt.to(torch.bfloat16)
    C = op(Bt)
    torch.cuda.synchronize()
    assert op.handle.error_flag() == 0
    assert S.rel_fro(C.cpu().numpy(), S.spmm_fp64(A, B)) <= 1e-5
