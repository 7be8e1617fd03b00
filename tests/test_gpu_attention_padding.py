"""Fused sparse attention of widths that fill no power of two of lanes: rows
whose padding holds NaN (views of padded buffers, taken as they are), and K
rows with an entry of -inf, whose weight is 0."""
import numpy as np
import pytest
import scipy.sparse as sp
import torch

import oracle.attention as OA
import oracle.semantics as S
from stile_gb300.api import SparseAttention

pytestmark = pytest.mark.gpu


def _pattern(n=50):
    rng = np.random.default_rng(15)
    A = sp.csr_matrix((rng.random((n, n)) < 0.3).astype(np.float64))
    A[:, 0] = 1.0          # every row keeps a finite entry
    A = sp.csr_matrix(A)
    A.sort_indices()
    return A


def _padded(x):
    """x as a view of rows of whole 16-byte vectors, NaN past its features."""
    h, n, f = x.shape
    buf = torch.full((h, n, (f + 3) // 4 * 4), float("nan"), device="cuda")
    buf[:, :, :f] = torch.as_tensor(x, device="cuda")
    return buf[:, :, :f]


@pytest.mark.parametrize("F,Fv", [(2, 2), (5, 7), (15, 13), (20, 20), (23, 40), (41, 41), (60, 9), (65, 127), (80, 80),
                                  (127, 126), (11, 128), (128, 3)])
def test_padding_and_infinite_keys(F, Fv):
    A = _pattern()
    rng = np.random.default_rng(16)
    n = A.shape[0]
    Q, K = (rng.standard_normal((2, n, F)).astype(np.float32) for _ in range(2))
    V = rng.standard_normal((2, n, Fv)).astype(np.float32)
    op = SparseAttention(A, F, Fv)
    out = op(_padded(Q), _padded(K), _padded(V)).cpu().numpy()
    assert S.rel_fro(out, OA.attention_fp64(A, Q, K, V, op.scale)) <= 1e-5   # the fp32 path's bound
    # the last feature of some K rows is -inf and every q's is positive: those
    # entries weigh nothing, as if they were not in the pattern
    Q[:, :, F - 1] = np.abs(Q[:, :, F - 1]) + 0.5
    dead = np.arange(7, n, 5)
    K[:, dead, F - 1] = -np.inf
    out = op(_padded(Q), _padded(K), _padded(V)).cpu().numpy()
    live = A.tolil()
    live[:, dead] = 0.0
    live = sp.csr_matrix(live)
    live.eliminate_zeros()
    K[:, dead, F - 1] = 0.0
    assert S.rel_fro(out, OA.attention_fp64(live, Q, K, V, op.scale)) <= 1e-5
