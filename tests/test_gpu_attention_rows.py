"""Fused sparse attention on rows of every length around its batches (0 to 19
entries, and the 2 to 16 lanes its feature widths take), and rows whose last
entry's V is infinite."""
import numpy as np
import pytest
import scipy.sparse as sp
import torch

import oracle.attention as OA
import oracle.semantics as S
from stile_gb300.api import SparseAttention

pytestmark = pytest.mark.gpu


def _pattern(n=61):
    rng = np.random.default_rng(5)
    rows, cols = [], []
    for r in range(n):
        c = np.sort(rng.choice(n, size=r % 20, replace=False))
        rows += [r] * len(c)
        cols += list(c)
    return sp.csr_matrix((np.ones(len(rows)), (rows, cols)), shape=(n, n))


@pytest.mark.parametrize("F,Fv", [(1, 1), (3, 16), (16, 16), (17, 5), (32, 32), (36, 60), (64, 64), (65, 64), (68, 100),
                                  (128, 128), (127, 33)])
def test_every_row_length(F, Fv):
    A = _pattern()
    rng = np.random.default_rng(6)
    Q, K = (rng.standard_normal((2, A.shape[0], F)).astype(np.float32) for _ in range(2))
    V = rng.standard_normal((2, A.shape[0], Fv)).astype(np.float32)
    out = SparseAttention(A, F, Fv)(*(torch.as_tensor(x, device="cuda") for x in (Q, K, V))).cpu().numpy()
    assert not out[:, np.diff(A.indptr) == 0].any()
    assert S.rel_fro(out, OA.attention_fp64(A, Q, K, V, 1.0 / np.sqrt(F))) <= 1e-5   # the fp32 path's bound


def test_infinite_v_of_a_rows_last_entry_stays_infinite():
    A = _pattern()
    rng = np.random.default_rng(7)
    Q, K, V = (rng.standard_normal((A.shape[0], 64)).astype(np.float32) for _ in range(3))
    V[A.shape[0] - 4:, 3] = np.inf
    out = SparseAttention(A, 64)(*(torch.as_tensor(x, device="cuda") for x in (Q, K, V))).cpu().numpy()
    hit = np.array([(A.indices[a:b] >= A.shape[0] - 4).any() for a, b in zip(A.indptr[:-1], A.indptr[1:])])
    assert hit.any() and np.all(np.isposinf(out[hit, 3]))
    assert np.isfinite(np.delete(out, 3, axis=1)).all() and np.isfinite(out[~hit]).all()
