"""What the digit products leave below the scales of a row and a column (GPU): only the digit products beyond the
leading 36, 2^-57 of the scales per term. One term per element, whose operand spreads over six decades in
its row: a sum rounded to 2^-54 of the scales would show."""
import numpy as np
import pytest
import torch

from torchtt_gb300 import TT, ops

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


@pytest.mark.parametrize("m,n", [(160, 400), (160, 9000)])   # digits made per tile and beforehand
@pytest.mark.parametrize("swap", [False, True])
def test_single_terms(m, n, swap):
    g = np.random.default_rng(m + n)
    q = np.zeros((m, m))
    q[np.arange(m), g.permutation(m)] = 1.0 + g.random(m)
    x = (1.0 + g.random((m, n))) * 10.0 ** g.uniform(-6, 0, (m, n))
    a, b = (x.T, q.T) if swap else (q, x)
    put = lambda v: torch.from_numpy(np.ascontiguousarray(v)).cuda()
    before, _ = ops.autotune(False)
    try:
        y = TT([put(a[None, :, :, None]), put(np.ones((1, 1, 1, 1)))]) @ \
            TT([put(b[None]), put(np.ones((b.shape[1], 1, 1)))])
    finally:
        ops.autotune(before)
    c = y.cores[0][0].cpu().numpy()
    c = c.T if swap else c
    # the digits of x below 2^-61 of its column's largest entry, and the products left out
    scale = 2.0 ** np.ceil(np.log2(np.abs(x).max(axis=0)))[None, :] * 2.0
    ref = q.argmax(axis=1)
    exact = q.max(axis=1)[:, None].astype(np.longdouble) * x[ref]
    assert np.all(np.abs(c - exact) <= 2 * U * np.abs(exact) + 1.25 * 2.0 ** -57 * scale)
