"""QR of wide matrices (GPU): Q from the leading square block, whatever its rank, the other columns of R as
products; at the edges of the routes that the square block takes."""
import numpy as np
import pytest
import torch

from torchtt_gb300 import ops

pytestmark = pytest.mark.gpu
EPS = 2.220446049250313e-16


@pytest.mark.parametrize("m,n", [(1, 2), (1, 7), (5, 9), (16, 17), (32, 33), (32, 48), (33, 60), (48, 200),
                                 (160, 161), (161, 230)])
@pytest.mark.parametrize("kind", ["regular", "lead_zero", "lead_rank1", "lead_cond12", "graded", "zero", "tiny",
                                  "huge"])
def test_wide_qr(m, n, kind):
    g = np.random.default_rng(m * n)
    a = g.standard_normal((m, n))
    if kind == "lead_zero":
        a[:, :(m + 1) // 2] = 0.0
    elif kind == "lead_rank1":
        a[:, :m] = np.outer(a[:, 0], g.standard_normal(m))
    elif kind == "lead_cond12":
        u, v = np.linalg.qr(a[:, :m])[0], np.linalg.qr(g.standard_normal((m, m)))[0]
        a[:, :m] = (u * np.logspace(0, -12, m)) @ v
    elif kind == "graded":
        a *= np.logspace(0, -12, n)
    else:
        a *= {"regular": 1.0, "zero": 0.0, "tiny": 1e-140, "huge": 1e140}[kind]
    q, r = ops.qr(torch.from_numpy(a).cuda())
    q, r = q.cpu().numpy(), r.cpu().numpy()
    assert q.shape == (m, m) and r.shape == (m, n)
    assert np.abs(np.tril(r, -1)).max(initial=0.0) == 0.0
    assert np.linalg.norm(q.T @ q - np.eye(m)) <= 16 * m * EPS
    # the products add the distance of Q from orthogonality to the residual of the block
    assert np.linalg.norm(q @ r - a) <= 32 * m * EPS * np.linalg.norm(a)
