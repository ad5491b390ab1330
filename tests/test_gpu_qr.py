"""QR routes (GPU): the one-launch CholeskyQR of small matrices, the grid-wide passes beyond it, and
the Householder factorisation where the Gram matrix breaks down, at the edges between them and of the
16-column panels."""
import numpy as np
import pytest
import torch

from torchtt_gb300 import ops

pytestmark = pytest.mark.gpu
EPS = 2.220446049250313e-16


def _matrix(m, n, kind, g):
    a = g.standard_normal((m, n))
    if kind.startswith("cond"):
        u, v = np.linalg.qr(a)[0], np.linalg.qr(g.standard_normal((n, n)))[0]
        return (u * np.logspace(0, -float(kind[4:]), n)) @ v
    if kind == "graded":
        return a * np.logspace(0, -12, n)
    if kind == "deficient":
        a[:, n // 2:] = a[:, : n - n // 2] * 2.0
        return a
    if kind == "zero":
        return 0.0 * a
    return a * {"regular": 1.0, "tiny": 1e-140, "huge": 1e140}[kind]


@pytest.mark.parametrize("m,n", [(1, 1), (5, 4), (16, 16), (17, 16), (48, 4), (300, 1), (136, 16), (137, 16),
                                 (500, 8), (546, 8), (548, 8), (33, 32), (34, 32), (35, 32), (36, 33),
                                 (200, 48), (400, 49), (161, 160), (400, 161)])
@pytest.mark.parametrize("kind", ["regular", "cond4", "cond8", "cond14", "graded", "deficient", "zero",
                                  "tiny", "huge"])
def test_qr_routes(m, n, kind):
    a = _matrix(m, n, kind, np.random.default_rng(m * n))
    q, r = ops.qr(torch.from_numpy(a).cuda())
    q, r = q.cpu().numpy(), r.cpu().numpy()
    # backward stable factors: orthonormal columns and a residual at rounding level
    assert np.abs(np.tril(r, -1)).max(initial=0.0) == 0.0
    assert np.linalg.norm(q.T @ q - np.eye(n)) <= 16 * n * EPS
    assert np.linalg.norm(q @ r - a) <= 16 * n * EPS * np.linalg.norm(a)
