"""SVD routes (GPU): one warp below 16 columns, the FP32-preconditioned cluster and grid Jacobi above, and
the routes without it (singular or out-of-range matrices, more than 224 columns), at the edges of the
register tiles and for graded, clustered, deficient and scaled spectra."""
import numpy as np
import pytest
import torch

from torchtt_gb300 import ops

pytestmark = pytest.mark.gpu
EPS = 2.220446049250313e-16


def _spectrum(n, kind):
    if kind == "clustered":
        return np.concatenate([np.ones(n - n // 2), np.full(n // 2, 1e-3)])
    if kind == "deficient":
        s = np.logspace(0, -6, n)
        s[n - n // 3:] = 0.0
        return s
    return np.logspace(0, {"mild": -3, "graded": -14, "tiny": -3, "huge": -3}[kind], n) * \
        {"tiny": 1e-130, "huge": 1e130}.get(kind, 1.0)


@pytest.mark.parametrize("m,n", [(1, 1), (7, 2), (20, 3), (15, 15), (60, 16), (17, 17), (90, 32), (33, 33),
                                 (64, 64), (200, 65), (300, 80), (81, 81), (97, 97), (500, 112), (113, 113),
                                 (400, 160), (161, 161), (300, 224), (226, 225)])
@pytest.mark.parametrize("kind", ["mild", "graded", "clustered", "deficient", "tiny", "huge"])
def test_svd_routes(m, n, kind):
    g = np.random.default_rng(m + n)
    s0 = _spectrum(n, kind)
    a = (np.linalg.qr(g.standard_normal((m, n)))[0] * s0) @ np.linalg.qr(g.standard_normal((n, n)))[0].T
    u, s, vh = (v.cpu().numpy() for v in ops.svd(torch.from_numpy(a).cuda()))
    top = s0[0]
    assert np.all(np.diff(s) <= 0.0) and np.abs(s - s0).max() <= 16 * n * EPS * top
    assert np.linalg.norm((u * s) @ vh - a) <= 16 * n * EPS * np.linalg.norm(a)
    k = int((s0 > 64 * n * EPS * top).sum())   # vectors that the matrix determines
    assert np.linalg.norm(u[:, :k].T @ u[:, :k] - np.eye(k)) <= 32 * n * EPS
    assert np.linalg.norm(vh[:k] @ vh[:k].T - np.eye(k)) <= 64 * n * EPS


def test_svd_of_special_matrices():
    dev = torch.device("cuda", 0)
    for n in (5, 40):
        u, s, vh = ops.svd(torch.zeros(50, n, dtype=torch.float64, device=dev))
        assert float(s.abs().max()) == 0.0 and torch.isfinite(u).all() and torch.isfinite(vh).all()
        d = torch.diag(torch.arange(1, n + 1, dtype=torch.float64, device=dev))
        u, s, vh = ops.svd(d)
        assert torch.equal(s, torch.arange(n, 0, -1, dtype=torch.float64, device=dev))
        assert float(((u * s) @ vh - d).abs().max()) <= 16 * n * EPS * n
