"""The dense local solve (GPU): a one-core solve is one direct solve of the core's matrix, so it is
compared with numpy on both sides of the panel and block sizes, and on systems that the FP32 inverse
cannot refine (ill-conditioned, badly scaled), which the FP64 LU takes."""
import numpy as np
import pytest
import torch

from torchtt_gb300 import TT, amen_solve

pytestmark = pytest.mark.gpu
EPS = 2.220446049250313e-16


def _matrix(n, kind, g):
    q = np.linalg.qr(g.standard_normal((n, n)))[0]
    p = np.linalg.qr(g.standard_normal((n, n)))[0]
    if kind == "regular":       # condition 1e3
        return (q * np.logspace(0, -3, n)) @ p
    if kind == "ill":           # condition 1e10: no FP32 refinement
        return (q * np.logspace(0, -10, n)) @ p
    if kind == "tiny":          # below the FP32 range
        return 1e-200 * ((q * np.logspace(0, -2, n)) @ p)
    a = np.eye(n)[g.permutation(n)]   # "pivots": every pivot off the diagonal, graded over 1e8
    return a * np.logspace(4, -4, n)


@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 33, 127, 128, 129, 257, 499, 512, 513])
@pytest.mark.parametrize("kind", ["regular", "pivots", "ill", "tiny"])
def test_one_core_solve_matches_numpy(n, kind):
    g = np.random.default_rng(n)
    a = _matrix(n, kind, g)
    b = a @ g.standard_normal(n)
    dev = torch.device("cuda", 0)
    x = amen_solve(TT([torch.from_numpy(a[None, :, :, None]).to(dev)]),
                   TT([torch.from_numpy(b[None, :, None]).to(dev)]), max_full=600)
    x = x.cores[0].cpu().numpy().reshape(-1)
    ref = np.linalg.solve(a, b)
    sv = np.linalg.svd(a, compute_uv=False)
    # backward stable: residual within a small multiple of n eps ||A|| ||x||, error within cond(A) of it
    assert np.linalg.norm(a @ x - b) <= 8 * n * EPS * sv[0] * np.linalg.norm(x)
    assert np.linalg.norm(x - ref) <= 16 * n * EPS * (sv[0] / sv[-1]) * np.linalg.norm(ref)
