"""The device-resident GMRES (GPU) across the shapes where its Arnoldi passes change: slices of 64,
128 and 256 elements (64 and 128 per SM), vectors per warp (8, 16, 32, 48 and up to 127), and lengths
that are no multiple of a slice. The cycle ends where the residual estimate meets the threshold, so
the true residual has to meet it too."""
import numpy as np
import pytest
import torch

from torchtt_gb300 import ops

pytestmark = pytest.mark.gpu


def _spd(k, cond, g):
    q = np.linalg.qr(g.standard_normal((k, k)))[0]
    return (q * np.linspace(1.0, cond, k)) @ q.T


@pytest.mark.parametrize("r,n,R", [(1, 2, 3), (3, 5, 7), (9, 31, 35), (21, 23, 21), (24, 33, 25),
                                   (31, 32, 40), (47, 31, 45)])
@pytest.mark.parametrize("cond,iters,resets", [(1.6, 40, 2), (3.0, 40, 3), (5.5, 126, 1)])
def test_residual_meets_the_threshold(r, n, R, cond, iters, resets):
    g = np.random.default_rng(r * n * R)
    dev = torch.device("cuda", 0)
    put = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)
    phl, phr = put(_spd(r, cond, g)[:, None, :]), put(_spd(R, cond, g)[:, None, :])
    A = put(_spd(n, cond, g)[None, :, :, None])
    rhs = put(g.standard_normal((r, n, R)))
    thr = 1e-7
    x, flag, nit = ops.local_gmres(phl, A, phr, rhs, iters=iters, threshold=thr, resets=resets)
    res = torch.einsum("lsr,smnS,LSR,rnR->lmL", phl, A, phr, x) - rhs
    assert flag == 1 and 1 <= nit <= iters * resets
    # the estimate equals the true residual up to the rounding of the operator, eps cond^3 << thr
    assert float(res.norm() / rhs.norm()) <= 1.001 * thr
