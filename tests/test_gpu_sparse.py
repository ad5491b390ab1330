"""The structured A stage built on the device (GPU): the local product and both interface updates of a
random sparse core against the dense contraction, at densities on both sides of the limit (a quarter),
with rows beyond the longest that the stage takes, with more keys than a block of the scan, and empty."""
import numpy as np
import pytest
import torch

from torchtt_gb300 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("s,m,S", [(1, 1, 1), (2, 5, 3), (3, 64, 3), (1, 200, 2), (7, 33, 1), (2, 300, 1)])
@pytest.mark.parametrize("density", [0.0, 0.02, 0.24, 0.4])
def test_random_sparse_core(s, m, S, density):
    g = np.random.default_rng(s * m * S)
    n = m
    A = g.standard_normal((s, m, n, S)) * (g.random((s, m, n, S)) < density)
    if density == 0.02:
        A[0, 0, :, 0] = 1.0   # one full row: longer than 64 where n is
    dev = torch.device("cuda", 0)
    put = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)
    r, R = 3, 5
    A, x = put(A), put(g.standard_normal((r, n, R)))
    phl, phr = put(g.standard_normal((r, s, r))), put(g.standard_normal((R, S, R)))

    def close(got, terms):
        ref, mag = terms(lambda t: t), terms(torch.abs)
        # FP64 sums of at most s n S r R terms in another order
        assert torch.all((got - ref).abs() <= 4 * (s * n + r + S * R) * 2.0 ** -53 * mag)

    close(ops.local_product(phr, phl, A, x),
          lambda f: torch.einsum("lsr,smnS,LSR,rnR->lmL", f(phl), f(A), f(phr), f(x)))
    y = put(g.standard_normal((r, m, R)))
    close(ops.compute_phi_fwd_A(phl, y, A, x),
          lambda f: torch.einsum("lsr,lmL,smnS,rnR->LSR", f(phl), f(y), f(A), f(x)))
    close(ops.compute_phi_bck_A(phr, y, A, x),
          lambda f: torch.einsum("LSR,lmL,smnS,rnR->lsr", f(phr), f(y), f(A), f(x)))
