"""FP64 contractions with more row tiles than a grid has in its second dimension (GPU): as multiply-adds, with a
triangular right factor (the Q of a tall QR) and in double-float arithmetic."""
import numpy as np
import pytest
import torch

from torchtt_gb300 import TT, ops

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


@pytest.fixture(params=[False, True], ids=["heuristic", "tuned"])
def tuning(request):
    before, _ = ops.autotune(request.param)
    yield
    ops.autotune(before)


@pytest.mark.parametrize("m,k,n", [(2_097_121, 1, 1), (2_200_003, 1, 1), (4_300_001, 2, 3)])
@pytest.mark.parametrize("adds", [False, True])
def test_products(tuning, m, k, n, adds):
    g = torch.Generator(device="cuda").manual_seed(m)
    a = torch.randn(m, k, generator=g, dtype=torch.float64, device="cuda")
    b = torch.randn(k, n, generator=g, dtype=torch.float64, device="cuda")
    one = torch.ones(1, 1, 1, dtype=torch.float64, device="cuda")
    with ops.fp64_multiply_adds(adds):
        y = TT([a[None, :, :, None].contiguous(), one[..., None]]) @ TT([b[None].contiguous(),
                                                                        one.expand(n, 1, 1).contiguous()])
    c = y.cores[0][0]
    ref = (a[:, :, None] * b[None]).sum(dim=1)
    assert torch.all((c - ref).abs() <= 2 * (k + 2) * U * (a[:, :, None] * b[None]).abs().sum(dim=1).max())


@pytest.mark.parametrize("m,n", [(2_200_003, 2), (2_097_153, 5)])
def test_qr(tuning, m, n):
    a = torch.randn(m, n, generator=torch.Generator(device="cuda").manual_seed(n), dtype=torch.float64, device="cuda")
    q, r = ops.qr(a)
    eps = 2.0 ** -52
    assert float((q.T @ q - torch.eye(n, dtype=torch.float64, device="cuda")).norm()) <= 16 * n * eps
    assert float((q @ r - a).norm()) <= 16 * n * eps * float(a.norm())
