"""The 8 x 8 tiles of the FP64 contraction (GPU): the first core of a TT product is one GEMM, compared with
extended precision at the edges of the tiles and of the slices of a K chunk."""
import numpy as np
import pytest
import torch

from torchtt_gb300 import TT, ops

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def gemm(a, b):
    dev = torch.device("cuda", 0)
    put = lambda v: torch.from_numpy(np.ascontiguousarray(v)).to(dev)
    y = TT([put(a[None, :, :, None]), put(np.ones((1, 1, 1, 1)))]) @ \
        TT([put(b[None]), put(np.ones((b.shape[1], 1, 1)))])
    return y.cores[0][0].cpu().numpy()


@pytest.mark.parametrize("k", [1, 7, 8, 9, 31, 32, 33, 64, 65, 200])
@pytest.mark.parametrize("mn", [(1, 1), (8, 8), (7, 9), (9, 7), (17, 24), (40, 240), (5, 600)])
def test_small_tiles(mn, k):
    g = np.random.default_rng(1000 * k + mn[0])
    a, b = g.standard_normal((mn[0], k)), g.standard_normal((k, mn[1]))
    before, _ = ops.autotune(False)
    try:
        c = gemm(a, b)
    finally:
        ops.autotune(before)
    ld = np.longdouble
    # k multiply-adds in four partial sums, three adds
    assert np.all(np.abs(c - a.astype(ld) @ b.astype(ld)) <= (k + 3) * U * (np.abs(a).astype(ld) @ np.abs(b)))
