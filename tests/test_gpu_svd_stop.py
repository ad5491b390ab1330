"""The stop of the FP64 Jacobi sweeps (GPU): a triangular factor whose rows are far apart in norm and orthogonal
to some 1e-6. The first sweep turns by tiny angles only, but it leaves cosines of the square of those it
found, so another one is due before the right singular vectors are orthogonal."""
import numpy as np
import pytest
import torch

from torchtt_gb300 import ops

pytestmark = pytest.mark.gpu
EPS = 2.220446049250313e-16


@pytest.mark.parametrize("n,ratio", [(3, 1e5), (3, 1e6), (4, 1e4), (5, 1e3), (8, 50.0), (15, 6.0)])
@pytest.mark.parametrize("off", [1e-7, 1e-6, 3e-6])
def test_graded_rows_end_orthogonal(n, ratio, off):
    g = np.random.default_rng(n)
    d = ratio ** -np.arange(n, dtype=float)
    a = d[:, None] * (np.eye(n) + off * np.triu(g.standard_normal((n, n)), 1))
    u, s, vh = (v.cpu().numpy() for v in ops.svd(torch.from_numpy(a).cuda()))
    assert np.linalg.norm(vh @ vh.T - np.eye(n)) <= 64 * n * EPS   # as in the other SVD tests
    assert np.linalg.norm((u * s) @ vh - a) <= 16 * n * EPS * np.linalg.norm(a)
