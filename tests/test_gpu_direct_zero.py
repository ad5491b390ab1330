"""The dense local solve of b = 0 (GPU): zero for a regular matrix, and for a singular one or one with a NaN not a
number, as the elimination gives it."""
import numpy as np
import pytest
import torch

from torchtt_gb300 import TT, amen_solve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 16, 33, 200, 512])
@pytest.mark.parametrize("kind", ["regular", "singular", "zero", "nan first", "nan last"])
def test_zero_right_hand_side(n, kind):
    g = np.random.default_rng(n)
    a = np.linalg.qr(g.standard_normal((n, n)))[0] * np.linspace(1.0, 10.0, n)
    if kind == "singular":
        a[:, n // 2] = 0.0
    elif kind == "zero":
        a[:] = 0.0
    elif kind.startswith("nan"):
        a[(0, 0) if kind == "nan first" else (n - 1, n - 1)] = np.nan
    put = lambda v: torch.from_numpy(np.ascontiguousarray(v)).cuda()
    x = amen_solve(TT([put(a[None, :, :, None])]), TT([put(np.zeros((1, n, 1)))]), max_full=600, nswp=1)
    x = x.cores[0]
    if kind == "regular":
        assert float(x.abs().max()) == 0.0
    else:
        assert not torch.isfinite(x).all()
