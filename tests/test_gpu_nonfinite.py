"""Operators and right-hand sides that are not finite (GPU): GMRES and the sweep report them instead of taking a
residual that compares false with everything as converged."""
import numpy as np
import pytest
import torch

from torchtt_gb300 import TT, amen_solve, ops, workloads as W
from torchtt_gb300.errors import GB300Error

pytestmark = pytest.mark.gpu


def _local(r=6, n=7, R=5):
    g = np.random.default_rng(0)
    put = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    spd = lambda k: np.eye(k) + 0.1 * np.diag(g.random(k))
    return [put(spd(r)[:, None, :]), put(spd(n)[None, :, :, None]), put(spd(R)[:, None, :]),
            put(g.standard_normal((r, n, R)))]


@pytest.mark.parametrize("where", [0, 1, 2, 3])
@pytest.mark.parametrize("value", [float("nan"), float("inf"), 1e200])
def test_local_gmres(where, value):
    s = _local()
    if where == 3 and value == 1e200:
        value = 1e155   # its square is not finite
    s[where].view(-1)[0] = value
    with pytest.raises(GB300Error, match="status 3"):
        ops.local_gmres(*s, iters=20, threshold=1e-8, resets=2)
    x, flag, _ = ops.local_gmres(*_local(), iters=20, threshold=1e-8, resets=2)
    assert flag == 1 and torch.isfinite(x).all()


@pytest.mark.parametrize("max_full", [500, 0])   # direct and iterative local solves
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("bad", ["A", "b"])
def test_whole_solve(max_full, precision, bad):
    A = [c.cuda() for c in W.laplace_ttm(3, 8)]
    b = [c.cuda() for c in W.random_tt([8] * 3, [1, 2, 2, 1], 3)]
    c = (A if bad == "A" else b)
    c[1] = c[1].clone()
    c[1].view(-1)[0] = float("nan")
    with pytest.raises(GB300Error, match="status 3"):
        amen_solve(TT(A), TT(b), eps=1e-8, max_full=max_full, precision=precision)


def test_zero_right_hand_side_is_still_solved():
    A = TT([c.cuda() for c in W.laplace_ttm(3, 8)])
    b = TT([0.0 * c.cuda() for c in W.random_tt([8] * 3, [1, 2, 2, 1], 3)])
    for max_full in (500, 0):
        amen_solve(A, b, eps=1e-8, max_full=max_full, nswp=2)
