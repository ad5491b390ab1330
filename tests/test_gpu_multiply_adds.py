"""FP64 products as multiply-adds (GPU): where a caller asks for them, every element keeps its own digits, also
those far below the scales of their row and column, which the digit products round to these scales."""
import numpy as np
import pytest
import torch

from torchtt_gb300 import TT, amen_solve, ops, workloads as W

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def gemm(a, b):
    dev = torch.device("cuda", 0)
    put = lambda v: torch.from_numpy(np.ascontiguousarray(v)).to(dev)
    y = TT([put(a[None, :, :, None]), put(np.ones((1, 1, 1, 1)))]) @ \
        TT([put(b[None]), put(np.ones((b.shape[1], 1, 1)))])
    return y.cores[0][0].cpu().numpy()


@pytest.fixture(params=[False, True], ids=["heuristic", "tuned"])
def tuning(request):
    before, _ = ops.autotune(request.param)
    yield
    ops.autotune(before)


# sizes of the 16 x 16 tiles, of the digits made per tile and of those made beforehand
@pytest.mark.parametrize("mnk", [(20, 30, 40), (300, 200, 100), (300, 6000, 161)])
def test_elements_keep_their_own_digits(tuning, mnk):
    m, n, k = mnk
    g = np.random.default_rng(m)
    a, b = g.standard_normal((m, k)), g.standard_normal((k, n))
    a[:, k // 2:] *= 2.0 ** -50   # rows (1, e) and columns (e, 1) or (1, e): every scale is 1
    b[: k // 2, ::2] *= 2.0 ** -50
    b[k // 2:, 1::2] *= 2.0 ** -50
    with ops.fp64_multiply_adds():
        c = gemm(a, b)
    ld = np.longdouble
    j = np.unique(np.linspace(0, n - 1, 300).astype(int))   # a sample of the columns, both kinds
    c, b = c[:, j], b[:, j]
    assert np.all(np.abs(c - a.astype(ld) @ b.astype(ld)) <= (k + 2) * U * (np.abs(a).astype(ld) @ np.abs(b)))
    x = g.standard_normal((m, n)) * 10.0 ** g.uniform(-12, 0, (m, n))
    with ops.fp64_multiply_adds():
        assert np.array_equal(gemm(np.eye(m), x), x)


def test_a_solve_takes_them_too():
    from torchtt_gb300.solvers import solve_cores
    dev = torch.device("cuda", 0)
    A = [c.to(dev) for c in W.laplace_ttm(4, 24)]
    b = [c.to(dev) for c in W.random_tt([24] * 4, [1, 5, 5, 5, 1], 3)]
    x = TT(solve_cores(A, b, eps=1e-8, max_full=0, seed=2, fp64_engine="native")[0]).full()
    with ops.fp64_multiply_adds():
        y = amen_solve(TT(A), TT(b), eps=1e-8, max_full=0, seed=2).full()
    assert ops._lib.lib().ttgb_fp64_multiply_adds(-1) == 0
    # both solve the same system to the same tolerance (condition 250)
    assert float((x - y).norm() / y.norm()) <= 250 * 1e-8
