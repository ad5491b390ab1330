"""The FP64 contraction kernels (GPU), the tensor-core one among them: the first core of a TT product
is one GEMM, compared with extended precision at the edges of tiles and K chunks, for graded
operands, and for infinities, NaN and subnormal numbers."""
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


@pytest.fixture(params=[False, True], ids=["heuristic", "tuned"])
def tuning(request):
    before, _ = ops.autotune(request.param)
    yield
    ops.autotune(before)


def _operands(kind, m, n, k, g):
    a, b = g.standard_normal((m, k)), g.standard_normal((k, n))
    s = 10.0 ** np.linspace(0, -8, k)
    if kind == "opposite":       # a_ik b_kj even, a_ik and b_kj graded over 8 decades
        a, b = a * s, b / s[:, None]
    elif kind == "graded":       # rows, columns and the sum graded
        a = a * s * 10.0 ** g.uniform(-100, 100, (m, 1))
        b = b * 10.0 ** g.uniform(-100, 100, n)
    elif kind == "zeros":
        a[::3] = 0.0
        b[:, ::2] = 0.0
        b[::4] = 0.0
    return a, b


@pytest.mark.parametrize("mnk", [(1, 1, 1), (7, 5, 3), (64, 32, 64), (65, 33, 65), (200, 300, 100),
                                 (300, 200, 129), (100, 700, 64), (97, 701, 67), (3000, 16, 100),
                                 (3001, 9, 193), (16, 3000, 100), (5, 4099, 257), (257, 129, 513)])
@pytest.mark.parametrize("kind", ["normal", "opposite", "graded", "zeros"])
def test_gemm_against_extended_precision(tuning, mnk, kind):
    m, n, k = mnk
    a, b = _operands(kind, m, n, k, np.random.default_rng(m + n + k))
    c = gemm(a, b)
    ld = np.longdouble
    ref = a.astype(ld) @ b.astype(ld)
    # a row's and a column's scale: the largest |a_ik| |b_kj| over j bounds the terms of row i, and the
    # largest |b_kj| relative to its row those of column j
    bk = np.abs(b).max(axis=1)
    rows = (np.abs(a) * bk).max(axis=1)
    cols = (np.abs(b) / np.where(bk > 0, bk, 1.0)[:, None]).max(axis=0)
    # one rounding per 64-element chunk or multiply-add of a native tile, and digits down to 2^-57 of
    # the scales, K of them at most
    bound = (k + 2) * U * (np.abs(a).astype(ld) @ np.abs(b).astype(ld)) + \
        k * 2.0 ** -56 * np.outer(rows, cols)
    assert np.all(np.abs(c - ref) <= bound)
    # as a whole no worse than FP64 multiply-adds, whose error grows with the square root of K
    if kind != "zeros" and k > 16:
        assert np.linalg.norm(((c - ref) / np.outer(rows, cols)).astype(float)) <= \
            4 * np.sqrt(k) * U * np.linalg.norm((ref / np.outer(rows, cols)).astype(float))


@pytest.mark.parametrize("mnk", [(7, 5, 3), (300, 200, 129), (100, 700, 64)])
def test_special_values(tuning, mnk):
    m, n, k = mnk
    g = np.random.default_rng(3)
    a, b = g.standard_normal((m, k)), g.standard_normal((k, n))
    a[0, 0], a[2, 1], b[1, 3] = np.inf, np.nan, -np.inf
    a[4], b[:, 1] = 5e-310, 3.0
    with np.errstate(all="ignore"):
        ref = a @ b
    c = gemm(a, b)
    assert np.array_equal(np.isnan(c), np.isnan(ref))
    assert np.array_equal(c[np.isinf(ref)], ref[np.isinf(ref)])
    fin = np.isfinite(ref)
    assert np.all(np.abs(c[fin] - ref[fin]) <= 8 * k * U * (np.abs(ref[fin]) + np.abs(ref[fin]).max()))
    assert abs(c[4, 1] - ref[4, 1]) <= 8 * k * U * abs(ref[4, 1])
