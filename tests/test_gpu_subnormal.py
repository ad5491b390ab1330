"""Subnormal numbers in the digit products (GPU): they have digits as any other number, with results that are normal
or subnormal, and cost no more."""
import numpy as np
import pytest
import torch

from torchtt_gb300 import TT, ops

pytestmark = pytest.mark.gpu
U = 2.0 ** -53
SIZES = [(300, 200, 100), (300, 6000, 161)]   # digits made per tile and beforehand


def _tts(a, b):
    put = lambda v: torch.from_numpy(np.ascontiguousarray(v)).cuda()
    return (TT([put(a[None, :, :, None]), put(np.ones((1, 1, 1, 1)))]),
            TT([put(b[None]), put(np.ones((b.shape[1], 1, 1)))]))


@pytest.fixture(autouse=True)
def heuristic_tiles():
    before, _ = ops.autotune(False)
    yield
    ops.autotune(before)


@pytest.mark.parametrize("mnk", SIZES)
@pytest.mark.parametrize("top", [1.0, 1e-150, 1e250])
def test_values(mnk, top):
    m, n, k = mnk
    g = np.random.default_rng(k)
    a, b = g.standard_normal((m, k)), top * g.standard_normal((k, n))
    a[1] = 5e-310 * g.standard_normal(k)      # a subnormal row, two at the bottom of the range
    a[2] = 4.9e-324
    a[3] = 4.9e-324 * g.integers(0, 9, k)
    a[5::7, ::3] = 3e-312
    b[:, 4] = 2e-311 * g.standard_normal(k)   # and a subnormal column
    x, y = _tts(a, b)
    cols = np.r_[0:8, 8:n:n // 60]   # a sample of the columns
    c = (x @ y).cores[0][0].cpu().numpy()[:, cols]
    # the scale of a k is that of all columns
    bk = np.abs(b).max(axis=1).astype(np.longdouble)
    b = b[:, cols]
    ld = np.longdouble
    ref, mag = a.astype(ld) @ b.astype(ld), np.abs(a).astype(ld) @ np.abs(b).astype(ld)
    # scales of a row and a column as in the tests of normal numbers, and the last place of the result
    rows = (np.abs(a) * bk).max(axis=1)
    cols = (np.abs(b) / bk[:, None]).max(axis=0)
    bound = (k + 2) * U * mag + k * ld(2.0) ** -53 * np.outer(rows, cols) + ld(2.0) ** -1074
    assert np.all(np.abs(c - ref) <= bound)


@pytest.mark.parametrize("mnk", SIZES)
def test_time(mnk):
    m, n, k = mnk
    g = np.random.default_rng(0)
    a, b = g.standard_normal((m, k)), g.standard_normal((k, n))

    def us(a, b):
        x, y = _tts(a, b)
        t = []
        for _ in range(10):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            x @ y
            e[1].record()
            torch.cuda.synchronize()
            t.append(e[0].elapsed_time(e[1]))
        return min(t)

    plain = us(a, b)
    a[0, 0] = b[0, 0] = 5e-310
    assert us(a, b) <= 1.5 * plain   # computed in multiply-adds the larger product took 3.4 times as long
