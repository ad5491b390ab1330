"""The FP64 contraction from digits made beforehand (GPU): the first core of a TT product is one GEMM, compared
with extended precision at the edges of its tiles, K chunks and operand sizes, for graded operands and
for infinities, NaN and subnormal numbers."""
import numpy as np
import pytest
import torch

from torchtt_gb300 import TT, ops

pytestmark = pytest.mark.gpu
U = 2.0 ** -53
CHUNK = 128


def gemm(a, b):
    dev = torch.device("cuda", 0)
    put = lambda v: torch.from_numpy(np.ascontiguousarray(v)).to(dev)
    y = TT([put(a[None, :, :, None]), put(np.ones((1, 1, 1, 1)))]) @ \
        TT([put(b[None]), put(np.ones((b.shape[1], 1, 1)))])
    return y.cores[0][0].cpu().numpy()


@pytest.fixture(autouse=True)
def heuristic_tiles():
    before, _ = ops.autotune(False)
    yield
    ops.autotune(before)


def _digit_bound(a, b):
    """What the digits leave out: 2^-57 of the scales per term and 2^-54 per chunk. The scales of a chunk
    are those of the smaller operand's columns Fq, and of the larger one's rows after each k was scaled by
    the largest that Fq leaves in it; exponents instead of values cost a factor 2."""
    q, p = (a.T, b.T) if a.shape[0] <= b.shape[1] else (b, a)      # q: k x rows, p: rows x k
    out = 0.0
    for k0 in range(0, a.shape[1], CHUNK):
        qc, pc = np.abs(q[k0:k0 + CHUNK]), np.abs(p[:, k0:k0 + CHUNK])
        f = qc.max(axis=0)
        kappa = (qc / np.where(f > 0, f, 1.0)).max(axis=1)
        e = (pc * kappa).max(axis=1)
        out = out + (qc.shape[0] * 2.0 ** -57 + 2.0 ** -54) * 2 * np.outer(e, f)
    return out.T if a.shape[0] <= b.shape[1] else out


@pytest.mark.parametrize("mnk", [(8, 30001, 129), (512, 513, 128), (129, 2049, 127), (2049, 129, 130),
                                 (97, 19393, 17), (300, 6000, 161), (6000, 50, 145), (161, 161, 5024)])
@pytest.mark.parametrize("kind", ["normal", "opposite", "graded", "zeros"])
def test_gemm_against_extended_precision(mnk, kind):
    m, n, k = mnk
    g = np.random.default_rng(m + n + k)
    a, b = g.standard_normal((m, k)), g.standard_normal((k, n))
    s = 10.0 ** np.linspace(0, -8, k)
    if kind == "opposite":
        a, b = a * s, b / s[:, None]
    elif kind == "graded":
        a = a * s * 10.0 ** g.uniform(-100, 100, (m, 1))
        b = b * 10.0 ** g.uniform(-100, 100, n)
    elif kind == "zeros":
        a[::3] = 0.0
        b[:, ::2] = 0.0
        b[::4] = 0.0
    c = gemm(a, b)
    # a sample of rows and columns that has the first and the last ones
    r = np.unique(np.linspace(0, m - 1, 40).astype(int))
    j = np.unique(np.linspace(0, n - 1, 700).astype(int))
    ld = np.longdouble
    ref = a[r].astype(ld) @ b[:, j].astype(ld)
    err = np.abs(c[np.ix_(r, j)] - ref)
    scale = np.abs(a[r]) @ np.abs(b[:, j])
    chunks = -(-k // CHUNK)
    assert np.all(err <= (2 * chunks + 2) * U * scale + _digit_bound(a, b)[np.ix_(r, j)])
    if kind != "zeros":   # as a whole no worse than FP64 multiply-adds
        assert np.linalg.norm((err / scale).astype(float)) <= 4 * U * np.sqrt(err.size)


@pytest.mark.parametrize("mnk", [(129, 2049, 130), (2049, 129, 130)])
def test_special_values(mnk):
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
