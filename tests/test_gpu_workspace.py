"""The workspace of the digit products (GPU) stays within what an admitted request reserves: a batch of many
short rows, whose digits would mostly be padding, takes a kernel without one."""
import numpy as np
import pytest
import torch

from torchtt_gb300 import ops
from torchtt_gb300.serving import pool_usage

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


@pytest.mark.parametrize("rl,n", [(4000, 128), (400, 1500)])
def test_short_rows_in_many_batch_entries(rl, n):
    g = np.random.default_rng(rl)
    put = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    m = R = 8
    phl, phr = put(g.standard_normal((rl, 1, 1))), put(g.standard_normal((3, 1, R)))
    A, x = put(g.standard_normal((1, m, n, 1))), put(g.standard_normal((1, n, R)))
    before, _ = ops.autotune(False)
    try:
        torch.cuda.synchronize()
        pool_usage(reset_high=True)
        base, _ = pool_usage()
        y = ops.local_product(phr, phl, A, x)
        torch.cuda.synchronize()
        _, high = pool_usage()
    finally:
        ops.autotune(before)
    # the two intermediates, and at most 48 bytes per element of the larger operand and 4 MiB
    assert high - base <= 8 * rl * R * (n + m) + 48 * rl * n * R + (8 << 20)
    terms = lambda f: torch.einsum("lsr,smnS,LSR,rnR->lmL", f(phl), f(A), f(phr), f(x))
    assert torch.all((y - terms(lambda t: t)).abs() <= 4 * (n + R + 1) * U * terms(torch.abs).max())
