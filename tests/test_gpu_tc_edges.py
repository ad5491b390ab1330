"""The tcgen05 local product at the edges of its output tiles (GPU): the last GEMM's columns L at and around
16, 32, 64 and 128, its rows at remainders of 32 and 128, which its epilogue turns in shared memory."""
import numpy as np
import pytest
import torch

from oracle import amen as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R", [1, 15, 16, 17, 31, 33, 63, 65, 127, 128, 129])
@pytest.mark.parametrize("rn", [(1, 3), (3, 11), (11, 12)])
def test_tc_local_product_edges(cuda, rn, R):
    from torchtt_gb300 import ops
    r, n = rn
    g = np.random.default_rng(100 * R + r)
    PhiL, A = g.standard_normal((r, 2, r)), g.standard_normal((2, n, n, 2))
    PhiR, x = g.standard_normal((R, 2, R)), g.standard_normal((r, n, R))
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
    y = ops.local_product_lowp(t(PhiR), t(PhiL), t(A), t(x), engine=ops.ENGINE_TC).cpu().numpy()
    # each of the three products keeps 2^-21 of its terms' absolute values
    terms = O.local_product(np.abs(PhiR), np.abs(PhiL), np.abs(A), np.abs(x))
    assert np.all(np.abs(y - O.local_product(PhiR, PhiL, A, x)) <= 4 * 2.0 ** -21 * terms)
