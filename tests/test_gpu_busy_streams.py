"""Whole calls beside other work (GPU): products and mixed solves on streams that are busy, several at once, give what
they give alone. The mixed solves run GMRES with a tolerated loss of orthogonality."""
import threading

import pytest
import torch

from torchtt_gb300 import TT, amen_mv, amen_solve, workloads as W

pytestmark = pytest.mark.gpu


def _together(calls):
    """The calls on a stream each, behind and beside matrix products that fill the GPU."""
    out, errors = [None] * len(calls), []

    def run(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                a = torch.randn(3000, 3000, device="cuda")
                for _ in range(4):
                    for _ in range(4):
                        a = torch.tanh(a @ a)
                    out[i] = calls[i]()
        except Exception as e:   # an error in a thread fails the test
            errors.append(e)

    threads = [threading.Thread(target=run, args=(i,)) for i in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    torch.cuda.synchronize()
    return out


def test_amen_mv(cuda):
    A = TT([c.to(cuda) for c in W.laplace_potential_ttm(8, 16)])
    xs = [TT([c.to(cuda) for c in W.random_tt([16] * 8, [1] + [5] * 7 + [1], 20 + i)]) for i in range(4)]
    exact = [A @ x for x in xs]
    torch.cuda.synchronize()
    for y, e in zip(_together([lambda x=x: amen_mv(A, x, eps=1e-8) for x in xs]), exact):
        assert float((y - e).norm() / e.norm()) <= 1e-7


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_solves(cuda, precision):
    A = TT([c.to(cuda) for c in W.laplace_ttm(4, 16)])
    bs = [TT([c.to(cuda) for c in W.random_tt([16] * 4, [1, 4, 4, 4, 1], 40 + i)]) for i in range(4)]
    solve = lambda b: amen_solve(A, b, eps=1e-8, max_full=0, seed=1, precision=precision).full()
    alone = [solve(b) for b in bs]
    torch.cuda.synchronize()
    for x, y in zip(_together([lambda b=b: solve(b) for b in bs]), alone):
        # both solve the same system to the same tolerance (condition 120)
        assert float((x - y).norm() / y.norm()) <= 120 * 1e-8
