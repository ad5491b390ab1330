"""GMRES on several streams at once (GPU): the passes of one solve meet others' blocks on the SMs, so that blocks of
a launch start late; every solve gives the bits that it gives alone. Operators near the identity take
the second projection and the directly computed norms, the others one projection."""
import threading

import numpy as np
import pytest
import torch

from torchtt_gb300 import ops

pytestmark = pytest.mark.gpu


def _spd(k, cond, g):
    q = np.linalg.qr(g.standard_normal((k, k)))[0]
    return (q * np.linspace(1.0, cond, k)) @ q.T


def _system(seed, cond, dev):
    g = np.random.default_rng(seed)
    put = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)
    r, n, R = 16 + seed, 20, 18
    return (put(_spd(r, cond, g)[:, None, :]), put(_spd(n, cond, g)[None, :, :, None]),
            put(_spd(R, cond, g)[:, None, :]), put(g.standard_normal((r, n, R))))


@pytest.mark.parametrize("cond,iters", [(1.0001, 12), (1.05, 20), (2.0, 40)])
def test_solves_on_many_streams_equal_single_ones(cond, iters):
    dev = torch.device("cuda", 0)
    before, _ = ops.autotune(False)   # tiles chosen by time could differ from run to run
    try:
        systems = [_system(i, cond, dev) for i in range(6)]
        solve = lambda s: ops.local_gmres(*s, iters=iters, threshold=1e-9, resets=3)
        alone = [solve(s) for s in systems]
        torch.cuda.synchronize()
        failures = []

        def work(i):
            try:
                with torch.cuda.stream(torch.cuda.Stream(dev)):
                    for _ in range(10):
                        x, flag, nit = solve(systems[i])
                        if flag != alone[i][1] or nit != alone[i][2] or not torch.equal(x, alone[i][0]):
                            failures.append(i)
            except Exception as e:   # an error in a thread fails the test
                failures.append(e)

        threads = [threading.Thread(target=work, args=(i,)) for i in range(6)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not failures
    finally:
        ops.autotune(before)
