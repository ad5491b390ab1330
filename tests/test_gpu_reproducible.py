"""Small solves (GPU) give the same bits in every process: no tile of theirs is chosen by time."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CODE = """
import hashlib
from torchtt_gb300 import TT, amen_solve, ops, workloads as W
h = hashlib.sha256()
for seed in range(5):
    w = W.small_random_system(seed)
    x = amen_solve(TT([c.cuda() for c in w["A"]]), TT([c.cuda() for c in w["b"]]), eps=1e-10)
    for c in x.cores:
        h.update(c.cpu().numpy().tobytes())
print(ops.autotune()[1], h.hexdigest())
"""


def test_small_solves_repeat_bit_for_bit(cuda):
    env = {**os.environ, "TTGB_AUTOTUNE": "1"}
    env.pop("TTGB_AUTOTUNE_TABLE", None)
    runs = {subprocess.run([sys.executable, "-c", CODE], cwd=ROOT, env=env, check=True, capture_output=True,
                           text=True).stdout for _ in range(4)}
    assert len(runs) == 1 and runs.pop().startswith("0 ")
