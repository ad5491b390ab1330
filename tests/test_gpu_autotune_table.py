"""Records of a tile table that name no candidate (GPU): their classes are tuned again and appended."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CODE = """
import torch
from torchtt_gb300 import ops
r = lambda *s: torch.randn(*s, dtype=torch.float64, device="cuda")
ops.local_product(r(19, 3, 19), r(22, 3, 22), r(3, 20, 20, 3), r(22, 20, 19))
torch.cuda.synchronize()
"""


def test_unknown_candidates_are_tuned_again(cuda, tmp_path):
    table = tmp_path / "tiles"

    def records():
        subprocess.run([sys.executable, "-c", CODE], cwd=ROOT, check=True,
                       env={**os.environ, "TTGB_AUTOTUNE_TABLE": str(table), "TTGB_AUTOTUNE": "1"})
        return [line.split() for line in table.read_text().splitlines()]

    first = records()
    assert len(first) == 3 and all(0 <= int(c) < 99 for _, c in first)
    assert records() == first
    table.write_text("".join("%s 99\n" % k for k, _ in first))
    again = records()
    assert [k for k, _ in again] == 2 * [k for k, _ in first]
    assert all(0 <= int(c) < 99 for _, c in again[3:])
