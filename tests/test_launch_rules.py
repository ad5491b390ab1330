"""Rules of the kernel sources that no run can show reliably (no compute: read from the files): a kernel
launched while the kernel before it drains waits for that one, and reads global memory with plain loads."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "torchtt_gb300", "csrc")


def _text(path):
    text = re.sub(r"//[^\n]*", "", open(path).read())
    return re.sub(r"/\*.*?\*/", "", text, flags=re.S)


def _kernels(text):
    """name -> (signature, body) of the __global__ functions of a source."""
    out = {}
    for m in re.finditer(r"__global__", text):
        brace = text.index("{", m.end())
        head = text[m.end():brace]
        name = re.findall(r"(\w+_kernel)\s*\(", head)[-1]
        depth, i = 1, brace + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        out[name] = (head, text[brace:i])
    return out


def _early_launches():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = _text(path)
        kernels = _kernels(text)
        for inc in re.findall(r'#include "(\w+\.cuh)"', text):
            kernels = {**_kernels(_text(os.path.join(CSRC, inc))), **kernels}
        for name in sorted(set(re.findall(r"launch_early\(\s*(\w+)", text))):
            yield pytest.param(name, kernels, id="%s-%s" % (os.path.basename(path), name))


@pytest.mark.parametrize("name,kernels", list(_early_launches()))
def test_early_launched_kernels_wait(name, kernels):
    head, body = kernels[name]
    assert "stream_wait();" in body
    assert "__restrict__" not in head and "__ldg(" not in body


def test_blocks_decide_together_on_a_flag_of_their_own_launch():
    """The Arnoldi finishing pass writes the stop flag in one of its blocks while others may still be
    starting, so a block takes one decision from it for all of its threads."""
    _, body = _kernels(_text(os.path.join(CSRC, "gmres.cu")))["arnoldi_finish_kernel"]
    reads = [line.strip() for line in body.splitlines() if "flag[" in line]
    assert reads == ["if (__syncthreads_or(flag[kGmresState] != 0)) return;"]


def test_the_lane_that_issues_the_mmas_asks_for_their_completion():
    """A commit covers the MMAs of the executing thread only, so every commit of the digit product stands in
    the issuing lane's branches, and the barriers are initialised once."""
    _, body = _kernels(_text(os.path.join(CSRC, "oz_gemm.cu")))["oz_gemm_kernel"]
    issuer = body[body.index("elect_one()"):body.index("double* turn")]
    assert body.count("commit(smem") == issuer.count("commit(smem") == 3
    for i in (m.start() for m in re.finditer(r"commit\(smem", issuer)):
        before = issuer[:i]
        branch = before[before.rindex("if (leader) {"):]
        assert branch.count("{") > branch.count("}")
    assert "mbar_init" not in body[body.index("stream_wait();"):]


def test_kernels_called_in_place_promise_nothing():
    """jacobi_columns passes one buffer as the input and the output of the cluster Jacobi."""
    text = _text(os.path.join(CSRC, "linalg.cu"))
    launch = re.search(r"jacobi_block_kernel<EPL><<<[^>]*>>>\((\w+), n, (\w+),", text)
    assert launch.group(1) == launch.group(2)
    assert "__restrict__" not in _kernels(text)["jacobi_block_kernel"][0]
