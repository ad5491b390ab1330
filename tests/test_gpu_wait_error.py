"""A digit product whose bounded wait gives up sets its thread's error word. Here the host sets the word, and
the next entry point that has waited for the GPU reports it, once and only to its own thread."""
import ctypes
import threading

import numpy as np
import pytest
import torch

from torchtt_gb300 import _lib, ops
from torchtt_gb300.errors import GB300Error

pytestmark = pytest.mark.gpu


def test_a_wait_that_gave_up_is_reported_once():
    word_of = getattr(_lib.lib(), "_ZN4ttgb15wait_error_wordEv")
    word_of.restype = ctypes.POINTER(ctypes.c_int)
    a = torch.from_numpy(np.random.default_rng(0).standard_normal((40, 9))).cuda()
    ops.qr(a)
    word = word_of()
    assert word[0] == 0
    word[0] = 1
    other = []

    def run():
        other.append(word_of()[0])
        other.append(ops.qr(a)[0].shape[1])

    t = threading.Thread(target=run)
    t.start()
    t.join()
    assert other == [0, 9]
    with pytest.raises(GB300Error, match="status 6.*wait gave up"):
        ops.qr(a)
    assert word[0] == 0
    ops.qr(a)
