"""The Python front's native per-call code: what it has to refuse before anything is launched.  CPU only: a context
without a library object behind it stands in for a real one, so a call that passed its checks would raise something else."""
import ctypes
import types

import pytest
import torch

from util import pkg

CTX = types.SimpleNamespace(handle=ctypes.c_void_p(0))


def test_an_int8_weight_without_scales_is_an_error():
    """(An integer division by their number would end the process.)"""
    w = {"q": torch.zeros((16, 64), dtype=torch.int8), "s": torch.zeros((16, 0), dtype=torch.bfloat16)}
    with pytest.raises(ZeroDivisionError):
        pkg().qwen3.linear(torch.zeros((1, 64), dtype=torch.bfloat16), w, ctx=CTX)
