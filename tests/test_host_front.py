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


@pytest.mark.parametrize("shape", [(4, 128), (1, 128), (2, 2, 32), (3, 96), (64, 1), ()])
def test_rows_of_another_length_are_refused(shape):
    """... also where their elements could be regrouped into rows of the right length."""
    w = torch.zeros((16, 64), dtype=torch.bfloat16)
    with pytest.raises(RuntimeError, match="rows of x"):
        pkg().qwen3.linear(torch.zeros(shape, dtype=torch.bfloat16), w, ctx=CTX)


@pytest.mark.parametrize("w", [{"q4": torch.zeros((16, 8, 1), dtype=torch.int32)}, {"q4h": torch.zeros((16, 1), dtype=torch.uint8)},
                               {"q": torch.zeros((16, 64, 1), dtype=torch.int8)}, torch.zeros((1, 16, 64), dtype=torch.bfloat16),
                               torch.zeros((64,), dtype=torch.bfloat16)])
def test_packed_weights_of_another_rank_are_refused(w):
    if isinstance(w, dict):
        w = dict(w, s=torch.zeros((16, 1), dtype=torch.bfloat16), b=torch.zeros((16, 1), dtype=torch.bfloat16))
    with pytest.raises(ValueError, match="dimensions"):
        pkg().qwen3.linear(torch.zeros((1, 64), dtype=torch.bfloat16), w, ctx=CTX)
