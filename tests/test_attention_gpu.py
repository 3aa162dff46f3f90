"""b200_attention_decode at the edges of its chunks and tiles, against a float64 softmax(q k^T) v."""
import numpy as np
import pytest

from util import pkg

pytestmark = pytest.mark.gpu


def _run(p, q, k, v, pos):
    import torch
    L = p.lib()
    B, H, D = q.shape
    KV, S = k.shape[1], k.shape[2]
    out = torch.empty_like(q)
    scratch = torch.empty(L.b200_attention_scratch_bytes(B, H, D, S) // 4, device="cuda")
    posd = torch.tensor([pos], dtype=torch.int32, device="cuda")
    p._lib.check(L.b200_attention_decode(p.default_context().handle, p._lib.current_stream(), q.data_ptr(), k.data_ptr(), v.data_ptr(),
                                         out.data_ptr(), posd.data_ptr(), scratch.data_ptr(), B, H, KV, D, S))
    torch.cuda.synchronize()
    return out.double()


def _reference(q, k, v, pos):
    import torch
    B, H, D = q.shape
    KV = k.shape[1]
    qg = q.double().reshape(B, KV, H // KV, D)
    s = torch.einsum("bkgd,bksd->bkgs", qg, k[:, :, :pos + 1].double()) * D ** -0.5
    return torch.einsum("bkgs,bkds->bkgd", torch.softmax(s, -1), v[..., :pos + 1].double()).reshape(B, H, D)


def _inputs(B, KV, G, D, S, pos, seed=0):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *shape: torch.randn(shape, generator=g, device="cuda").to(torch.bfloat16)
    q, k, v = r(B, KV * G, D), r(B, KV, S, D), r(B, KV, D, S)
    k[:, :, pos + 1:] = float("nan")       # what lies beyond the position may be anything
    v[..., pos + 1:] = float("nan")
    return q, k, v


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("G", [1, 2, 4, 8])
@pytest.mark.parametrize("S,pos", [(128, 0), (128, 7), (128, 63), (128, 64), (131, 65), (131, 130), (1000, 999), (4099, 4000)])
def test_edges(D, G, S, pos):
    q, k, v = _inputs(2, 2, G, D, S, pos)
    got, want = _run(pkg(), q, k, v, pos), _reference(q, k, v, pos)
    # one rounding to bf16 of a sum of f32 terms (of order one: probabilities times normal values)
    tol = 2.0 ** -8 * want.abs() + 2e-6
    assert bool(((got - want).abs() <= tol).all())


def test_infinite_values_stay_infinite():
    import torch
    p = pkg()
    q, k, v = _inputs(1, 2, 4, 128, 256, 200)
    v[0, 0, 5, 3], v[0, 1, 100, 199], v[0, 1, 7, 0] = float("inf"), float("-inf"), float("nan")
    got = _run(p, q, k, v, 200).reshape(2, 4, 128)
    assert bool((got[0, :, 5] == float("inf")).all()) and bool((got[1, :, 100] == float("-inf")).all())
    assert bool(torch.isnan(got[1, :, 7]).all()) and int((~torch.isfinite(got)).sum()) == 12


@pytest.mark.parametrize("D,G,pos,sigma", [(128, 4, 100, 1), (128, 4, 777, 1), (128, 1, 500, 1), (64, 8, 1000, 1), (64, 2, 500, 2)])
def test_partial_sums_keep_f32_precision(D, G, pos, sigma):
    """The merged f32 partials, before their rounding to bf16, within 2^-22 of float64 (2-norm): four roundings of one in f32, about what
    the sums of D scores and of 64 values may take.  Accumulator chains on the tensor core were at 1.3 to 1.5 times that."""
    import torch
    B, KV, S = 4, 8, (pos + 128) // 128 * 128
    p = pkg()
    L = p.lib()
    q, k, v = _inputs(B, KV, G, D, S, pos)
    q = (q.float() * sigma).to(torch.bfloat16)
    out, splits = torch.empty_like(q), (S + 63) // 64
    scratch = torch.empty(B * KV * splits * G * (D + 2), device="cuda")
    posd = torch.tensor([pos], dtype=torch.int32, device="cuda")
    p._lib.check(L.b200_attention_decode(p.default_context().handle, p._lib.current_stream(), q.data_ptr(), k.data_ptr(), v.data_ptr(),
                                         out.data_ptr(), posd.data_ptr(), scratch.data_ptr(), B, KV * G, KV, D, S))
    torch.cuda.synchronize()
    part = scratch.view(B, KV, splits, G, D + 2)[:, :, :pos // 64 + 1].double()
    e = torch.exp(part[..., D] - part[..., D].amax(2, keepdim=True))
    got = ((part[..., :D] * e[..., None]).sum(2) / (part[..., D + 1] * e).sum(2)[..., None]).reshape(B, KV * G, D)
    want = _reference(q, k, v, pos)
    assert float((got - want).norm() / want.norm()) <= 2.0 ** -22
