"""b200_sample against the NumPy restatement of the reference's sample() (oracle/sampling.py):
greedy, temperature, top-k, top-k + top-p, ties, and the argument errors the reference raises."""
import numpy as np
import pytest

from oracle import sampling
from util import dev, host, pkg

pytestmark = pytest.mark.gpu


def _run(p, logits, u, **kw):
    import torch
    ld = dev(logits.astype(np.float32))
    ud = dev(u.astype(np.float32)) if u is not None else None
    out = p.qwen3.sample(ld, ud, **kw)
    torch.cuda.synchronize()
    return host(out)


@pytest.mark.parametrize("B,V", [(3, 1000), (2, 151936), (5, 4099), (2, 16384), (2, 16385), (96, 30000), (128, 70001)])
def test_greedy(B, V):
    p = pkg()
    rng = np.random.default_rng(1)
    logits = rng.standard_normal((B, V)).astype(np.float32) * 3
    logits[0, 7] = logits[0, V - 3] = logits[0].max() + 1       # a tie: the lower index wins
    got = _run(p, logits, None, temperature=0.0)
    want, _ = sampling.sample(logits, None, 0.0)
    assert np.array_equal(got, want) and got[0] == 7


@pytest.mark.parametrize("kw", [dict(temperature=0.8), dict(temperature=1.3, top_k=50), dict(temperature=0.7, top_k=1024),
                                dict(temperature=1.0, top_k=40, top_p=0.9), dict(temperature=0.5, top_k=200, top_p=0.5),
                                dict(temperature=2.0, top_k=1), dict(temperature=1.0, top_k=64, top_p=1e-6)])
@pytest.mark.parametrize("V", [2048, 151936])
def test_sampling_matches_the_oracle(kw, V):
    p = pkg()
    rng = np.random.default_rng(7)
    B = 24
    logits = (rng.standard_normal((B, V)) * 3).astype(np.float32)
    logits[1, :100] = logits[1, 100]                             # many equal values around the top-k boundary
    logits[2] = np.round(logits[2])                              # heavy ties everywhere
    u = rng.random(B).astype(np.float32)
    u[0], u[3] = 0.0, np.float32(1.0 - 2 ** -24)                 # the ends of the range
    got = _run(p, logits, u, **kw)
    want, margin = sampling.sample(logits, u.astype(np.float64), **kw)
    # draws whose target sits within f32 rounding of a CDF step may legitimately land on the neighbour
    sure = margin > 1e-4
    assert sure.sum() >= B // 2
    assert np.array_equal(got[sure], want[sure]), (kw, got, want)
    # every draw, sure or not, is one of the candidates the reference would keep
    if kw.get("top_k"):
        for r in range(B):
            z = logits[r].astype(np.float64)
            kth = np.sort(z)[::-1][kw["top_k"] - 1]
            assert z[got[r]] >= kth


@pytest.mark.parametrize("B,V,k", [(3, 50257, 50), (18, 50257, 50), (19, 50257, 50), (2, 1, 1), (3, 700, 700), (3, 1024, 1), (3, 1025, 1024),
                                   (3, 8193, 1000), (2, 1 << 19, 40), (33, 2050, 2), (2, 40000, 0), (33, 4099, 0), (2, 131072, 0),
                                   (2, 1 << 19, 0), (2, 37, 0),
                                   # one CTA per row, and the last batch that clusters take
                                   (112, 1, 1), (112, 33, 33), (80, 4099, 50), (79, 4099, 50), (96, 16384, 255), (160, 32001, 3), (112, 1025, 1024), (96, 50257, 256),
                                   (96, 32000, 0), (95, 32000, 0), (37, 16384, 0), (36, 9000, 0)])
def test_shares_of_a_row(B, V, k):
    """Around the limits of a CTA's share: empty shares, fewer logits than threads, shares beyond shared memory."""
    rng = np.random.default_rng(V + k)
    logits = (rng.standard_normal((B, V)) * 3).astype(np.float32)
    logits[0] = 1.5                                              # one long run of equals
    if V > 5:
        logits[1, 5:] = -np.inf
    u = rng.random(B).astype(np.float32)
    got = _run(pkg(), logits, u, temperature=0.9, top_k=k)
    want, margin = sampling.sample(logits, u.astype(np.float64), temperature=0.9, top_k=k)
    # the largest cumulative sum is V terms of f32: its rounding (below V * 2^-24, in units of the total) decides nothing else
    sure = margin > max(1e-4, V * 2.0 ** -24)
    assert np.array_equal(got[sure], want[sure])
    assert np.all((got >= 0) & (got < V)) and (V <= 5 or got[1] < 5)


def test_nan_and_infinite_rows():
    for V in (5000, 40000):
        _nan_and_infinite_rows(V)


def _nan_and_infinite_rows(V):
    logits = np.zeros((100, V), np.float32)
    logits[0] = -np.inf
    logits[1] = np.nan
    logits[2, 77] = np.inf
    logits[3, ::2] = -np.nan
    for B in (4, 100):
        for kw in (dict(temperature=0.0), dict(temperature=1.0), dict(temperature=1.0, top_k=30), dict(temperature=1.0, top_k=1024, top_p=0.5)):
            got = _run(pkg(), logits[:B], np.full(B, 0.5, np.float32), **kw)
            assert np.all((got >= 0) & (got < V)), kw
            if kw["temperature"] == 0.0:
                assert got[2] == 77 and got[0] == 0


def test_refusals():
    import torch
    p = pkg()
    L, lib = p._lib, p.lib()
    ctx = p.default_context()
    x = torch.zeros((2, 100), device="cuda")
    u = torch.zeros((2,), device="cuda")
    o = torch.zeros((2,), dtype=torch.int32, device="cuda")
    call = lambda t, k, pp, uu: lib.b200_sample(ctx.handle, L.current_stream(), x.data_ptr(), 2, 100, t, k, pp,
                                                uu.data_ptr() if uu is not None else None, o.data_ptr())
    assert call(-0.1, 0, 1.0, u) == L.INVALID_ARGUMENT and b"temperature" in lib.b200_last_error()
    assert call(1.0, 101, 1.0, u) == L.INVALID_ARGUMENT and b"top_k" in lib.b200_last_error()
    assert call(1.0, -1, 1.0, u) == L.INVALID_ARGUMENT
    assert call(1.0, 0, 0.9, u) == L.UNIMPLEMENTED
    assert call(1.0, 10, 0.9, None) == L.INVALID_ARGUMENT
    assert call(0.0, 0, 1.0, None) == L.OK
    assert ctx.error() == 0


def test_numbers_of_any_type():
    """top_k, top_p and temperature are numbers: what int() and float() take."""
    import torch
    rng = np.random.default_rng(5)
    logits, u = rng.standard_normal((2, 500)).astype(np.float32), rng.random(2).astype(np.float32)
    want = _run(pkg(), logits, u, temperature=0.75, top_k=20, top_p=0.5)
    got = _run(pkg(), logits, u, temperature=np.float32(0.75), top_k=20.0, top_p=torch.tensor(0.5))
    assert np.array_equal(got, want)


@pytest.mark.parametrize("rows", [24, 4096])
@pytest.mark.parametrize("kw", [dict(), dict(top_k=100), dict(top_k=1000, top_p=0.9)])
def test_the_draw_is_monotone_in_the_uniform_number(rows, kw):
    """An inverse CDF: of rows with the same logits, a larger number never draws an earlier candidate.  The numbers lie within 4 steps of f32 around
    the edges between candidates (or chunks), where sums formed in different orders overlap and leave gaps."""
    import torch
    p = pkg()
    rng = np.random.default_rng(3)
    V, T = 2050, 0.7
    logits = (rng.standard_normal(V) * 2).astype(np.float32)
    order = np.argsort(-logits, kind="stable")[:kw["top_k"]] if kw else np.arange(V)
    pr = np.exp((logits[order].astype(np.float64) - logits.max()) / T)
    if "top_p" in kw:
        pr = pr[:np.searchsorted(np.cumsum(pr), kw["top_p"] * pr.sum()) + 1]
    edges = np.cumsum(pr)[:-1] / pr.sum()
    u = np.sort(np.concatenate([np.float32(edges) + np.float32(2.0 ** -24) * i for i in range(-4, 5)])).astype(np.float32)
    u = u[(u > 0) & (u < 1)]
    place = np.full(V, -1)
    place[order] = np.arange(len(order))
    got = []
    for i in range(0, len(u), rows):
        part = u[i:i + rows]
        ld = dev(logits)[None].expand(len(part), V).contiguous()
        got.append(host(p.qwen3.sample(ld, dev(part), temperature=T, **kw)))
    at = place[np.concatenate(got)]
    assert (at >= 0).all() and (np.diff(at) >= 0).all(), np.flatnonzero(np.diff(at) < 0)[:10]


def test_no_draw_of_an_impossible_token():
    """Tokens masked with -inf have probability zero: not drawn whatever the number, the largest included."""
    rng = np.random.default_rng(4)
    for V in (1000, 50257):
        logits = rng.standard_normal((64, V)).astype(np.float32)
        logits[:, rng.permutation(V)[:V - 30]] = -np.inf
        u = np.concatenate([rng.random(60), [0.0, 1 - 2.0 ** -24, 1 - 2.0 ** -23, 0.5]]).astype(np.float32)
        for B in (64, 20):
            for kw in (dict(), dict(top_k=25)):
                got = _run(pkg(), logits[:B], u[64 - B:], temperature=0.9, **kw)
                assert np.isfinite(logits[np.arange(B), got]).all()
