"""linear() with 9 rows of x and more at the sizes where its kernels can go wrong: tiles, slices of K, boxes and groups that
end early, rows that allow no wide loads.  The reference is a float64 product with the f32 weights of dequantize()."""
import numpy as np
import pytest

from util import pkg

pytestmark = pytest.mark.gpu


def _weight(p, kind, n, k, seed):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    w = torch.randn((n, k), generator=g, device="cuda") * 0.02
    if kind == "bf16":
        return w.to(torch.bfloat16), w.to(torch.bfloat16).double()
    q = p.qwen3.quantize_int4(w) if kind.startswith("int4") else p.qwen3.quantize_int8(w, 64 if kind == "int8_g64" else None)
    if kind == "int4_half":   # the reference's split-half bytes of the same values
        words = q["q4"].cpu().numpy().view(np.uint32)
        nib = ((words[:, :, None] >> (4 * np.arange(8, dtype=np.uint32))) & 15).reshape(n, k // 64, 64).astype(np.uint8)
        q = {"q4h": torch.from_numpy(nib[:, :, :32] | (nib[:, :, 32:] << 4)).cuda(), "s": q["s"], "b": q["b"]}
    return q, p.qwen3.dequantize(q, torch.float32).double()


def _check(p, m, n, k, kind, form="plain", pad=0, shift=0):
    """pad: elements between the rows of x; shift: elements before its first."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    w, w64 = _weight(p, kind, n, k, m)
    cols = 2 * k if form == "silu" else k
    x = torch.randn((m * (cols + pad) + shift,), generator=g, device="cuda").to(torch.bfloat16)[shift:].view(m, cols + pad)[:, :cols]
    a = x.double()
    if form == "silu":      # bf16 roundings of the sigmoid, gate * sigmoid and the product
        gate, up = x[:, :k].float(), x[:, k:].float()
        sig = torch.sigmoid(gate).to(torch.bfloat16).float()
        a = ((gate * sig).to(torch.bfloat16).float() * up).to(torch.bfloat16).double()
    res = torch.randn((m, n), generator=g, device="cuda").to(torch.bfloat16) if form == "residual" else None
    assert x.data_ptr() % 16 == 2 * shift % 16 and (m == 1 or x.stride(0) == cols + pad)
    got = p.qwen3.linear(x, w, residual=res, silu_mul=form == "silu").double()
    v, mag = a @ w64.T, a.abs() @ w64.abs().T
    want = v + (res.double() if res is not None else 0)
    # results are rounded to bf16 (2^-8 in all for two roundings); sums of k f32 terms; above 32 rows the weights are bf16 (2^-9)
    tol = 2.0 ** -8 * (v.abs() + want.abs()) + mag * (k * 2.0 ** -24 + (2.0 ** -9 if m > 32 and kind != "bf16" else 0.0))
    if form == "silu":      # a sigmoid that lies on the edge of a bf16 step may round the other way: 2^-8 of one factor
        tol = tol + mag * 2.0 ** -7
    err = (got - want).abs()
    assert bool((err <= tol).all()), (kind, form, float((err - tol).max()))


@pytest.mark.parametrize("kind", ["int4", "int4_half", "int8", "int8_g64", "bf16"])
@pytest.mark.parametrize("n,k", [(1, 64), (31, 192), (130, 576), (257, 4160), (4100, 1088), (6144, 4096)])
def test_batched_edges(n, k, kind):
    p = pkg()
    for m in (9, 16, 17, 32, 33, 129, 513):
        _check(p, m, n, k, kind)


@pytest.mark.parametrize("kind", ["int4", "int4_half", "int8", "int8_g64", "bf16"])
@pytest.mark.parametrize("pad,shift", [(1, 0), (3, 0), (8, 0), (0, 1), (0, 8), (5, 3)])
def test_rows_that_allow_no_wide_loads(pad, shift, kind):
    """x whose rows or first element are not 16-byte aligned (or just are): staged element by element, or copied into aligned rows."""
    p = pkg()
    for m in (9, 17, 32, 33, 129):
        _check(p, m, 257, 1088, kind, pad=pad, shift=shift)
        _check(p, m, 130, 576, kind, form="residual", pad=pad, shift=shift)
    _check(p, 24, 130, 576, kind, form="silu", pad=pad, shift=shift)


@pytest.mark.parametrize("kind", ["int4", "int4_half", "int8", "int8_g64"])
@pytest.mark.parametrize("m,n,k", [(320, 4096, 4096), (640, 1031, 1024), (8200, 1026, 1088)])
def test_panels(m, n, k, kind):
    """Many rows: dequantised panels (of the other formats from thousands of rows on), or weights widened in the GEMM, as the times say."""
    p = pkg()
    _check(p, m, n, k, kind)
    if m < 1000:
        _check(p, m, n, k, kind, form="residual")


@pytest.mark.parametrize("kind", ["int4", "int8", "int8_g64"])
@pytest.mark.parametrize("m", [9, 24, 40])
def test_batched_forms(m, kind):
    p = pkg()
    _check(p, m, 1000, 2048, kind, form="residual")
    if m <= 32:
        _check(p, m, 520, 6144, kind, form="silu")


@pytest.mark.parametrize("kind", ["int4", "int4_half", "int8", "int8_g64", "bf16"])
def test_batched_without_scratch(kind):
    """Route 1: 9 to 32 rows on the kernel that needs no scratch."""
    p = pkg()
    p.lib().b200_qmm_force_route(p.default_context().handle, 1)
    try:
        for m, n, k in ((9, 31, 192), (16, 257, 1088), (17, 130, 576), (32, 4100, 4096), (32, 1000, 12288)):
            _check(p, m, n, k, kind)
            _check(p, m, n, k, kind, form="residual")
        _check(p, 24, 520, 6144, kind, form="silu")
    finally:
        p.lib().b200_qmm_force_route(p.default_context().handle, 0)


def test_batched_under_capture():
    """A captured call replays to the same bytes (the slices' scratch is an allocation of the graph)."""
    import torch
    p = pkg()
    w, _ = _weight(p, "int4", 4096, 4096, 1)
    x = torch.randn((24, 4096), device="cuda").to(torch.bfloat16)
    want = p.qwen3.linear(x, w)
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        p.qwen3.linear(x, w)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = p.qwen3.linear(x, w)
    for _ in range(3):
        got.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(got, want)


def _overlapped(p, weights, xs, rounds=6):
    """The products on one stream per weight, enqueued in turn without a wait between them."""
    import torch
    streams = [torch.cuda.Stream() for _ in weights]
    torch.cuda.synchronize()
    out = [[] for _ in weights]
    for _ in range(rounds):
        for i, s in enumerate(streams):
            with torch.cuda.stream(s):
                out[i].append(p.qwen3.linear(xs[i], weights[i]))
    torch.cuda.synchronize()
    return out


@pytest.mark.parametrize("m,pad", [(600, 0), (100, 1), (24, 0)])
def test_overlapping_streams(m, pad):
    """Calls of one context on several streams: each has scratch of its own (panels; panels for rows TMA cannot read; slices of K)."""
    import torch
    p = pkg()
    weights = [_weight(p, "int4", 2048, 4096, i)[0] for i in range(3)]
    xs = [torch.randn((m, 4096 + pad), device="cuda").to(torch.bfloat16)[:, :4096] for _ in weights]
    want = [p.qwen3.linear(x, w) for x, w in zip(xs, weights)]
    for i, got in enumerate(_overlapped(p, weights, xs)):
        assert all(torch.equal(g, want[i]) for g in got), i


def test_overlapping_threads():
    import threading
    import torch
    p = pkg()
    weights = [_weight(p, "int4", 2048, 4096, i)[0] for i in range(3)]
    xs = [torch.randn((m, 4096), device="cuda").to(torch.bfloat16) for m in (600, 700, 20)]
    want = [p.qwen3.linear(x, w) for x, w in zip(xs, weights)]
    torch.cuda.synchronize()
    got = [[] for _ in weights]

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(8):
                got[i].append(p.qwen3.linear(xs[i], weights[i]))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for i in range(3):
        assert len(got[i]) == 8 and all(torch.equal(g, want[i]) for g in got[i]), i


def test_captured_panels_outlive_larger_calls():
    """A graph captured without a warm-up call of its shape, replayed after calls that need larger panels."""
    import torch
    p = pkg()
    w, _ = _weight(p, "int4", 1024, 1024, 1)
    x = torch.randn((600, 1024), device="cuda").to(torch.bfloat16)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = p.qwen3.linear(x, w)
    big, _ = _weight(p, "int4", 8192, 4096, 2)
    xb = torch.randn((600, 4096), device="cuda").to(torch.bfloat16)
    want = p.qwen3.linear(x, w)
    p.qwen3.linear(xb, big)
    for _ in range(3):
        got.zero_()
        graph.replay()
        p.qwen3.linear(xb, big)
        torch.cuda.synchronize()
        assert torch.equal(got, want)
