"""Weights that the kernel just before the product writes: no product may fetch them earlier than that kernel's stores."""
import pytest

from util import pkg

pytestmark = pytest.mark.gpu


def _rounds(make, use, rounds=12):
    """make(i) writes weight i, use(w) multiplies by it at once; the same products once more after everything has finished."""
    import torch
    got, kept = [], []
    for i in range(rounds):
        w = make(i)
        got.append(use(w))
        kept.append({k: v.clone() for k, v in w.items()} if isinstance(w, dict) else w.clone())
    torch.cuda.synchronize()
    for i, w in enumerate(kept):
        torch.cuda.synchronize()
        assert torch.equal(got[i], use(w)), i


@pytest.mark.parametrize("m", [1, 4, 16, 32])
@pytest.mark.parametrize("in_place", [False, True])
def test_weights_written_by_a_gemm(m, in_place):
    """A bf16 weight that a dense product has just formed, as a fresh tensor or by an update in place (beta = 1)."""
    import torch
    p = pkg()
    n, k = 4096, 4096
    u, v = torch.randn((12, n, 256), device="cuda").to(torch.bfloat16), (torch.randn((256, k), device="cuda") / 16).to(torch.bfloat16)
    x = torch.randn((m, k), device="cuda").to(torch.bfloat16)
    w = torch.zeros((n, k), dtype=torch.bfloat16, device="cuda")

    def make(i):
        if not in_place:
            return p.blas.matmul(u[i], v)
        B = p.blas
        B.run_steel_gemm(B.GemmParams(n, k, 256, B.Operand(u[i], 256), B.Operand(v, k), B.Operand(w, k), 1, 1.0, 1.0))
        return w

    _rounds(make, lambda w: p.qwen3.linear(x, w))
    if m <= 8:
        _rounds(make, lambda w: p.blas.matmul(x, w, transpose_b=True))     # the few-row route


@pytest.mark.parametrize("m", [1, 8, 16])
@pytest.mark.parametrize("kind", ["int4", "int8"])
def test_weights_written_by_the_quantiser(m, kind):
    import torch
    p = pkg()
    w = torch.randn((12, 2048, 2048), device="cuda")
    x = torch.randn((m, 2048), device="cuda").to(torch.bfloat16)
    quantise = p.qwen3.quantize_int4 if kind == "int4" else p.qwen3.quantize_int8
    _rounds(lambda i: quantise(w[i]), lambda q: p.qwen3.linear(x, q))
