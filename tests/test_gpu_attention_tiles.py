"""Attention at the edges of its tiles and of its two work splits (query tiles of 64 with two key groups, of 128 with one; one and
two groups in the backward), through the calls on fp32 tensors, against torch in fp64."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,HQ,HK", [(63, 2, 1), (65, 3, 3), (128, 2, 2), (129, 4, 1), (193, 8, 2), (1025, 18, 2), (640, 32, 4)])
def test_attention_tiles(T, HQ, HK):
    """bf16 operands (P and dS rounded too): 1e-2 of the result's norm.  A score of norm up to 5 from operands rounded to 2^-9 each
    is off by at most 5 * 2^-8 = 2e-2, and so is the log-sum-exp."""
    import torch
    from glacier.tune_b200 import capi as G
    eng = G.Engine(0, G.MATH_BF16)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(T + HQ)
    rand = lambda h: torch.randn((T, h, 128), generator=gen, device="cuda")      # noqa: E731
    q, do, k, v = rand(HQ), rand(HQ), rand(HK), rand(HK)
    out, dq, dk, dv = torch.empty_like(q), torch.empty_like(q), torch.empty_like(k), torch.empty_like(v)
    lse = torch.empty(HQ, T, device="cuda")
    torch.cuda.synchronize()
    eng.attention_forward(q, k, v, out, lse, T, HQ, HK)
    eng.attention_backward(do, q, k, v, out, lse, dq, dk, dv, T, HQ, HK)
    eng.sync()
    a, b, c = (t.double().requires_grad_(True) for t in (q, k, v))
    g = HQ // HK
    s = torch.einsum("thd,shd->hts", a, b.repeat_interleave(g, 1)) / 128 ** 0.5
    s = s.masked_fill(torch.ones(T, T, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    y = torch.einsum("hts,shd->thd", s.softmax(-1), c.repeat_interleave(g, 1))
    y.backward(do.double())
    for got, want in ((out, y.detach()), (dq, a.grad), (dk, b.grad), (dv, c.grad)):
        assert ((got.double() - want).norm() / want.norm()).item() < 1e-2
    assert (lse.double() * 0.6931471805599453 - s.detach().logsumexp(-1)).abs().max().item() < 2e-2
