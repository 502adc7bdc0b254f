"""Logits of a few positions (k_logits_few) and staged copies of pageable host arrays (gt_hostcopy.cu) at their edges."""
import numpy as np
import pytest

from glacier.tune_b200 import synth as S

pytestmark = pytest.mark.gpu


# one tile and a ragged last one, one and two token columns of MMAs and one token past them (the large kernel), contractions of
# 4 to 20 runs of 32 over 8 warps
@pytest.mark.parametrize("V,H,T", [(16, 128, 1), (1000, 640, 8), (1004, 256, 9), (516, 384, 16), (516, 384, 17), (40000, 512, 3)])
def test_few_logits(V, H, T):
    """fp16 weights and hidden rounded to fp16, fp32 sums: 2^-11 / sqrt(3) per rounded operand of zero-mean sums, 1e-3."""
    import torch
    from glacier.tune_b200 import capi as G
    rng = np.random.default_rng(V + T)
    eng = G.Engine(0, G.MATH_BF16)
    W = (rng.standard_normal((V, H)) * 0.05).astype(np.float16)
    x = rng.standard_normal((T, H)).astype(np.float32)
    w = eng.upload_weight(G.TYPE_F16, W, V, H)
    out = torch.full((T, V), 9.0, device="cuda")
    X = torch.from_numpy(x).cuda()
    torch.cuda.synchronize()
    eng.lm_head_logits(w, X, out)
    eng.sync()
    want = x.astype(np.float64) @ W.astype(np.float64).T
    assert np.linalg.norm(out.cpu().numpy() - want) / np.linalg.norm(want) < 1e-3
    w.free()


@pytest.mark.parametrize("T", [1, 70, 600, 5000])
def test_pageable_host_calls(T):
    """Host arrays below the staging size, above it, larger than the ring of page-locked pieces (8 MB), repeated so that slots are
    reused in both directions: the same bits as the call on device tensors.  (Few splits here: one CTA owns each output tile
    at 600 tokens and more, and the few-token kernel adds in a fixed order; in between atomics move the last bits.)"""
    import torch
    from glacier.tune_b200 import capi as G
    N, K = 4096, 1024
    rng = np.random.default_rng(T)
    eng = G.Engine(0, G.MATH_BF16)
    w = eng.upload_weight(S.TYPE_Q4_K, S.make_weight(S.TYPE_Q4_K, N, K, 3), N, K)
    x, dy = rng.standard_normal((T, K)).astype(np.float32), rng.standard_normal((T, N)).astype(np.float32)
    X, Y = torch.from_numpy(x).cuda(), torch.empty(T, N, device="cuda")
    dY, dX = torch.from_numpy(dy).cuda(), torch.empty(T, K, device="cuda")
    torch.cuda.synchronize()
    eng.forward(w, None, X, Y)
    eng.backward(w, None, dY, None, dX, flags=G.FLAG_DX_ASSIGN)
    eng.sync()
    for _ in range(3):
        y = eng.forward(w, None, x)
        dx = np.zeros((T, K), np.float32)
        eng.backward(w, None, dy, None, dx)
        assert np.allclose(y, Y.cpu().numpy(), rtol=0, atol=1e-5 * np.abs(y).max())
        assert np.allclose(dx, dX.cpu().numpy(), rtol=0, atol=1e-5 * np.abs(dx).max())
    w.free()
