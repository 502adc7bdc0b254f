"""The few-token group launch (gt_decode.cu) at its edges: Q4_K and Q6_K members in one launch, one token and several, a last
row tile that is partly out of range, one super-block per row (half an item), rows cut over clusters, the dual gate | up form."""
import numpy as np
import pytest

from glacier.tune_b200 import synth as S

pytestmark = pytest.mark.gpu

Q4, Q6 = S.TYPE_Q4_K, S.TYPE_Q6_K
# (types, rows, K, T, rank): ranks 16 and 8 take the cluster kernel for X*A, 24 the general pass
CASES = [((Q4,), (16,), 256, 1, 16), ((Q6,), (40,), 256, 8, 8), ((Q4, Q4, Q6), (200, 24, 33), 768, 3, 16), ((Q6, Q4), (300, 17), 1280, 1, 24),
         ((Q6,), (48,), 18944, 2, 16), ((Q4,), (2500,), 4864, 8, 16), ((Q4, Q6, Q4), (64, 64, 64), 3584, 5, 32)]


@pytest.fixture(scope="module")
def eng():
    from glacier.tune_b200 import capi as G
    return G.Engine(0, G.MATH_BF16)


def _x(T, K, rng):
    return S.bf16_round(rng.standard_normal((T, K)).astype(np.float32))


@pytest.mark.parametrize("types,rows,K,T,rank", CASES)
def test_decode_group_edges(eng, types, rows, K, T, rank):
    """bf16-representable X, exact weights, fp32 rank-r terms: what is left is fp32 summation.  The MMAs sum 128 + q (150 at
    most, 190 for Q6_K) where the result keeps q - 7.5 (q - 32) of it: a factor of about 20 on 2^-24, and the products of
    a sub-block are exact - 1e-5 covers it.  The rank-24 case rounds X*A's operands to bf16
    and a mixed group the constants of its Q4_K members: 2e-2, the bf16 mode's gate."""
    import torch
    from glacier.tune_b200 import capi as G
    rng = np.random.default_rng(K + T)
    x = _x(T, K, rng)
    ws, ads, want = [], [], []
    for qt, N in zip(types, rows):
        bias = rng.standard_normal(N).astype(np.float32)
        w = eng.upload_weight(qt, S.make_weight(qt, N, K, N + K), N, K, bias)
        ad = eng.create_adapter(K, N, rank, 32.0)
        A, B = rng.standard_normal((K, rank)).astype(np.float32), rng.standard_normal((rank, N)).astype(np.float32) * np.float32(0.02)
        ad.upload(A, B)
        W = eng.dequant_rows(w, 0, N).astype(np.float64)
        want.append(x.astype(np.float64) @ W.T + bias + 32.0 / rank * (x.astype(np.float64) @ A) @ B)
        ws.append(w)
        ads.append(ad)
    X = torch.from_numpy(x).cuda()
    Ys = [torch.full((T, N), 3.0, device="cuda") for N in rows]
    torch.cuda.synchronize()
    for _ in range(2):      # (the second call overwrites the first one's outputs)
        eng.forward_group(ws, ads, X, Ys)
    eng.sync()
    for Y, ref in zip(Ys, want):
        err = np.linalg.norm(Y.cpu().numpy() - ref) / np.linalg.norm(ref)
        assert err < (2e-2 if rank == 24 or len(set(types)) > 1 else 1e-5), err
    for h in ws + ads:
        h.free()


@pytest.mark.parametrize("qt,F,H,T", [(Q4, 520, 512, 1), (Q6, 256, 256, 4), (Q4, 1024, 768, 8)])
def test_decode_ffn(eng, qt, F, H, T):
    """gate | up with the product formed in the launch, with and without gate and up as outputs.  SiLU's slope is at most 1.1,
    its argument and the other factor carry the 1e-5 of the projections."""
    import torch
    F -= F % 256
    rng = np.random.default_rng(F + T)
    x = _x(T, H, rng)
    ws = [eng.upload_weight(qt, S.make_weight(qt, n, k, n + k + i), n, k) for i, (n, k) in enumerate([(F, H), (F, H), (H, F)])]
    Wg, Wu, Wd = (eng.dequant_rows(w, 0, w.N).astype(np.float64) for w in ws)
    scale = np.float32(2.0 ** -6)      # SiLU arguments of order one
    xs = S.bf16_round(x * scale)
    g, u = xs.astype(np.float64) @ Wg.T, xs.astype(np.float64) @ Wu.T
    h = g / (1 + np.exp(-g)) * u
    X = torch.from_numpy(xs).cuda()
    out, G_, U_, H_ = torch.empty(T, H, device="cuda"), torch.empty(T, F, device="cuda"), torch.empty(T, F, device="cuda"), torch.empty(T, F, device="cuda")
    out2 = torch.empty_like(out)
    torch.cuda.synchronize()
    eng.ffn_forward(*ws, None, X, out, G_, U_, H_)
    eng.ffn_forward(*ws, None, X, out2)
    eng.sync()
    rel = lambda a, b: np.linalg.norm(a.cpu().numpy() - b) / np.linalg.norm(b)      # noqa: E731
    assert rel(G_, g) < 1e-5 and rel(U_, u) < 1e-5 and rel(H_, h) < 3e-5
    assert rel(out, h @ Wd.T) < 1e-2 and torch.equal(out, out2)
    for w in ws:
        w.free()
