"""The fp32-accurate GEMM (gt_exact_gemm.cu) at the edges of its tiles, slabs and cluster splits, against fp64."""
import numpy as np
import pytest

from glacier.tune_b200 import synth as S

pytestmark = pytest.mark.gpu

F32, F16 = 0, 1
# (type, N, K, T, rank): one token and one past each token tile (32, 64, 128); features and contraction below one tile and
# one past it; contractions cut over clusters of 2, 4 and 8; rows of an odd number of half blocks; F32 / F16 rows whose
# length is no multiple of anything; ranks below, at and above one slab
CASES = [(8, 66, 64, 1, 8), (2, 130, 96, 33, 16), (8, 65, 4864, 129, 32), (2, 896, 1024, 200, 40), (8, 2, 32, 65, 64),
         (12, 9, 1152, 40, 16), (14, 64, 224, 31, 16), (12, 128, 512, 128, 16), (14, 200, 768, 257, 8), (F32, 67, 37, 66, 5), (F16, 33, 130, 3, 7)]


def _weight_bytes(qtype, N, K, rng):
    if qtype == F32:
        return rng.standard_normal((N, K)).astype(np.float32).view(np.uint8).reshape(-1)
    if qtype == F16:
        return rng.standard_normal((N, K)).astype(np.float16).view(np.uint8).reshape(-1)
    return S.make_weight(qtype, N, K, N + K)


@pytest.mark.parametrize("qtype,N,K,T,rank", CASES)
def test_exact_gemm_edges(qtype, N, K, T, rank):
    """fp32 mode.  Bound on the relative error: a slab's at most 12 truncated additions of 2^-23 of its partial sum, then
    fp32 additions over up to 153 slabs, 2^-24 each and of random sign: under 12 * 2^-23 / 2 + sqrt(153) * 2^-24 = 1.5e-6
    of the terms' norm; the sums of zero-mean terms keep about that norm, and the rank-r term goes through two such sums."""
    from glacier.tune_b200 import capi as G
    rng = np.random.default_rng(N * K + T)
    if qtype in (12, 14) and N * K % 256:
        N += -N % 8
    eng = G.Engine(0, G.MATH_FP32)
    bias = rng.standard_normal(N).astype(np.float32)
    w = eng.upload_weight(qtype, _weight_bytes(qtype, N, K, rng), N, K, bias)
    W = eng.dequant_rows(w, 0, N).astype(np.float64)
    A, B = rng.standard_normal((K, rank)).astype(np.float32), rng.standard_normal((rank, N)).astype(np.float32)
    x, dy = rng.standard_normal((T, K)).astype(np.float32), rng.standard_normal((T, N)).astype(np.float32)
    ad = eng.create_adapter(K, N, rank, 0.5 * rank)
    ad.upload(A, B)
    rel = lambda a, b: np.linalg.norm(a - b) / np.linalg.norm(b)      # noqa: E731
    x64, dy64, A64, B64 = (v.astype(np.float64) for v in (x, dy, A, B))
    y = eng.forward(w, ad, x)
    assert rel(y, x64 @ W.T + bias + 0.5 * (x64 @ A64) @ B64) < 4e-6
    assert rel(eng.forward(w, None, x), x64 @ W.T + bias) < 4e-6
    want = dy64 @ W + 0.5 * (dy64 @ B64.T) @ A64.T
    dx = np.full((T, K), 2.0, np.float32)
    eng.backward(w, ad, dy, x, dx)
    assert rel(dx.astype(np.float64) - 2.0, want) < 4e-6
    eng.backward(w, ad, dy, x, dx, flags=G.FLAG_DX_ASSIGN)
    assert rel(dx, want) < 4e-6
    again = dx.copy()
    eng.backward(w, None, dy, None, dx, flags=G.FLAG_DX_ASSIGN)
    assert rel(dx, dy64 @ W) < 4e-6 and not np.array_equal(again, dx)
    w.free()
    ad.free()
