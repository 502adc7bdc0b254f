"""The tensor-core GEMM's token chunks: one CTA alone up to 256 tokens, CTA pairs above, several chunks with a ragged last one, and
adapter ranks whose rank-update stage takes its sixteen warps one step (16), several (64), or rows that are no multiple of 16 bytes."""
import numpy as np
import pytest

from glacier.tune_b200 import synth as S

pytestmark = pytest.mark.gpu

Q4, Q6 = S.TYPE_Q4_K, S.TYPE_Q6_K


@pytest.mark.parametrize("qt,N,K,T,rank", [(Q4, 1024, 1024, 256, 16), (Q6, 640, 1024, 257, 64), (Q4, 512, 512, 193, 5), (Q4, 2816, 1024, 609, 36),
                                           (Q6, 1152, 2048, 777, 16), (Q4, 1024, 2816, 129, 64)])
def test_token_chunks(qt, N, K, T, rank):
    """Gate of the bf16 mode (2e-2: operands of 8 significant bits, random signs) against fp64 on the dequantized weights."""
    from glacier.tune_b200 import capi as G
    c = S.make_projection_case(qt, N, K, T, seed=N + K + T, rank=rank, with_bias=True)
    eng = G.Engine(0, 0)
    w = eng.upload_weight(qt, c["w"], N, K, c["bias"])
    W = eng.dequant_rows(w, 0, N).astype(np.float64)
    ad = eng.create_adapter(K, N, rank, c["alpha"])
    ad.upload(c["a"], c["b"])
    x, dy, A, B = (c[k].astype(np.float64) for k in ("x", "dy", "a", "b"))
    rel = lambda a, b: np.linalg.norm(a - b) / np.linalg.norm(b)      # noqa: E731
    # the last rows too: they are in the ragged chunk
    got, want = eng.forward(w, ad, c["x"]), x @ W.T + c["bias"] + c["scaling"] * (x @ A) @ B
    assert rel(got, want) < 2e-2 and rel(got[-33:], want[-33:]) < 2e-2
    dx = np.full((T, K), 3.0, np.float32)
    eng.backward(w, ad, c["dy"], c["x"], dx, flags=G.FLAG_DX_ASSIGN)
    want = dy @ W + c["scaling"] * (dy @ B.T) @ A.T
    assert rel(dx, want) < 2e-2 and rel(dx[-33:], want[-33:]) < 2e-2
    w.free()
    ad.free()
