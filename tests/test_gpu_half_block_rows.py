"""K-quant rows of an odd number of half super-blocks (in_features % 256 == 128) on the tensor-core kernel: two weight rows share
a row of the tensor maps.  One half-block per row, row counts below and past a 128-row tile and a 64-row contraction unit, the
single-CTA and the CTA-pair kernels, split contractions, a padding tile in the backward pair (odd tile counts)."""
import numpy as np
import pytest

from glacier.tune_b200 import synth as S

pytestmark = pytest.mark.gpu

Q4, Q6 = S.TYPE_Q4_K, S.TYPE_Q6_K


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("qt,N,K,T,rank", [(Q4, 2, 128, 1, 8), (Q6, 130, 128, 40, 16), (Q4, 62, 384, 130, 16), (Q6, 258, 896, 33, 32), (Q4, 1000, 1152, 300, 16),
                                           (Q6, 514, 640, 600, 24), (Q4, 4864, 896, 513, 16)])
def test_half_block_rows(qt, N, K, T, rank, mode):
    """Gates of the 16-bit modes (2e-2 with bf16 operands, 1e-3 with fp16) against fp64 on the dequantized weights."""
    from glacier.tune_b200 import capi as G
    c = S.make_projection_case(qt, N, K, T, seed=N + K + T, rank=rank, with_bias=True)
    eng = G.Engine(0, mode)
    w = eng.upload_weight(qt, c["w"], N, K, c["bias"])
    W = eng.dequant_rows(w, 0, N).astype(np.float64)
    ad = eng.create_adapter(K, N, rank, c["alpha"])
    ad.upload(c["a"], c["b"])
    x, dy, A, B = (c[k].astype(np.float64) for k in ("x", "dy", "a", "b"))
    tol = 2e-2 if mode == 0 else 1e-3
    rel = lambda a, b: np.linalg.norm(a - b) / np.linalg.norm(b)      # noqa: E731
    assert rel(eng.forward(w, ad, c["x"]), x @ W.T + c["bias"] + c["scaling"] * (x @ A) @ B) < tol
    want = dy @ W + c["scaling"] * (dy @ B.T) @ A.T
    dx = np.full((T, K), 3.0, np.float32)
    eng.backward(w, ad, c["dy"], c["x"], dx)
    assert rel(dx - 3.0, want) < tol
    eng.backward(w, None, c["dy"], None, dx, flags=G.FLAG_DX_ASSIGN)
    assert rel(dx, dy @ W) < tol
    w.free()
    ad.free()
