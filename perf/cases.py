"""Timed cases over the framework's public entry points: what they stand for, their inputs, one pass, its work.

Kinds of case, each with the ranges that `draw` spreads over:

* ``layer``  - the seven projections of one decoder layer on device tensors, the way a transformer block calls them
  (q | k | v as a group, o, the FFN call), LoRA on all of them; forward only (decode, scoring) or forward and backward
  (training).  1 to 2048 tokens, hidden 512 to 3584, FFN up to 18944, all Q4_K or the Q4_K_M mix (v, down in Q6_K).
* ``proj``   - one LoRA-adapted projection on device tensors, forward and backward.  Q4_K and Q6_K, rows of whole
  super-blocks or of half a super-block more, Q4_0 and Q8_0; 1 to 1024 tokens, any even number of output features.
* ``host``   - one projection, forward and backward, called on host arrays: the drop-in use from a host that keeps its
  activations in its own memory.  1 to 512 tokens.
* ``logits`` - logits of a few positions over the fp16 LM head (sampling).  1 to 16 positions, vocabulary 1000 to 152064.
* ``eval``   - loss of one sequence without gradients, token ids in host memory (the trainer's validation loss).
* ``train``  - one optimizer step of a model of up to four blocks: forward, loss, backward, clip, AdamW.
* ``micro``  - forward, loss and backward of a deeper model, the gradients accumulating (one micro-batch of a step).

`eval`, `train` and `micro` run 16 to 2048 tokens, hidden 512 to 3584, vocabulary 1000 to 152064, with and without
activation checkpointing; adapter ranks are 8 to 32 everywhere.
"""
from __future__ import annotations

import numpy as np
import torch

from glacier.tune_b200 import capi as G
from glacier.tune_b200 import synth as S

TYPES = {"q4_k": G.TYPE_Q4_K, "q6_k": G.TYPE_Q6_K, "q4_0": G.TYPE_Q4_0, "q8_0": G.TYPE_Q8_0, "f16": G.TYPE_F16}
BITS = {"q4_k": 4.5, "q6_k": 6.5625, "q4_0": 4.5, "q8_0": 8.5, "f16": 16}
ALPHA = 32.0
NAMES = ("q", "k", "v", "o", "gate", "up", "down")
HYPER = dict(lr=2e-4, beta1=0.9, beta2=0.999, eps=1e-8, weight_decay=0.01)
STD = 0.02      # of base weights, LM head and B: what trained checkpoints of these shapes have


def _layer(name, tokens, mix, backward, hidden=3584, kv=512, ffn=18944, rank=16):
    return dict(name=name, kind="layer", tokens=tokens, hidden=hidden, kv=kv, ffn=ffn, mix=mix, rank=rank, backward=backward)


def _model(name, kind, layers, hidden, heads, kv_heads, ffn, vocab, tokens, checkpoint, rank=16):
    return dict(name=name, kind=kind, layers=layers, hidden=hidden, heads=heads, kv_heads=kv_heads, ffn=ffn, vocab=vocab,
                tokens=tokens, checkpoint=checkpoint, rank=rank)


def listed():
    return [
        # decoding one token through a 7B-shaped layer of a Q4_K_M file: weight streaming, launches
        _layer("layer_decode_1", 1, True, False),
        # a short training sequence, ragged, on the same layer
        _layer("layer_train_131", 131, True, True),
        # the benchmark's workload: the layer in Q4_K at 512 tokens
        _layer("layer_train_512", 512, False, True),
        # a long sequence
        _layer("layer_train_2048", 2048, True, True),
        # the FFN projection of a half-billion-parameter model: rows of three and a half super-blocks
        dict(name="proj_q4k_half_block", kind="proj", type="q4_k", n=4864, k=896, tokens=512, rank=16),
        # the same model kept in Q8_0
        dict(name="proj_q8_0", kind="proj", type="q8_0", n=896, k=4864, tokens=200, rank=16),
        # a host that hands over its own arrays, call by call
        dict(name="host_proj_512", kind="host", type="q4_k", n=3584, k=3584, tokens=512, rank=16),
        # the next token's logits
        dict(name="logits_1", kind="logits", vocab=152064, hidden=3584, tokens=1),
        # validation loss on a ragged sequence of a small model: many short launches
        _model("eval_777", "eval", 8, 1024, 8, 2, 2816, 32000, 777, True),
        # training a small model on a short sequence, every block's state kept: launch latency
        _model("train_small_200", "train", 4, 1024, 8, 2, 2816, 32000, 200, False),
        # training on a long ragged sequence: attention counts
        _model("train_long_1999", "train", 2, 2048, 16, 4, 5632, 32000, 1999, True),
        # the full training workload: 28 blocks, one 512-token sequence, activation checkpointing
        _model("micro_7b_512", "micro", 28, 3584, 28, 4, 18944, 152064, 512, True),
    ]


def _log_int(rng, lo, hi, step=1):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random() / step)) * step))


def _draw_dims(rng, hi=3584):
    hidden = _log_int(rng, 512, hi, 256)
    heads = hidden // 128
    kv_heads = rng.choice([g for g in range(1, heads + 1) if heads % g == 0 and heads // g >= 2 and g <= 8])
    ffn = min(18944, max(512, int(hidden * rng.uniform(2.0, 5.3)) // 256 * 256))
    return hidden, heads, kv_heads, ffn


def draw(rng):
    kind = rng.choice(["layer", "layer", "layer", "proj", "proj", "host", "logits", "eval", "train", "train", "micro"])
    rank = rng.choice([8, 16, 16, 32])
    if kind == "layer":
        backward = rng.random() < 0.75
        tokens = _log_int(rng, 16, 2048) if backward else _log_int(rng, 1, 512)
        if rng.random() < 0.5:
            return dict(kind=kind, tokens=tokens, hidden=3584, kv=512, ffn=18944, mix=rng.random() < 0.5, rank=rank, backward=backward)
        hidden, _, kv_heads, ffn = _draw_dims(rng)
        return dict(kind=kind, tokens=tokens, hidden=hidden, kv=128 * kv_heads, ffn=ffn, mix=rng.random() < 0.5, rank=rank, backward=backward)
    if kind == "proj":
        t = rng.choice(["q4_k", "q6_k", "q4_0", "q8_0"])
        k = _log_int(rng, 256, 4992, 128 if t in ("q4_k", "q6_k") else 32)
        n = _log_int(rng, 128, 4864, 2)
        return dict(kind=kind, type=t, n=n, k=k, tokens=_log_int(rng, 1, 1024), rank=rank)
    if kind == "host":
        return dict(kind=kind, type=rng.choice(["q4_k", "q6_k"]), n=_log_int(rng, 256, 4864, 2), k=_log_int(rng, 512, 4864, 256),
                    tokens=_log_int(rng, 1, 512), rank=rank)
    if kind == "logits":
        return dict(kind=kind, vocab=_log_int(rng, 1000, 152064), hidden=_log_int(rng, 512, 3584, 128), tokens=_log_int(rng, 1, 16))
    hidden, heads, kv_heads, ffn = _draw_dims(rng, 2560)
    layers = {"eval": rng.randint(2, 8), "train": rng.randint(1, 4), "micro": rng.randint(5, 8)}[kind]
    return dict(kind=kind, layers=layers, hidden=hidden, heads=heads, kv_heads=kv_heads, ffn=ffn, vocab=_log_int(rng, 1000, 64000),
                tokens=_log_int(rng, 16, 2048), checkpoint=rng.random() < 0.5, rank=rank)


# ---- inputs ----------------------------------------------------------------------------------------------------------
_engine = None


def _eng():
    """The program's one engine, on the stream that torch's own operations use as well."""
    global _engine
    if _engine is None:
        stream = torch.cuda.Stream()
        torch.cuda.set_stream(stream)
        _engine = G.Engine(0, G.MATH_BF16, stream=stream.cuda_stream)
    return _engine


class _Pools:
    """Random contents of one state, drawn once from its seed; tensors take stretches of them at offsets of their own."""

    BLOCKS = 16381      # a prime: rows of a large tensor do not repeat in step with its row length

    def __init__(self, seed):
        self.rng = np.random.default_rng(seed)
        self.blocks, self.floats, self.long = {}, None, {}

    def _block_pool(self, t, std):
        rng, n = self.rng, self.BLOCKS
        spread = rng.uniform(0.5, 1.5, n)
        if t == "q4_k":      # w = d * sc * (q - 7.5): zero mean, as trained weights have
            b = S.make_q4k_blocks(n, rng)
            sc = rng.integers(8, 64, (n, 8), dtype=np.uint8)
            b[:, 4:16] = S.pack_scales_q4k(sc, sc)
            d = (spread * std / (4.61 * 38)).astype(np.float16)
            b[:, 0:2] = d.view(np.uint8).reshape(n, 2)
            b[:, 2:4] = (7.5 * d.astype(np.float32)).astype(np.float16).view(np.uint8).reshape(n, 2)
            return b
        make, unit, at = {"q6_k": (S.make_q6k_blocks, 18.5 * 18.5, 208), "q4_0": (S.make_q40_blocks, 4.61, 0),
                          "q8_0": (S.make_q80_blocks, 73.3, 0)}[t]
        b = make(n, rng)
        b[:, at:at + 2] = (spread * std / unit).astype(np.float16).view(np.uint8).reshape(n, 2)
        return b

    def weight(self, t, n, k, std=STD):
        """The bytes of an [n, k] tensor."""
        key = t, std
        if key not in self.blocks:
            if t == "f16":
                self.blocks[key] = (self.rng.standard_normal((1 << 21) + 7, np.float32) * np.float32(std)).astype(np.float16)
            else:
                self.blocks[key] = self._block_pool(t, std)
        pool = self.blocks[key]
        if t == "f16":
            unit, count = 1, n * k
        else:
            unit = pool.shape[1]
            count = n * k // (256 if t in ("q4_k", "q6_k") else 32)
        flat = self.long.get(key)
        if flat is None or flat.shape[0] < (count + len(pool)) * unit:
            flat = self.long[key] = np.resize(pool.reshape(-1), (count + len(pool)) * unit)
        at = int(self.rng.integers(0, len(pool))) * unit
        return flat[at:at + count * unit]

    def normal(self, shape, std=1.0):
        n = int(np.prod(shape))
        if self.floats is None or len(self.floats) < n + 4099:
            self.floats = np.resize(self.rng.standard_normal(262147, np.float32) if self.floats is None else self.floats[:262147], 2 * n + 262147)
        at = int(self.rng.integers(0, len(self.floats) - n))
        return np.ascontiguousarray((self.floats[at:at + n] * np.float32(std)).reshape(shape))


class _Handles:
    """The library's handles of one state, given back when neither the state nor a view of their memory is left."""

    def __init__(self):
        self.items, self.model = [], None

    def __del__(self):
        try:
            if self.model is not None:
                self.model.close()
            for h in self.items:
                h.free()
        except Exception:      # the interpreter is going down
            pass


class _State:
    """What a program keeps between passes."""

    def __init__(self, case, seed):
        self.case, self.eng, self.pools, self.handles = case, _eng(), _Pools(seed), _Handles()
        self.gen = torch.Generator(device="cuda")
        self.gen.manual_seed(seed)

    def weight(self, t, n, k, bias=None, std=STD):
        w = self.eng.upload_weight(TYPES[t], self.pools.weight(t, n, k, std), n, k, bias)
        self.handles.items.append(w)
        return w

    def adapter(self, k, n):
        r = self.case["rank"]
        ad = self.eng.create_adapter(k, n, r, ALPHA)
        ad.upload(self.pools.normal((k, r), k ** -0.5), self.pools.normal((r, n), STD))
        self.handles.items.append(ad)
        return ad

    def randn(self, *shape):
        return torch.randn(shape, generator=self.gen, device="cuda")

    def bind(self, adapters):
        """One flat gradient buffer for all adapters; also A's and B's gradients as views of it."""
        flat = torch.zeros(sum(a.rank * (a.K + a.N) for a in adapters), device="cuda")
        at = 0
        for a in adapters:
            cut = at + a.K * a.rank
            end = cut + a.rank * a.N
            a.bind_grads(flat[at:cut], flat[cut:end])
            at = end
        return flat


class _DeviceArray:
    """Device memory that the library owns, for torch.as_tensor."""

    def __init__(self, address, shape, owner):
        self.owner = owner
        self.__cuda_array_interface__ = dict(data=(address, False), shape=shape, typestr="<f4", version=3)


def _view(address, shape, owner):
    return torch.as_tensor(_DeviceArray(address, shape, owner), device="cuda")


def _shapes(hidden, kv, ffn):
    return dict(q=(hidden, hidden), k=(kv, hidden), v=(kv, hidden), o=(hidden, hidden), gate=(ffn, hidden), up=(ffn, hidden), down=(hidden, ffn))


def _type_of(name, mix):
    return "q6_k" if mix and name in ("v", "down") else "q4_k"


def _prepare_layer(s):
    c, T = s.case, s.case["tokens"]
    shapes = _shapes(c["hidden"], c["kv"], c["ffn"])
    s.w = {n: s.weight(_type_of(n, c["mix"]), *shapes[n]) for n in NAMES}
    s.ad = {n: s.adapter(shapes[n][1], shapes[n][0]) for n in NAMES}
    bf = lambda t: t.to(torch.bfloat16).to(torch.float32)      # noqa: E731 - activations as a bf16 model has them
    s.x_attn, s.x_o, s.x_ffn = (bf(s.randn(T, c["hidden"])) for _ in range(3))
    s.y = {n: torch.empty(T, shapes[n][0], device="cuda") for n in NAMES}
    s.h = torch.empty(T, c["ffn"], device="cuda")
    if c["backward"]:
        s.flat = s.bind([s.ad[n] for n in NAMES])
        s.dy = {n: s.randn(T, shapes[n][0]) for n in ("q", "k", "v", "o", "down")}
        s.dx_attn, s.dx_o, s.dx_ffn = (torch.empty(T, c["hidden"], device="cuda") for _ in range(3))


def _run_layer(s):
    e, w, ad, y = s.eng, s.w, s.ad, s.y
    qkv, ffn = ("q", "k", "v"), ("gate", "up", "down")
    e.forward_group([w[n] for n in qkv], [ad[n] for n in qkv], s.x_attn, [y[n] for n in qkv])
    e.forward(w["o"], ad["o"], s.x_o, y["o"])
    fad = [ad[n] for n in ffn]
    if not s.case["backward"]:
        e.ffn_forward(w["gate"], w["up"], w["down"], fad, s.x_ffn, y["down"])
        return [y[n] for n in ("q", "k", "v", "o", "down")]
    e.ffn_forward(w["gate"], w["up"], w["down"], fad, s.x_ffn, y["down"], y["gate"], y["up"], s.h)
    s.flat.zero_()
    flags = G.FLAG_REUSE_LOW | G.FLAG_DX_ASSIGN
    e.ffn_backward(w["gate"], w["up"], w["down"], fad, s.dy["down"], s.x_ffn, y["gate"], y["up"], s.h, s.dx_ffn, flags=flags)
    e.backward(w["o"], ad["o"], s.dy["o"], s.x_o, s.dx_o, flags=flags)
    e.backward_group([w[n] for n in qkv], [ad[n] for n in qkv], [s.dy[n] for n in qkv], s.x_attn, s.dx_attn, flags=flags)
    return [y[n] for n in NAMES] + [s.h, s.dx_ffn, s.dx_o, s.dx_attn, s.flat]


def _prepare_proj(s):
    c, T = s.case, s.case["tokens"]
    s.w, s.ad = s.weight(c["type"], c["n"], c["k"]), s.adapter(c["k"], c["n"])
    s.flat = s.bind([s.ad])
    if c["kind"] == "host":
        s.x, s.dy = s.pools.normal((T, c["k"])), s.pools.normal((T, c["n"]))
        s.y, s.dx = np.empty((T, c["n"]), np.float32), np.empty((T, c["k"]), np.float32)
    else:
        s.x, s.dy = s.randn(T, c["k"]), s.randn(T, c["n"])
        s.y, s.dx = torch.empty(T, c["n"], device="cuda"), torch.empty(T, c["k"], device="cuda")


def _run_proj(s):
    s.flat.zero_()
    s.eng.forward(s.w, s.ad, s.x, s.y)
    s.eng.backward(s.w, s.ad, s.dy, s.x, s.dx, flags=G.FLAG_REUSE_LOW | G.FLAG_DX_ASSIGN)
    return [s.y, s.dx, s.flat]


def _prepare_logits(s):
    c = s.case
    s.w = s.weight("f16", c["vocab"], c["hidden"])
    s.x = s.randn(c["tokens"], c["hidden"])
    s.y = torch.empty(c["tokens"], c["vocab"], device="cuda")


def _run_logits(s):
    return [s.eng.lm_head_logits(s.w, s.x, s.y)]


def _prepare_model(s):
    c, p = s.case, s.pools
    s.model = s.handles.model = m = G.Model(s.eng, c["layers"], c["hidden"], c["heads"], c["kv_heads"], 128, c["ffn"], c["vocab"], c["tokens"],
                          checkpoint=c["checkpoint"])
    shapes = _shapes(c["hidden"], 128 * c["kv_heads"], c["ffn"])
    adapters = []
    # a residual stream of order one that every block adds a fraction to
    add = STD * (8 * c["layers"]) ** -0.5
    for l in range(c["layers"]):
        ws = [s.weight(_type_of(n, True), *shapes[n], p.normal((shapes[n][0],), STD) if n in ("q", "k", "v") else None,
                       add if n in ("o", "down") else STD) for n in NAMES]
        ads = [s.adapter(shapes[n][1], shapes[n][0]) for n in NAMES]
        m.set_block(l, ws, ads, 1 + p.normal((c["hidden"],), 0.05), 1 + p.normal((c["hidden"],), 0.05))
        adapters += ads
    m.set_head(s.weight("f16", c["vocab"], c["hidden"], std=1.0), 1 + p.normal((c["hidden"],), 0.05), s.weight("f16", c["vocab"], c["hidden"]))
    s.tokens = p.rng.integers(0, c["vocab"], c["tokens"]).astype(np.int32)
    s.labels = np.roll(s.tokens, -1).astype(np.int32)
    s.labels[-1] = -100
    if c["kind"] == "eval":
        return
    s.tokens, s.labels = torch.from_numpy(s.tokens).cuda(), torch.from_numpy(s.labels).cuda()
    s.loss = torch.zeros(1, device="cuda")
    s.step = 0
    address, n = m.bind_grads()
    if c["kind"] == "micro":
        s.out = [s.loss, _view(address, (n,), s.handles)]
    else:
        s.out = [s.loss]
        for a in adapters:
            pa, pb, _, _ = a.device_ptrs()
            s.out += [_view(pa, (a.K, a.rank), s.handles), _view(pb, (a.rank, a.N), s.handles)]


def _run_eval(s):
    return list(s.model.loss(s.tokens, s.labels))


def _run_train(s):
    s.model.forward_backward(s.tokens, s.labels, loss_dev=s.loss)
    if s.case["kind"] == "train":
        s.step += 1
        s.model.optimizer_step(max_norm=1.0, step=s.step, **HYPER)
    return s.out


_KINDS = dict(layer=(_prepare_layer, _run_layer), proj=(_prepare_proj, _run_proj), host=(_prepare_proj, _run_proj),
              logits=(_prepare_logits, _run_logits), eval=(_prepare_model, _run_eval), train=(_prepare_model, _run_train),
              micro=(_prepare_model, _run_train))


def prepare(case, seed):
    s = _State(case, seed)
    _KINDS[case["kind"]][0](s)
    s.pools = None
    return s


def run(state):
    return _KINDS[state.case["kind"]][1](state)


# ---- work ------------------------------------------------------------------------------------------------------------
def _proj_work(t, n, k, T, rank, backward):
    """Weights once; X in, Y out; backward: dY in, dX out, A, B in, dA, dB out."""
    adapter = rank * (n + k)
    nbytes = n * k * BITS[t] / 8 + 4 * (T * (n + k) * (2 if backward else 1) + adapter * (2 if backward else 1))
    flops = 2 * T * n * k * (2 if backward else 1) + 2 * T * adapter * (3 if backward else 1)
    return nbytes, flops


def work(case):
    c, T = case, case["tokens"]
    if c["kind"] in ("proj", "host"):
        b, f = _proj_work(c["type"], c["n"], c["k"], T, c["rank"], True)
        return dict(bytes=b, flops=f)
    if c["kind"] == "logits":
        return dict(bytes=2 * c["vocab"] * c["hidden"] + 4 * T * (c["vocab"] + c["hidden"]), flops=2 * T * c["vocab"] * c["hidden"])
    if c["kind"] == "layer":
        b = f = 0
        for n, (rows, cols) in _shapes(c["hidden"], c["kv"], c["ffn"]).items():
            pb, pf = _proj_work(_type_of(n, c["mix"]), rows, cols, T, c["rank"], c["backward"])
            b, f = b + pb, f + pf
        return dict(bytes=b, flops=f)
    # a model: weights and adapters once (and their gradients, moments), the LM head once, the block inputs; attention is causal
    training = c["kind"] != "eval"
    b, f = 2 * c["vocab"] * c["hidden"] + 2 * T * c["hidden"], (6 if training else 2) / (1 if not training else 1.5) * T * c["vocab"] * c["hidden"]
    passes = (1 if not training else 2)
    for n, (rows, cols) in _shapes(c["hidden"], 128 * c["kv_heads"], c["ffn"]).items():
        adapter = c["rank"] * (rows + cols)
        b += c["layers"] * (rows * cols * BITS[_type_of(n, True)] / 8 + 4 * adapter * (2 if training else 1))
        if c["kind"] == "train":
            b += c["layers"] * 4 * adapter * 5
        f += c["layers"] * (2 * T * rows * cols * passes + 2 * T * adapter * (3 if training else 1))
    f += c["layers"] * 2 * T * T * c["heads"] * 128 * (3.5 if training else 1)
    b += 4 * c["layers"] * T * c["hidden"] * (2 if training else 1)
    return dict(bytes=b, flops=f)


def tolerance(case):
    """bf16 operands with fp32 sums; a whole model compounds the roundings of its blocks."""
    if case["kind"] == "logits":
        return dict(rel=1e-3)
    if case["kind"] == "eval":
        return dict(rel=1e-3)
    if case["kind"] in ("train", "micro"):
        return dict(rel=2e-2, max=0.5)
    return dict(rel=1e-2)
