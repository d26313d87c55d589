"""The work that users of this package have it do, as cases that a timing program runs.

A case is a dict of plain values; its ``kind`` says which path it takes:

``linear``    QuantizedLinear.forward: the INT4 module that replaces nn.Linear, from one activation row to the
              rows of a prompt.
``mlp``       fused_swiglu_mlp: gate, up and down of one layer in one call.
``generate``  a chat turn of one user: INT4 decoder, greedy tokens produced on the device, the last logits read.
``batch``     a server's step: one token for each of several sequences of unequal length, logits left on the
              device for its sampler.
``prompt``    a new message behind a conversation that is in the cache already: INT4 decoder, logits of its last token.
``dabevik_decode``, ``dabevik_prompt``, ``sukalorn_decode``, ``sukalorn_prompt``
              the same two directions of the bfloat16 decoders described layer by layer.

Sizes are those of the benchmark: the Llama-3-8B widths with eight layers, and the Qwen2.5-0.5B model.  Weights
are normal numbers, quantized here for the INT4 paths, the caches normal numbers as well.
"""
import math

import numpy as np
import torch

import torchburn_b200 as tb

SIZES = {
    "8b": dict(hidden=4096, inter=14336, layers=8, heads=32, kv=8, dim=128, vocab=128256, theta=500000.0, bias=False, ff=21504,
               q_rank=1536, kv_rank=512, rot=64),
    "0.5b": dict(hidden=896, inter=4864, layers=24, heads=14, kv=2, dim=64, vocab=151936, theta=1000000.0, bias=True, ff=7296,
                 q_rank=448, kv_rank=256, rot=32),
}
EPS = 1e-6
TAPS = 4
KEEP_FIRST = 4
STEP_ROWS = 32      # rows of the INT4 decoders that take prompts
PROMPT_ROWS = 512   # rows of the layered decoders that take prompts


def listed():
    return [
        # the smallest call: one token through one square projection
        dict(name="linear_one_row", kind="linear", rows=1, n=4096, k=4096, group=32, bias=False),
        # a prompt through the module, the default group size; neither the rows nor the outputs are whole tiles
        dict(name="linear_prompt", kind="linear", rows=301, n=14330, k=4096, group=64, bias=True),
        # a feed-forward block for a server's batch of sixteen
        dict(name="mlp_16_rows", kind="mlp", size="8b", rows=16, group=32),
        # one user of a small model
        dict(name="generate_small", kind="generate", size="0.5b", context=1024, tokens=16, group=32),
        # one user of a large model, long context
        dict(name="generate_large", kind="generate", size="8b", context=4096, tokens=16, group=32),
        # a server with few and with many sequences
        dict(name="batch_8", kind="batch", size="8b", batch=8, context=4096, group=32),
        dict(name="batch_32", kind="batch", size="8b", batch=32, context=4096, group=32),
        # an odd number of new tokens behind a thousand old ones
        dict(name="prompt_333", kind="prompt", size="8b", start=1024, tokens=333, group=32),
        # the bfloat16 designs, decoding and reading a prompt
        dict(name="dabevik_decode_8", kind="dabevik_decode", size="8b", batch=8, context=2048, span=4096),
        dict(name="dabevik_prompt", kind="dabevik_prompt", size="8b", tokens=2501, span=4096),
        dict(name="sukalorn_decode_32", kind="sukalorn_decode", size="8b", batch=32, context=1024, span=4096),
        dict(name="sukalorn_prompt", kind="sukalorn_prompt", size="8b", tokens=4001, span=4096),
    ]


def _log(rng, lo, hi):
    """A whole number from lo to hi, spread over its logarithm."""
    return min(hi, max(lo, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    kind = rng.choice(["linear", "linear", "mlp", "generate", "batch", "batch", "prompt", "dabevik_decode", "dabevik_prompt",
                       "sukalorn_decode", "sukalorn_prompt"])
    group = rng.choice([32, 64])
    size = rng.choice(["8b", "0.5b"])
    if kind == "linear":
        n, k = rng.choice([(4096, 4096), (6144, 4096), (14336, 4096), (4096, 14336), (1152, 896), (4864, 896), (896, 4864)])
        n -= rng.choice([0, 0, rng.randrange(64)])
        return dict(kind=kind, rows=_log(rng, 1, 512), n=n, k=k, group=rng.choice([32, 64, 128]), bias=rng.random() < 0.5)
    if kind == "mlp":
        return dict(kind=kind, size=size, rows=_log(rng, 1, 64), group=group)
    if kind == "generate":
        return dict(kind=kind, size=size, context=_log(rng, 16, 4096), tokens=rng.randrange(4, 17), group=group)
    if kind == "batch":
        return dict(kind=kind, size=size, batch=_log(rng, 2, 32), context=_log(rng, 64, 4096), group=group)
    if kind == "prompt":
        return dict(kind=kind, size=size, start=rng.choice([0, _log(rng, 16, 3600)]), tokens=_log(rng, 3, 400), group=group)
    span = rng.choice([1024, 4096])
    if kind == "dabevik_decode":
        return dict(kind=kind, size=size, batch=_log(rng, 1, 16), context=_log(rng, 64, 2048), span=span)
    if kind == "sukalorn_decode":
        return dict(kind=kind, size=size, batch=_log(rng, 1, 32), context=_log(rng, 64, 1024), span=span)
    return dict(kind=kind, size=size, tokens=_log(rng, 16, 2501 if kind == "dabevik_prompt" else 4001), span=span)


# ------------------------------------------------------------------ inputs, made from the seed alone
class _Random:
    """Seeded numbers on the GPU."""

    def __init__(self, seed):
        self.gen = torch.Generator("cuda").manual_seed(int(seed))

    def normal(self, *shape, std=1.0, mean=0.0):
        t = torch.empty(*shape, device="cuda")
        return t.normal_(mean, std, generator=self.gen)

    def bf16(self, *shape, std=0.02, mean=0.0):
        return self.normal(*shape, std=std, mean=mean).to(torch.bfloat16)

    def ids(self, n, vocab):
        return torch.randint(vocab, (n,), device="cuda", generator=self.gen).tolist()

    def int4(self, n, k, group):
        """Normal weights as (codes in bytes, low nibble first; one scale per group)."""
        w = self.normal(n, k // group, group, std=0.02)
        scale = (w.abs().amax(-1) / 7).clamp_min(1e-8)
        code = (w / scale[..., None]).round_().clamp_(-8, 7).add_(8).to(torch.uint8).reshape(n, k)
        return code[:, 0::2] | (code[:, 1::2] << 4), scale


def _int4_model(case, rnd):
    z, g = SIZES[case["size"]], case["group"]
    h, i, q, kv = z["hidden"], z["inter"], z["heads"] * z["dim"], z["kv"] * z["dim"]
    layers = []
    for _ in range(z["layers"]):
        layers.append(dict(norm1=rnd.normal(h, std=0.1, mean=1.0), qkv=rnd.int4(q + 2 * kv, h, g), o=rnd.int4(h, q, g),
                           norm2=rnd.normal(h, std=0.1, mean=1.0), gate=rnd.int4(i, h, g), up=rnd.int4(i, h, g), down=rnd.int4(h, i, g),
                           bias=rnd.normal(q + 2 * kv, std=0.1) if z["bias"] else None))
    return dict(layers=layers, embed=rnd.normal(z["vocab"], h, std=0.02), norm=rnd.normal(h, std=0.1, mean=1.0), head=rnd.int4(z["vocab"], h, g))


def _contexts(case):
    """Positions in the cache in front of the step, per sequence."""
    if case["kind"] == "generate":
        return [case["context"]]
    if case["kind"] == "prompt":
        return [case["start"]]
    b = case["batch"]
    return [max(1, case["context"] * (i + 1) // b - i % 3) for i in range(b)]


def _caches(case, rnd):
    """Per sequence and layer the keys (rotated) and values in the cache, [kv heads, positions, dim]."""
    z = SIZES[case["size"]]
    return [[(rnd.normal(z["kv"], n, z["dim"], std=0.5), rnd.normal(z["kv"], n, z["dim"])) for _ in range(z["layers"])] for n in _contexts(case)]


def _dabevik_weights(case, rnd):
    z = SIZES[case["size"]]
    w, q, kv, ff = z["hidden"], z["heads"] * z["dim"], z["kv"] * z["dim"], z["ff"]
    layers = []
    for _ in range(z["layers"]):
        t = {n: rnd.bf16(w, mean=1.0) for n in ("norm1", "norm1_after", "norm2", "norm2_after")}
        t.update(conv1=rnd.bf16(w, TAPS, std=0.2), conv2=rnd.bf16(w, TAPS, std=0.2), q_w=rnd.bf16(q, w), q_b=rnd.bf16(q), k_w=rnd.bf16(kv, w),
                 k_b=rnd.bf16(kv), v_w=rnd.bf16(kv, w), v_b=rnd.bf16(kv), q_norm=rnd.bf16(q, mean=1.0), k_norm=rnd.bf16(kv, mean=1.0),
                 talk=rnd.bf16(z["heads"], z["heads"], std=0.2), o_w=rnd.bf16(w, q), o_b=rnd.bf16(w), up_w=rnd.bf16(ff, w), down_w=rnd.bf16(w, ff),
                 act=rnd.bf16(4, std=0.5))
        layers.append(t)
    return layers, dict(embed=rnd.bf16(z["vocab"], w, std=1.0), norm=rnd.bf16(w, mean=1.0), pos=rnd.bf16(_positions(case), w))


def _is_latent(i):
    return i % 3 == 1


def _sukalorn_weights(case, rnd):
    z = SIZES[case["size"]]
    w, h, d, ff = z["hidden"], z["heads"], z["dim"], z["ff"]
    layers = []
    for i in range(z["layers"]):
        t = dict(norm1=rnd.bf16(w), norm2=rnd.bf16(w), up_w=rnd.bf16(ff, w), down_w=rnd.bf16(w, ff), o_w=rnd.bf16(w, h * d))
        if _is_latent(i):
            qr, kr, rd = z["q_rank"], z["kv_rank"], z["rot"]
            t.update(dq_w=rnd.bf16(qr, w), dq_norm=rnd.bf16(qr, mean=1.0), uq_w=rnd.bf16(h * (d + rd), qr), dkv_w=rnd.bf16(kr + rd, w),
                     dkv_norm=rnd.bf16(kr, mean=1.0), uk_w=rnd.bf16(h * d, kr), uv_w=rnd.bf16(h * d, kr))
        else:
            t.update(q_w=rnd.bf16(h * d, w), k_w=rnd.bf16(z["kv"] * d, w), v_w=rnd.bf16(z["kv"] * d, w), gate_w=rnd.bf16(h, w),
                     vmix=rnd.bf16(1, std=0.1, mean=0.5))
        layers.append(t)
    return layers, dict(embed=rnd.bf16(z["vocab"], w, std=1.0), embed_norm=rnd.bf16(w), norm=rnd.bf16(w), head=rnd.bf16(z["vocab"], w))


def _positions(case):
    return (case["tokens"] if "tokens" in case else case["context"]) + 64


# ------------------------------------------------------------------ what a program has in hand, and the pass
def _module(weights, bias, k, group):
    packed, scales = weights
    m = tb.QuantizedLinear(k, packed.shape[0], bias=bias is not None, group_size=group).cuda()
    m.qweight.copy_(packed)
    m.scales.copy_(scales)
    if bias is not None:
        m.bias.data.copy_(bias)
    return m


def _linear_inputs(case, rnd):
    w = rnd.int4(case["n"], case["k"], case["group"])
    return w, rnd.normal(case["n"]) if case["bias"] else None, rnd.normal(case["rows"], case["k"])


def _mlp_inputs(case, rnd):
    z, g = SIZES[case["size"]], case["group"]
    h, i = z["hidden"], z["inter"]
    return rnd.int4(i, h, g), rnd.int4(i, h, g), rnd.int4(h, i, g), rnd.normal(case["rows"], h)


class _DeviceLogits:
    """The decoder's logits buffer, seen by torch without a copy.  A tensor made from it keeps the decoder alive."""

    def __init__(self, dec, rows):
        self.dec = dec
        self.__cuda_array_interface__ = dict(shape=(rows, dec.vocab_size), typestr="<f4", version=2,
                                             data=(tb.lib().tb_decoder_logits_device(dec.handle), False))


def prepare(case, seed):
    rnd, kind = _Random(seed), case["kind"]
    if kind == "linear":
        w, bias, x = _linear_inputs(case, rnd)
        return dict(kind=kind, x=x, module=_module(w, bias, case["k"], case["group"]).requires_grad_(False))
    if kind == "mlp":
        *ws, x = _mlp_inputs(case, rnd)
        z = SIZES[case["size"]]
        ks = (z["hidden"], z["hidden"], z["inter"])
        return dict(kind=kind, x=x, modules=[_module(w, None, k, case["group"]).requires_grad_(False) for w, k in zip(ws, ks)])
    z = SIZES[case["size"]]
    if kind in ("generate", "batch", "prompt"):
        model, caches = _int4_model(case, rnd), _caches(case, rnd)
        contexts = _contexts(case)
        rows = {"generate": 1, "batch": case.get("batch"), "prompt": STEP_ROWS}[kind]
        data = [[w["norm1"], *w["qkv"], *w["o"], w["norm2"], *w["gate"], *w["up"], *w["down"], w["bias"]] for w in model["layers"]]
        dec = tb.B200QwenDecoder(model["embed"], data, model["norm"], *model["head"], z["layers"], z["hidden"], z["inter"], z["heads"], z["kv"],
                                 z["dim"], case["group"], EPS, max(contexts) + case.get("tokens", 1) + 64, z["theta"], max_batch=rows)
        for b, (n, layers) in enumerate(zip(contexts, caches)):
            if n:
                dec.copy_kv_cache_from_tensors([k for k, _ in layers], [v for _, v in layers], n, seq=b)
        ids = rnd.ids(max(case.get("tokens", 1), len(contexts)), z["vocab"])
        state = dict(kind=kind, dec=dec, start=contexts[0], ids=ids, tokens=case.get("tokens", 1))
    else:
        build, batch = (_dabevik, kind == "dabevik_decode") if kind.startswith("dabevik") else (_sukalorn, kind == "sukalorn_decode")
        dec = build(case, rnd, case["batch"] if batch else 1)
        if not batch:
            return dict(kind=kind, dec=dec, ids=rnd.ids(case["tokens"], z["vocab"]))
        contexts = _contexts(case)
        texts = [rnd.ids(n + 1, z["vocab"]) for n in contexts]
        for b, t in enumerate(texts):
            dec.extend(t[:-1], 0, seq=b)
        state = dict(kind="batch", dec=dec, ids=[t[-1] for t in texts])
    if state["kind"] == "batch":
        state.update(ids=np.array(state["ids"], np.int64), offsets=np.array(contexts, np.int64),
                     logits=torch.as_tensor(_DeviceLogits(state["dec"], len(contexts)), device="cuda"))
    return state


def _dabevik(case, rnd, batch):
    z = SIZES[case["size"]]
    layers, t = _dabevik_weights(case, rnd)
    specs = [tb.LayerSpec(z["heads"], z["kv"], z["dim"], z["dim"], z["dim"] ** -0.5, case["span"], KEEP_FIRST, z["ff"], None, w) for w in layers]
    return tb.LayeredDecoder(specs, t["embed"], t["norm"], t["pos"], hidden_size=z["hidden"], vocab_size=z["vocab"], norm_eps=1e-5,
                             max_seq_len=_positions(case), embed_scale=1.0, conv_taps=TAPS, max_batch=batch, prefill_rows=PROMPT_ROWS)


def _sukalorn(case, rnd, batch):
    z = SIZES[case["size"]]
    layers, t = _sukalorn_weights(case, rnd)
    specs = []
    for i, w in enumerate(layers):
        common = dict(ff=z["ff"], activation="relu2", tensors=w)
        if _is_latent(i):
            specs.append(tb.LayerSpec(z["heads"], 1, z["dim"], z["dim"], (z["dim"] + z["rot"]) ** -0.5, q_rank=z["q_rank"], kv_rank=z["kv_rank"],
                                      rot_dim=z["rot"], rot_dims=z["rot"], rot_base=50000.0, **common))
        else:
            specs.append(tb.LayerSpec(z["heads"], z["kv"], z["dim"], z["dim"], z["dim"] ** -0.5, mask_chunk=case["span"], qk_unit_norm=True,
                                      score_softcap=50.0, distance_bias=8.0, value_mix=True, **common))
    return tb.LayeredDecoder(specs, t["embed"], t["norm"], embed_norm=t["embed_norm"], head=t["head"], hidden_size=z["hidden"],
                             vocab_size=z["vocab"], norm_eps=EPS, norm_offset=1.0, max_seq_len=_positions(case), max_batch=batch,
                             prefill_rows=PROMPT_ROWS)


def run(state):
    kind = state["kind"]
    if kind == "linear":
        return state["module"](state["x"])
    if kind == "mlp":
        return tb.fused_swiglu_mlp(state["x"], *state["modules"])
    dec = state["dec"]
    if kind == "generate":
        tokens = dec.generate_greedy(state["ids"][0], state["start"], state["tokens"])
        return dict(tokens=np.array(tokens), logits=dec.get_logits())
    if kind == "batch":
        status = tb.lib().tb_decoder_step_batch(dec.handle, state["ids"].ctypes.data, state["offsets"].ctypes.data, len(state["ids"]), None)
        if status:
            raise tb.TorchBurnB200Error(status, tb.last_error())
        return state["logits"]
    return dec.extend(state["ids"], state.get("start", 0), want=[len(state["ids"]) - 1])


# ------------------------------------------------------------------ what a pass cannot do without
def _int4_bytes(n, k, group):
    return n * k // 2 + n * (k // group) * 4


def work(case):
    kind = case["kind"]
    if kind == "linear":
        m, n, k = case["rows"], case["n"], case["k"]
        return dict(bytes=_int4_bytes(n, k, case["group"]) + 4 * (m * k + m * n + (n if case["bias"] else 0)), flops=2 * m * n * k)
    z = SIZES[case["size"]]
    h, i, q, kv, vocab, layers = z["hidden"], z["inter"], z["heads"] * z["dim"], z["kv"] * z["dim"], z["vocab"], z["layers"]
    if kind == "mlp":
        m, g = case["rows"], case["group"]
        return dict(bytes=2 * _int4_bytes(i, h, g) + _int4_bytes(h, i, g) + 8 * m * h, flops=6 * m * h * i)
    if kind in ("generate", "batch", "prompt"):
        g = case["group"]
        body = layers * (_int4_bytes(q + 2 * kv, h, g) + _int4_bytes(h, q, g) + 2 * _int4_bytes(i, h, g) + _int4_bytes(h, i, g))
        head = _int4_bytes(vocab, h, g)
        per_row = 2 * layers * (h * (2 * q + 2 * kv) + 3 * h * i)
        past, new = sum(_contexts(case)), case["tokens"] if kind == "prompt" else 1
        rows, steps = len(_contexts(case)) * new, case["tokens"] if kind == "generate" else 1
        seen = rows * past / len(_contexts(case)) + rows * new / 2 + steps / 2   # keys over all rows of a step
        last = rows if kind != "prompt" else 1
        return dict(bytes=steps * (body + head + layers * 2 * kv * 4 * (past + rows) + 4 * rows * h + 4 * last * vocab),
                    flops=steps * (rows * per_row + layers * 4 * q * seen + 2 * last * vocab * h))
    if kind.startswith("dabevik"):
        per_layer = h * (2 * q + 2 * kv) + 2 * h * z["ff"]
        body, cache, per_key = layers * per_layer, layers * 2 * kv * 2, layers * 4 * q
    else:
        latent = sum(_is_latent(j) for j in range(layers))
        plain = layers - latent
        up = z["q_rank"] * (h + q + z["heads"] * z["rot"]) + h * (z["kv_rank"] + z["rot"]) + 2 * q * z["kv_rank"] + q * h
        body = latent * up + plain * (h * (2 * q + 2 * kv) + z["heads"] * h) + layers * 2 * h * z["ff"]
        cache = plain * 2 * kv * 2 + latent * 2 * (z["kv_rank"] + z["rot"])
        per_key = plain * 4 * q + latent * (4 * q + 2 * z["heads"] * z["rot"])
    if "tokens" in case:
        n = case["tokens"]
        return dict(bytes=2 * (body + vocab * h) + 2 * n * h + n * cache + 4 * vocab, flops=2 * n * body + per_key * n * (n + 1) / 2 + 2 * vocab * h)
    rows, past = case["batch"], sum(_contexts(case))
    return dict(bytes=2 * (body + vocab * h) + 2 * rows * h + (past + rows) * cache + 4 * rows * vocab,
                flops=2 * rows * (body + vocab * h) + per_key * (past + rows))


def tolerance(case):
    # about four times the error against 64 bits that was measured: 4e-7, 2.5e-6 and 5.5e-3
    if case["kind"] in ("linear", "mlp"):
        return dict(rel=2e-6)                 # 32-bit sums
    if case["kind"] in ("generate", "batch", "prompt"):
        return dict(rel=1e-5, differ=0.0)     # 32-bit sums through every layer
    return dict(rel=0.02, max=0.2)            # bfloat16 activations through every layer


# ------------------------------------------------------------------ the same in 64 bits
def _wide(weights):
    packed, scale = weights
    code = torch.stack([packed & 15, packed >> 4], -1).reshape(scale.shape[0], scale.shape[1], -1).double() - 8
    return (code * scale.double()[..., None]).reshape(scale.shape[0], -1)


def _unit(x, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)


def _attend(q, k, v, mask, scale, cap=None, bias=None, talk=None):
    """q [rows, heads, dim], k and v [positions, kv heads, dim], mask(lo, hi) [hi - lo, positions]; 256 rows at a time."""
    heads = q.shape[1]
    k, v = (t.permute(1, 0, 2).repeat_interleave(heads // t.shape[1], 0) for t in (k, v))
    out = []
    for lo in range(0, q.shape[0], 256):
        hi = min(lo + 256, q.shape[0])
        s = q[lo:hi].transpose(0, 1) @ k.transpose(1, 2) * scale
        if cap is not None:
            s = cap * torch.tanh(s / cap)
        if bias is not None:
            s = s - bias(lo, hi)
        p = torch.softmax(s.masked_fill(~mask(lo, hi)[None], -math.inf), -1)
        if talk is not None:
            p = (talk @ p.reshape(heads, -1)).reshape(p.shape)
        out.append((p @ v).transpose(0, 1))
    return torch.cat(out).reshape(q.shape[0], -1)


def _exact_int4(case, rnd):
    z, g = SIZES[case["size"]], case["group"]
    model, caches = _int4_model(case, rnd), _caches(case, rnd)
    contexts = _contexts(case)
    ids = rnd.ids(max(case.get("tokens", 1), len(contexts)), z["vocab"])
    heads, kv, dim = z["heads"], z["kv"], z["dim"]
    layers = [{n: (_wide(t) if isinstance(t, tuple) else None if t is None else t.double()) for n, t in w.items()} for w in model["layers"]]
    head, norm = _wide(model["head"]), model["norm"].double()
    caches = [[(k.double().transpose(0, 1), v.double().transpose(0, 1)) for k, v in seq] for seq in caches]
    freq = z["theta"] ** (-2.0 * torch.arange(dim // 2, device="cuda", dtype=torch.float64) / dim)

    def turn(x, pos):
        a = (pos[:, None] * freq)[:, None, :]
        lo, hi = x[..., : dim // 2], x[..., dim // 2:]
        return torch.cat([lo * a.cos() - hi * a.sin(), hi * a.cos() + lo * a.sin()], -1)

    def step(tokens, per_seq):
        """per_seq tokens of every sequence behind what its cache holds; the logits of all rows."""
        x = model["embed"][tokens].double()
        for l, w in enumerate(layers):
            y = _unit(x, EPS) * w["norm1"] @ w["qkv"].T
            if w["bias"] is not None:
                y = y + w["bias"]
            q, k, v = y.split([heads * dim, kv * dim, kv * dim], 1)
            outs = []
            for b, seq in enumerate(caches):
                r = slice(b * per_seq, (b + 1) * per_seq)
                n0 = seq[l][0].shape[0]
                pos = torch.arange(n0, n0 + per_seq, device="cuda").double()
                keys = torch.cat([seq[l][0], turn(k[r].reshape(-1, kv, dim), pos)])
                values = torch.cat([seq[l][1], v[r].reshape(-1, kv, dim)])
                seq[l] = (keys, values)
                at = torch.arange(keys.shape[0], device="cuda")[None, :]
                outs.append(_attend(turn(q[r].reshape(-1, heads, dim), pos), keys, values, lambda lo, hi: at <= pos[lo:hi, None], dim ** -0.5))
            x = x + torch.cat(outs) @ w["o"].T
            y = _unit(x, EPS) * w["norm2"]
            x = x + (torch.nn.functional.silu(y @ w["gate"].T) * (y @ w["up"].T)) @ w["down"].T
        if case["kind"] == "prompt":
            x = x[-1:]
        return _unit(x, EPS) * norm @ head.T

    if case["kind"] != "generate":
        return step(ids if case["kind"] == "prompt" else ids[: len(contexts)], case["tokens"] if case["kind"] == "prompt" else 1)
    tokens, token = [], ids[0]
    for _ in range(case["tokens"]):
        logits = step([token], 1)[0]
        token = int(logits.argmax())
        tokens.append(token)
    return dict(tokens=np.array(tokens), logits=logits)


def _texts(case, rnd):
    z = SIZES[case["size"]]
    return [rnd.ids(case["tokens"], z["vocab"])] if "tokens" in case else [rnd.ids(n + 1, z["vocab"]) for n in _contexts(case)]


def _pieces(texts):
    ends = np.cumsum([len(t) for t in texts]).tolist()
    return [slice(e - len(t), e) for t, e in zip(texts, ends)]


def _exact_dabevik(case, rnd):
    z, eps = SIZES[case["size"]], 1e-5
    layers, tables = _dabevik_weights(case, rnd)
    texts = _texts(case, rnd)
    pieces = _pieces(texts)
    heads, kv, dim = z["heads"], z["kv"], z["dim"]
    x = torch.cat([tables["embed"][t].double() + tables["pos"][: len(t)].double() for t in texts])

    def conv(h, taps):
        out = h.clone()
        for p in pieces:
            for j in range(TAPS):
                back = TAPS - 1 - j
                if p.stop - p.start > back:
                    out[p.start + back:p.stop] += taps[:, j] * h[p.start:p.stop - back]
        return out

    for w in layers:
        w = {n: t.double() for n, t in w.items()}
        h = conv(_unit(x, eps) * w["norm1"], w["conv1"])
        q = (_unit(h @ w["q_w"].T + w["q_b"], eps) * w["q_norm"]).reshape(-1, heads, dim)
        k = (_unit(h @ w["k_w"].T + w["k_b"], eps) * w["k_norm"]).reshape(-1, kv, dim)
        v = (h @ w["v_w"].T + w["v_b"]).reshape(-1, kv, dim)
        outs = []
        for p in pieces:
            at = torch.arange(p.stop - p.start, device="cuda")

            def mask(lo, hi, at=at):
                i = at[lo:hi, None]
                return (at <= i) & ((i - at < case["span"]) | (at < KEEP_FIRST))
            outs.append(_attend(q[p], k[p], v[p], mask, dim ** -0.5, talk=w["talk"]))
        x = x + _unit(torch.cat(outs) @ w["o_w"].T + w["o_b"], eps) * w["norm1_after"]
        h = conv(_unit(x, eps) * w["norm2"], w["conv2"])
        u = h @ w["up_w"].T
        a, b, c, e = w["act"]
        u = a * _unit(u, eps) + b * _unit(u ** 2, eps) + c * _unit(u ** 3, eps) + e
        x = x + _unit(u @ w["down_w"].T, eps) * w["norm2_after"]
    last = x[[p.stop - 1 for p in pieces]]
    return _unit(last, eps) * tables["norm"].double() @ tables["embed"].double().T


def _exact_sukalorn(case, rnd):
    z = SIZES[case["size"]]
    layers, tables = _sukalorn_weights(case, rnd)
    texts = _texts(case, rnd)
    pieces = _pieces(texts)
    heads, kv, dim, rot = z["heads"], z["kv"], z["dim"], z["rot"]
    x = _unit(tables["embed"][sum(texts, [])].double(), EPS) * (1 + tables["embed_norm"].double())
    slope = 2.0 ** (-8.0 * (torch.arange(heads, device="cuda").double() + 1) / heads)
    pos = torch.cat([torch.arange(len(t), device="cuda") for t in texts]).double()

    def turn(t):
        a = pos[:, None] * 50000.0 ** (-2.0 * torch.arange(rot // 2, device="cuda").double() / rot)
        a = a[:, None, :]
        u, v = t[..., 0::2], t[..., 1::2]
        return torch.stack([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()], -1).flatten(-2)

    first = None
    for i, w in enumerate(layers):
        w = {n: t.double() for n, t in w.items()}
        h = _unit(x, EPS) * (1 + w["norm1"])
        if _is_latent(i):
            c = _unit(h @ w["dq_w"].T, EPS) * w["dq_norm"]
            q = (c @ w["uq_w"].T).reshape(-1, heads, dim + rot)
            q = torch.cat([q[..., :dim], turn(q[..., dim:])], -1)
            d = h @ w["dkv_w"].T
            c = _unit(d[:, : z["kv_rank"]], EPS) * w["dkv_norm"]
            k = torch.cat([(c @ w["uk_w"].T).reshape(-1, heads, dim), turn(d[:, None, z["kv_rank"]:]).expand(-1, heads, -1)], -1)
            v = (c @ w["uv_w"].T).reshape(-1, heads, dim)
        else:
            q = _unit((h @ w["q_w"].T).reshape(-1, heads, dim), EPS)
            k = _unit((h @ w["k_w"].T).reshape(-1, kv, dim), EPS)
            v = (h @ w["v_w"].T).reshape(-1, kv, dim)
            if first is None:
                first = v
            else:
                v = (1 - w["vmix"]) * v + w["vmix"] * first
        outs = []
        for p in pieces:
            at = torch.arange(p.stop - p.start, device="cuda")

            def mask(lo, hi, at=at, latent=_is_latent(i)):
                r = at[lo:hi, None]
                return (at <= r) if latent else (at <= r) & (r // case["span"] == at // case["span"])

            def bias(lo, hi, at=at):
                return slope[:, None, None] * (at[lo:hi, None] - at)[None].double()
            if _is_latent(i):
                outs.append(_attend(q[p], k[p], v[p], mask, (dim + rot) ** -0.5))
            else:
                outs.append(_attend(q[p], k[p], v[p], mask, dim ** -0.5, cap=50.0, bias=bias))
        o = torch.cat(outs)
        if not _is_latent(i):
            o = (o.reshape(-1, heads, dim) * torch.sigmoid(h @ w["gate_w"].T)[..., None]).reshape(o.shape)
        x = x + o @ w["o_w"].T
        x = x + (_unit(x, EPS) * (1 + w["norm2"]) @ w["up_w"].T).relu().square() @ w["down_w"].T
    last = x[[p.stop - 1 for p in pieces]]
    return _unit(last, EPS) * (1 + tables["norm"].double()) @ tables["head"].double().T


def exact(case, seed):
    rnd, kind = _Random(seed), case["kind"]
    if kind == "linear":
        w, bias, x = _linear_inputs(case, rnd)
        y = x.double() @ _wide(w).T
        return y if bias is None else y + bias.double()
    if kind == "mlp":
        gate, up, down, x = _mlp_inputs(case, rnd)
        y = x.double()
        return (torch.nn.functional.silu(y @ _wide(gate).T) * (y @ _wide(up).T)) @ _wide(down).T
    if kind in ("generate", "batch", "prompt"):
        return _exact_int4(case, rnd)
    return _exact_dabevik(case, rnd) if kind.startswith("dabevik") else _exact_sukalorn(case, rnd)
