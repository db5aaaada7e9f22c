"""The steps that a program serving a model with this engine has it run, as cases to time.

A case is one call of `StepFunction`: a batch of requests with their next tokens goes in, 32-bit logits of the
wanted rows come out. Sizes are those of the package's presets and of `bench.py`:

  qwen3-4b, qwen3-8b    the presets, all layers, in bfloat16; the 4B shape in 32-bit as well
  topidra               three linear-attention layers and a windowed one, the 4B shape's widths (`bench.py --config topidra`)
  limazen               four layers of chunked attention beside 32 routed experts (`bench.py --config limazen`)

A case names the model, its type and the batch: `prompts` requests that come with `new` tokens and hold none,
`portions` requests that hold `held` tokens and take `new` more (a long prompt fed in portions), and `decoding`
requests that hold about `context` tokens and take one more; `uneven` spreads their lengths over 0.1 .. 1 of it.
"""

import math
import zlib

import numpy as np
import torch

import layover_b200 as lb
from layover_b200.config.limazen import limazen_layer
from layover_b200.engine.step import DEFAULT_GRAPH_SIZES, StepFunction

PAGE = 16
NORM_STD = 0.1
# matrices ~ N(0, std): as in a trained model, what a sub-layer adds is a part of the stream it is added to, so that
# rounding is not blown up layer by layer and an expert chosen the other way in a near tie moves a row by little
STD = {"qwen3-4b": 0.001, "qwen3-8b": 0.001, "topidra": 0.02, "limazen": 0.002}
TYPES = {"bf16": torch.bfloat16, "fp32": torch.float32}


# ------------------------------------------------------------------------------------------- the cases
def _case(model="qwen3-4b", dtype="bf16", prompts=0, new=0, portions=0, held=0, decoding=0, context=0, uneven=False, **name):
    return {**name, "model": model, "dtype": dtype, "prompts": prompts, "new": new, "portions": portions, "held": held,
            "decoding": decoding, "context": context, "uneven": uneven}


def listed():
    return [
        # one chat, a token at a time: nothing to share the weights with, launches and their gaps count
        _case(name="decode one", decoding=1, context=700),
        # the benchmark's headline: eight requests in the middle of their answers
        _case(name="decode 8", decoding=8, context=3072),
        # a full server: requests of all lengths, the captured batch of 64
        _case(name="decode 64 uneven", decoding=64, context=4095, uneven=True),
        # a short question of no particular length, alone in its step: few tiles for the many-token products
        _case(name="prompt 333", prompts=1, new=333),
        # the benchmark's prompt, one portion of the largest size the engine is run with
        _case(name="prompt 2048", prompts=1, new=2048),
        # a portion in the middle of a long document, the attention reads all that came before
        _case(name="portion 512 after 8209", portions=1, new=512, held=8209),
        # continuous batching on the 8B shape: a portion of a prompt beside decoding requests, never captured
        _case("qwen3-8b", name="mixed 1000 + 24", portions=1, new=1000, held=1000, decoding=24, context=2100, uneven=True),
        # the true 32-bit path, in which users compare logits: decoding and a prompt
        _case(name="fp32 decode 4", dtype="fp32", decoding=4, context=900),
        _case(name="fp32 prompt 261", dtype="fp32", prompts=1, new=261),
        # a recurrent design's prompt: the scan beside products and a windowed attention
        _case("topidra", name="topidra prompt 1500", prompts=1, new=1500),
        # routed experts, few rows each: which experts' weights are read is up to the tokens
        _case("limazen", name="limazen decode 16", decoding=16, context=1500, uneven=True),
        # routed experts over two prompts at once: grouped products with ragged groups
        _case("limazen", name="limazen 2 prompts 611", prompts=2, new=611),
    ]


def draw(rng):
    def spread(low, high):                      # an odd size as likely as an even one, even over the logarithm
        return min(high, int(math.exp(rng.uniform(math.log(low), math.log(high + 1)))))

    kind = rng.choice(("decode", "decode", "decode", "prompt", "prompt", "portion", "mixed", "fp32", "topidra", "limazen", "limazen"))
    uneven = rng.random() < 0.5
    dense = rng.choice(("qwen3-4b", "qwen3-4b", "qwen3-8b"))
    if kind == "decode":
        batch = spread(1, 64)
        return _case(dense, decoding=batch, context=spread(48, min(8192, 160_000 // batch)), uneven=uneven)
    if kind == "prompt":
        return _case("qwen3-4b", prompts=1, new=spread(17, 2048)) if rng.random() < 0.7 else _case("qwen3-4b", prompts=3, new=spread(17, 680))
    if kind == "portion":
        return _case("qwen3-4b", portions=1, new=spread(128, 1024), held=spread(64, 12000))
    if kind == "mixed":
        return _case(dense, portions=1, new=spread(64, 1024), held=spread(16, 4000), decoding=spread(2, 48), context=spread(100, 3000), uneven=uneven)
    if kind == "fp32":
        if rng.random() < 0.5:
            return _case(dtype="fp32", decoding=spread(1, 8), context=spread(48, 2000), uneven=uneven)
        return _case(dtype="fp32", prompts=1, new=spread(5, 300))
    if kind == "topidra":
        return _case("topidra", prompts=rng.choice((1, 1, 2)), new=spread(17, 1024) if rng.random() < 0.5 else spread(300, 1024))
    if rng.random() < 0.5:
        return _case("limazen", decoding=spread(1, 64), context=spread(48, 4000), uneven=uneven)
    return _case("limazen", prompts=rng.choice((1, 2, 3)), new=spread(17, 700))


# ------------------------------------------------------------------------------------------- sizes
TOPIDRA = dict(width=2560, heads=32, kv=8, dim=128, ff=9728, window=1024, vocab=32768, layers=4, eps=1e-6)
LIMAZEN = dict(width=2048, heads=16, kv=4, dim=128, experts=32, top=4, expert_ff=1024, shared_ff=2048, chunk=1024, vocab=32768, layers=4,
               eps=1e-5, base=10000.0, factor=2.0, cap=25.0)


def _config(name):
    if name == "topidra":
        s = TOPIDRA
        mlp = {"kind": "dense", "ff": s["ff"]}
        linear = {"type": "lightning", "mlp": mlp, "mixer": {"heads": s["heads"], "dim": s["dim"], "vdim": s["dim"], "decay": _decays()}}
        softmax = {"type": "attention", "mlp": mlp, "mixer": {"heads": s["heads"], "kv_heads": s["kv"], "dim": s["dim"], "vdim": s["dim"],
                                                              "scale": s["dim"] ** -0.5, "mask": {"size": s["window"]}}}
        return lb.TopidraConfig(vocab=s["vocab"], width=s["width"], norm_eps=s["eps"],
                                layers=tuple(softmax if i % 4 == 3 else linear for i in range(s["layers"])))
    if name == "limazen":
        s = LIMAZEN
        layer = limazen_layer(s["heads"], s["kv"], s["dim"], s["dim"], s["chunk"], rot_dims=s["dim"] // 2, base=s["base"], factor=s["factor"],
                              experts=s["experts"], top=s["top"], expert_ff=s["expert_ff"], shared_ff=s["shared_ff"])
        return lb.LimazenConfig(vocab=s["vocab"], width=s["width"], norm_eps=s["eps"], layers=(layer,) * s["layers"], logit_softcap=s["cap"])
    return lb.preset(name)


def _decays():
    return [1.0 - 2.0 ** -(3 + 6 * h / TOPIDRA["heads"]) for h in range(TOPIDRA["heads"])]


def _lengths(case):
    """(tokens held, tokens that come) of every request, in the order of the batch."""
    n = case["decoding"]
    held = [case["context"]] * n
    if case["uneven"] and n > 1:
        held = [max(1, round(case["context"] * (0.1 + 0.9 * ((i * 7919) % n) / (n - 1)))) for i in range(n)]
    if case["model"] == "limazen":              # a chunk ends within a request, not with the very token of the step
        held = [h - 1 if (h + 1) % LIMAZEN["chunk"] == 0 else h for h in held]
    return [(0, case["new"])] * case["prompts"] + [(case["held"], case["new"])] * case["portions"] + [(h, 1) for h in held]


# ------------------------------------------------------------------------------------------- inputs
_model_in_use = {}


def _model(case):
    """The model with its weights, which a serving program loads once and keeps for all requests."""
    key = (case["model"], case["dtype"])
    if key not in _model_in_use:
        _model_in_use.clear()
        torch.cuda.empty_cache()
        _model_in_use[key] = lb.models.random_model(_config(case["model"]), seed=0, dtype=case["dtype"], std=STD[case["model"]], norm_std=NORM_STD)
    return _model_in_use[key]


def _tokens(case, seed, vocab):
    rng = np.random.default_rng(seed)
    return [rng.integers(0, vocab, new).tolist() for _, new in _lengths(case)]


def _kept(case, seed, layer, kv_heads, dim):
    """Keys and values that the requests hold, end to end, as large as the model's own projections make them."""
    width = {"limazen": LIMAZEN["width"], "topidra": TOPIDRA["width"]}.get(case["model"]) or lb.preset(case["model"]).hidden_size
    large = STD[case["model"]] * math.sqrt(width)
    gen = torch.Generator(device="cuda").manual_seed(seed * 1009 + layer)
    total = sum(held for held, _ in _lengths(case))
    return [(scale * torch.randn((total, kv_heads, dim), generator=gen, device="cuda")).to(TYPES[case["dtype"]])
            for scale in (large if case["model"] == "limazen" else 1.0, large)]      # Qwen3 norms its keys


class _State:
    pass


def prepare(case, seed):
    s = _State()
    model, lengths = _model(case), _lengths(case)
    s.prompt = case["prompts"] > 0
    s.tokens = _tokens(case, seed, model.spec.vocab_size)
    s.lengths = lengths
    pages = sum(-(-(held + new) // PAGE) + 1 for held, new in lengths)
    s.cache = lb.PagedKVCache(model, pages, block_tokens=PAGE, max_requests=max(DEFAULT_GRAPH_SIZES))
    if s.prompt:
        s.step = StepFunction(model, s.cache, cuda_graphs=True)
        return s
    s.seqs = [s.cache.open(str(i)) for i in range(len(lengths))]
    longest = max(held for held, _ in lengths)
    for upto in range(PAGE, longest + PAGE, PAGE):          # pages as requests that grow side by side get them
        for seq, (held, _) in zip(s.seqs, lengths):
            if upto - PAGE < held:
                s.cache.grow(seq, min(upto, held))
    where = torch.tensor([seq.tables[0].blocks[t // PAGE] * PAGE + t % PAGE for seq, (held, _) in zip(s.seqs, lengths) for t in range(held)],
                         device="cuda")
    for layer in range(len(model.spec.schedule)):
        view = s.cache.view(layer)
        for pool, rows in zip((view.k_pool, view.v_pool), _kept(case, seed, layer, view.k_pool.shape[1], view.k_pool.shape[3])):
            pool[where // PAGE, :, where % PAGE] = rows
    for seq, (held, _) in zip(s.seqs, lengths):
        s.cache.commit(seq, held)
    size = next(size for size in DEFAULT_GRAPH_SIZES if size >= len(lengths))
    s.step = StepFunction(model, s.cache, cuda_graphs=True, graph_sizes=(size,))
    if all(new == 1 for _, new in lengths):                 # a server captures its decode steps before it takes requests
        s.step.capture_all(tokens=longest + 1, from_tokens=longest + 1, sampled=False, skews=(1, 2))
    return s


def run(s):
    if s.prompt:                                            # new requests: opened, fed, and done
        s.seqs = [s.cache.open(str(i)) for i in range(len(s.lengths))]
    logits = s.step([lb.StepEntry(seq, ids, [len(ids) - 1]) for seq, ids in zip(s.seqs, s.tokens)])
    for seq, (held, _) in zip(s.seqs, s.lengths):
        if s.prompt:
            s.cache.close(seq)
        else:                                               # the new tokens are dropped again, as drafted ones are
            seq.num_tokens = held
    return logits


# ------------------------------------------------------------------------------------------- work and tolerance
def work(case):
    lengths, size = _lengths(case), {"bf16": 2, "fp32": 4}[case["dtype"]]
    tokens, rows = sum(new for _, new in lengths), len(lengths)
    pairs = sum(new * held + new * (new + 1) // 2 for held, new in lengths)          # (query, key) pairs under the mask
    held = sum(h for h, _ in lengths)
    if case["model"] == "topidra":
        s = TOPIDRA
        w, d, heads = s["width"], s["dim"], s["heads"]
        attention_in = (heads + 2 * s["kv"]) * d + heads
        weights = 3 * (5 * heads * d * w) + (attention_in + heads * d) * w + 4 * 3 * s["ff"] * w
        seen = sum(sum(min(t + 1, s["window"]) for t in range(new)) for _, new in lengths)
        flops = 2 * tokens * weights + 4 * heads * d * seen + 3 * 4 * tokens * heads * d * d + 2 * rows * w * s["vocab"]
        return {"bytes": 2 * (weights + w * s["vocab"]) + 4 * rows * s["vocab"], "flops": flops}
    if case["model"] == "limazen":
        s = LIMAZEN
        w, d, heads, kv, layers = s["width"], s["dim"], s["heads"], s["kv"], s["layers"]
        shared = ((3 * heads + 2 * kv) * d + 3 * s["shared_ff"] + s["experts"]) * w     # q, gate, k, v and o rows, shared expert, router
        expert = 3 * s["expert_ff"] * w
        touched = s["experts"] * (1 - (1 - s["top"] / s["experts"]) ** tokens)
        seen = sum(sum((h + t) % s["chunk"] + 1 for t in range(new)) for h, new in lengths)
        read = sum(h % s["chunk"] for h, _ in lengths) * 2 * kv * d * layers
        flops = layers * (2 * tokens * (shared + s["top"] * expert) + 4 * heads * d * seen) + 2 * rows * w * s["vocab"]
        return {"bytes": 2 * (layers * (shared + touched * expert) + w * s["vocab"] + read) + 4 * rows * s["vocab"], "flops": flops}
    c = lb.preset(case["model"])
    w, d, heads, kv, layers = c.hidden_size, c.head_dim, c.num_attention_heads, c.num_key_value_heads, c.num_hidden_layers
    weights = ((2 * heads + 2 * kv) * d + 3 * c.intermediate_size) * w
    cached = (held + tokens) * 2 * kv * d * layers
    return {"bytes": size * (layers * weights + w * c.vocab_size + cached) + 4 * rows * c.vocab_size,
            "flops": layers * (2 * tokens * weights + 4 * heads * d * pairs) + 2 * rows * w * c.vocab_size}


def tolerance(case):
    """About four times the distance to `exact`, at most 0.03. The 36 layers of a bfloat16 stream with its 73 roundings are
    0.011 (prompts) to 0.017 (decoding) off; the 4 layers of the others, over a 32-bit stream, 0.006 and 0.002 to 0.004; the 32-bit
    path 6e-6, of which the 32-bit angles of the rotation are the most."""
    if case["dtype"] == "fp32":
        return {"rel": 2.5e-5, "max": 2e-4}
    if case["model"] == "limazen":
        return {"rel": 0.016, "max": 0.2}
    return {"rel": 0.026 if case["model"] == "topidra" else 0.03, "max": 0.35}


# ------------------------------------------------------------------------------------------- the same in 64 bits
def exact(case, seed):
    """The step's logits in 64 bits: one function per design, plain torch over the same weights and inputs."""
    plain = {"topidra": _plain_topidra, "limazen": _plain_limazen}.get(case["model"], _plain_qwen3)
    with torch.no_grad():
        return plain(case, seed)


class _Weights:
    """The model's random weights by name, drawn again: each from a generator of its own, rounded as the run keeps them."""

    def __init__(self, case):
        self.dtype, self.std = TYPES[case["dtype"]], STD[case["model"]]

    def _noise(self, name, shape):
        gen = torch.Generator(device="cuda").manual_seed(zlib.crc32(name.encode()))
        return torch.randn(shape, generator=gen, device="cuda")

    def __call__(self, name, *shape):
        return (self.std * self._noise(name, shape)).to(self.dtype).double()

    def kept32(self, name, *shape):
        return (self.std * self._noise(name, shape)).double()

    def norm(self, name, size):
        return (1.0 + NORM_STD * self._noise(name, (size,))).to(self.dtype).double()


def _rms(x, weight, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * weight


def _attend(q, k, v, scale, seen, sink=None):
    """q [n, H, d] over k, v [m, G, d] under the mask `seen` [n, m] -> [n, H * d]; a head at a time, to spare memory."""
    n, heads, d = q.shape
    out = torch.empty_like(q)
    for h in range(heads):
        g = h // (heads // k.shape[1])
        scores = (q[:, h] @ k[:, g].T * scale).masked_fill(~seen, -math.inf)
        if sink is not None:
            scores = torch.cat((scores, sink[h].expand(n, 1)), 1)
        p = torch.softmax(scores, -1)
        out[:, h] = p[:, : k.shape[0]] @ v[:, g]
    return out.reshape(n, heads * d)


def _turn(x, positions, rotated, base, factor=1.0):
    """Channels i and i + rotated/2 of every head by the angle position * base^(-2i/rotated) / factor."""
    half = rotated // 2
    angle = positions.double()[:, None] * (base ** (-2.0 * torch.arange(half, device="cuda").double() / rotated) / factor)
    cos, sin = torch.cos(angle)[:, None], torch.sin(angle)[:, None]
    a, b = x[..., :half], x[..., half:rotated]
    return torch.cat((a * cos - b * sin, b * cos + a * sin, x[..., rotated:]), -1)


def _layout(case, seed, vocab):
    """Token ids and positions end to end, and every request's (first kept row, tokens held, first row, tokens)."""
    lengths, tokens = _lengths(case), _tokens(case, seed, vocab)
    ids = torch.tensor([t for part in tokens for t in part], device="cuda")
    positions = torch.cat([torch.arange(held, held + new, device="cuda") for held, new in lengths])
    spans, past, row = [], 0, 0
    for held, new in lengths:
        spans.append((past, held, row, new))
        past, row = past + held, row + new
    last = torch.tensor([row + new - 1 for _, _, row, new in spans], device="cuda")
    return ids, positions, spans, last


def _attend_all(q, k, v, kept, spans, scale, visible, sink=None):
    out = []
    for past, held, row, new in spans:
        keys, values = (torch.cat((old[past: past + held].double(), own[row: row + new])) for old, own in zip(kept, (k, v)))
        i, j = torch.arange(held, held + new, device="cuda")[:, None], torch.arange(held + new, device="cuda")[None]
        out.append(_attend(q[row: row + new], keys, values, scale, (j <= i) & visible(i, j), sink))
    return torch.cat(out)


def _plain_qwen3(case, seed):
    c, w = lb.preset(case["model"]), _Weights(case)
    hid, d, heads, kv, ff, eps = c.hidden_size, c.head_dim, c.num_attention_heads, c.num_key_value_heads, c.intermediate_size, c.rms_norm_eps
    ids, positions, spans, last = _layout(case, seed, c.vocab_size)
    embedding = w("model.embed_tokens.weight", c.vocab_size, hid)
    x = embedding[ids]
    for layer in range(c.num_hidden_layers):
        p = f"model.layers.{layer}."
        h = _rms(x, w.norm(p + "input_layernorm.weight", hid), eps)
        q = (h @ w(p + "self_attn.q_proj.weight", heads * d, hid).T).view(-1, heads, d)
        k = (h @ w(p + "self_attn.k_proj.weight", kv * d, hid).T).view(-1, kv, d)
        v = (h @ w(p + "self_attn.v_proj.weight", kv * d, hid).T).view(-1, kv, d)
        q = _turn(_rms(q, w.norm(p + "self_attn.q_norm.weight", d), eps), positions, d, c.rope_theta)
        k = _turn(_rms(k, w.norm(p + "self_attn.k_norm.weight", d), eps), positions, d, c.rope_theta)
        o = _attend_all(q, k, v, _kept(case, seed, layer, kv, d), spans, d ** -0.5, lambda i, j: j >= 0)
        x = x + o @ w(p + "self_attn.o_proj.weight", hid, heads * d).T
        h = _rms(x, w.norm(p + "post_attention_layernorm.weight", hid), eps)
        gated = torch.nn.functional.silu(h @ w(p + "mlp.gate_proj.weight", ff, hid).T) * (h @ w(p + "mlp.up_proj.weight", ff, hid).T)
        x = x + gated @ w(p + "mlp.down_proj.weight", hid, ff).T
    head = embedding if c.tie_word_embeddings else w("lm_head.weight", c.vocab_size, hid)
    return _rms(x[last], w.norm("model.norm.weight", hid), eps) @ head.T


def _plain_topidra(case, seed):
    s, w = TOPIDRA, _Weights(case)
    hid, d, heads, kv, ff, eps = s["width"], s["dim"], s["heads"], s["kv"], s["ff"], s["eps"]
    silu = torch.nn.functional.silu
    ids, _, spans, last = _layout(case, seed, s["vocab"])
    decay = torch.tensor(_decays(), device="cuda").double()[:, None, None]
    x = w("embed", s["vocab"], hid)[ids]
    for layer in range(s["layers"]):
        p = f"l{layer}."
        h = _rms(x, w.norm(p + "norm1", hid), eps)
        if layer % 4 == 3:
            q = _rms(h @ w(p + "mix.q", heads * d, hid).T, w.norm(p + "mix.q.norm", heads * d), eps).view(-1, heads, d)
            k = _rms(h @ w(p + "mix.k", kv * d, hid).T, w.norm(p + "mix.k.norm", kv * d), eps).view(-1, kv, d)
            v = (h @ w(p + "mix.v", kv * d, hid).T).view(-1, kv, d)
            o = _attend_all(q, k, v, _kept(case, seed, layer, kv, d), spans, d ** -0.5, lambda i, j: i - j < s["window"], w(p + "mix.sink", heads))
            o = (o.view(-1, heads, d) * torch.sigmoid(h @ w(p + "mix.g", heads, hid).T)[..., None]).view(-1, heads * d)
        else:
            q, k, v = (silu(h @ w(p + f"mix.{n}", heads * d, hid).T).view(-1, heads, d) for n in "qkv")
            o = torch.empty_like(q)
            for _, _, row, new in spans:
                state = torch.zeros(heads, d, d, dtype=torch.float64, device="cuda")
                for t in range(row, row + new):
                    state = decay * state + k[t, :, :, None] * v[t, :, None, :]
                    o[t] = (q[t, :, None, :] @ state)[:, 0]
            gate = torch.sigmoid(h @ w(p + "mix.g", heads * d, hid).T)
            o = _rms(o.reshape(-1, heads * d), w.norm(p + "mix.norm", heads * d), eps) * gate
        x = x + _rms(o @ w(p + "mix.o", hid, heads * d).T, w.norm(p + "norm1b", hid), eps)
        h = _rms(x, w.norm(p + "norm2", hid), eps)
        h = (torch.relu(h @ w(p + "mlp.gate", ff, hid).T) * (h @ w(p + "mlp.up", ff, hid).T)) @ w(p + "mlp.down", hid, ff).T
        x = x + _rms(h, w.norm(p + "norm2b", hid), eps)
    return _rms(x[last], w.norm("final.norm", hid), eps) @ w("head", s["vocab"], hid).T


def _plain_limazen(case, seed):
    s, w = LIMAZEN, _Weights(case)
    hid, d, heads, kv, eps = s["width"], s["dim"], s["heads"], s["kv"], s["eps"]
    ids, positions, spans, last = _layout(case, seed, s["vocab"])

    def layer_norm(x, name):
        return torch.nn.functional.layer_norm(x, (hid,), w.norm(name, hid), w(name + ".b", hid), eps)

    def expert(h, prefix, ff):
        gated = torch.nn.functional.silu(h @ w(prefix + "gate", ff, hid).T) * (h @ w(prefix + "up", ff, hid).T)
        return gated @ w(prefix + "down", hid, ff).T

    x, first_values = w("embed", s["vocab"], hid)[ids], None
    for layer in range(s["layers"]):
        p = f"l{layer}."
        h = layer_norm(x, p + "norm1")
        q, k, v = ((h @ w(p + f"mix.{n}", count * d, hid).T + w(p + f"mix.{n}.b", count * d)).view(-1, count, d)
                   for n, count in (("q", heads), ("k", kv), ("v", kv)))
        q, k = (_turn(t, positions, d // 2, s["base"], s["factor"]) for t in (q, k))
        if first_values is None:
            first_values = v
        else:
            blend = w(p + "mix.vmix")
            v = (1 - blend) * v + blend * first_values
        o = _attend_all(q, k, v, _kept(case, seed, layer, kv, d), spans, d ** -0.5, lambda i, j: i // s["chunk"] == j // s["chunk"])
        mixed = (o * torch.sigmoid(h @ w(p + "mix.g", heads * d, hid).T)) @ w(p + "mix.o", hid, heads * d).T
        scores = torch.sigmoid(h @ w.kept32(p + "mlp.router", s["experts"], hid).T)
        chosen = torch.zeros_like(scores).scatter_(1, scores.topk(s["top"]).indices, 1.0).bool()
        fed = torch.sigmoid(h @ w.kept32(p + "mlp.shared.sg", 1, hid).T) * expert(h, p + "mlp.shared.", s["shared_ff"])
        for e in range(s["experts"]):
            rows = chosen[:, e].nonzero()[:, 0]
            if rows.numel():
                fed[rows] += expert(scores[rows, e, None] * h[rows], p + f"mlp.e{e}.", s["expert_ff"])
        x = x + mixed + fed
    logits = layer_norm(x[last], "final.norm") @ w("head", s["vocab"], hid).T
    return s["cap"] * torch.tanh(logits / s["cap"])
