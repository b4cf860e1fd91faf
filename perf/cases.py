"""Steps of the engine whose speed is followed: what a user's requests are made of, one step each.

A case is one step of a live engine.  ``decodes`` requests that hold up to ``context`` tokens decode one
token each, and ``prompts`` requests that hold ``history`` tokens run a portion of up to ``tokens`` tokens
(with ``ragged`` the requests' lengths run from the longest down to a quarter of it).  Steps of decoded
tokens alone replay the engine's decode graphs, sampling included; the others go through the step function
every prompt goes through.  Weights are the engine's own random ones at the layer sizes of the benchmark,
with all 28 layers at the smallest size and 4 at the larger ones.

``exact`` makes the logits again in 64 bits with plain torch: it draws the same weights by the law the
engine documents (one seeded generator, tensors in checkpoint order) and runs every request whole.
"""

import json
import math
import random
import tempfile
from pathlib import Path

import torch

VOCAB = 151936
PAGE = 16
EPS = 1e-6
# layer sizes: width, query heads, key/value heads, head size, feed-forward width
SIZES = {
    "0.6b": (1024, 16, 8, 128, 3072),
    "8b": (4096, 32, 8, 128, 12288),
    "32b": (5120, 64, 8, 128, 25600),
}
ROPE_BASE = 1000000.0
GUMAPEL_BASE, GUMAPEL_WINDOW, GUMAPEL_KEPT = 500000.0, 1024, 4
BIMOLIX_CHUNK, BIMOLIX_ROWS = 1024, 32


def _case(name, model="qwen3", size="0.6b", layers=28, dtype="bfloat16", decodes=0, context=0, prompts=0, tokens=0,
          history=0, ragged=False, sampled=False):
    made = dict(model=model, size=size, layers=layers, dtype=dtype, decodes=decodes, context=context, prompts=prompts,
                tokens=tokens, history=history, ragged=ragged, sampled=sampled)
    return made if name is None else dict(name=name, **made)


def listed():
    return [
        # one user chatting: the latency of a single token
        _case("decode-1", decodes=1, context=601),
        # the usual small batch at a few thousand tokens of context
        _case("decode-8", decodes=8, context=2048),
        # a busy server: many requests of all lengths, some greedy, some sampled
        _case("decode-48-sampled", decodes=48, context=2503, ragged=True, sampled=True),
        # a single short prompt: time to the first token of a question
        _case("prompt-61", prompts=1, tokens=61),
        # one prompt of a document's length
        _case("prompt-2048", prompts=1, tokens=2048),
        # continuous batching: portions of two long prompts beside decoding requests
        _case("mixed-24-and-2", decodes=24, context=1811, prompts=2, tokens=491, history=512, ragged=True),
        # a long document at wide layers, where the matrix products and the attention are large
        _case("prompt-8192-wide", size="8b", layers=4, prompts=1, tokens=8192),
        # decoding at the widest layers with long contexts of different lengths: weights and cache from memory
        _case("decode-8-widest", size="32b", layers=4, decodes=8, context=6007, ragged=True),
        # the 32-bit path, used to check a model's numbers: a batch of prompts, and decoding
        _case("float32-prompts", dtype="float32", prompts=3, tokens=301, ragged=True),
        _case("float32-decode-4", dtype="float32", decodes=4, context=701, ragged=True),
        # the other designs: windows with kept first tokens over a 32-bit stream; linear attention with a state a
        # request beside attention in chunks
        _case("gumapel-prompt-2048", model="gumapel", layers=4, prompts=1, tokens=2048),
        _case("bimolix-prompts", model="bimolix", layers=4, prompts=3, tokens=1501, ragged=True),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "prompt", "prompt", "mixed", "float32", "gumapel", "bimolix"])
    ragged = rng.random() < 0.6
    if kind == "decode":
        size, layers = rng.choice([("0.6b", 28), ("0.6b", 28), ("8b", 4), ("32b", 4)])
        decodes = _log_int(rng, 1, 64)
        context = _log_int(rng, 16, min(8000, 130000 // decodes))
        return _case(None, size=size, layers=layers, decodes=decodes, context=context, ragged=ragged,
                     sampled=decodes >= 24 and rng.random() < 0.5)
    if kind == "prompt":
        size, layers, most = rng.choice([("0.6b", 28, 4000), ("0.6b", 28, 4000), ("8b", 4, 8000), ("32b", 4, 3000)])
        prompts = _log_int(rng, 1, 6)
        return _case(None, size=size, layers=layers, prompts=prompts, tokens=_log_int(rng, 9, most // prompts),
                     history=rng.choice([0, 0, _log_int(rng, 16, 2000)]), ragged=ragged)
    if kind == "mixed":
        return _case(None, decodes=_log_int(rng, 1, 40), context=_log_int(rng, 40, 2400), prompts=rng.randint(1, 3),
                     tokens=_log_int(rng, 9, 700), history=rng.choice([0, _log_int(rng, 16, 1500)]), ragged=ragged)
    if kind == "float32":
        if rng.random() < 0.5:
            return _case(None, dtype="float32", decodes=_log_int(rng, 1, 12), context=_log_int(rng, 16, 1000), ragged=ragged)
        prompts = rng.randint(1, 3)
        return _case(None, dtype="float32", prompts=prompts, tokens=_log_int(rng, 9, 600 // prompts), ragged=ragged)
    if kind == "gumapel" and rng.random() < 0.4:
        return _case(None, model="gumapel", layers=4, decodes=_log_int(rng, 1, 32), context=_log_int(rng, 16, 3000), ragged=ragged)
    prompts = rng.randint(1, 4)
    return _case(None, model=kind, layers=4, prompts=prompts, tokens=_log_int(rng, 9, 4000 // prompts), ragged=ragged)


# ------------------------------------------------------------------------------------------ what a case's requests are
def _lengths(count, longest, ragged):
    if not ragged:
        return [longest] * count
    return [max(1, longest - (3 * longest * i) // (4 * count)) for i in range(count)]


def _requests(case, seed):
    """(tokens in the cache before the step, tokens of the step) of every request, decoding ones first."""
    rng = random.Random(1000003 * int(seed) + 17)
    made = []
    for length in _lengths(case["decodes"], case["context"], case["ragged"]):
        ids = [rng.randrange(VOCAB) for _ in range(length + 1)]
        made.append((ids[:length], ids[length:]))
    for length in _lengths(case["prompts"], case["tokens"], case["ragged"]):
        ids = [rng.randrange(VOCAB) for _ in range(case["history"] + length)]
        made.append((ids[:case["history"]], ids[case["history"]:]))
    return made


def _model_json(case):
    width, heads, kv, dim, ff = SIZES[case["size"]]
    layers = case["layers"]
    if case["model"] == "qwen3":
        return dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", vocab_size=VOCAB, hidden_size=width,
                    intermediate_size=ff, num_hidden_layers=layers, num_attention_heads=heads, num_key_value_heads=kv,
                    head_dim=dim, max_position_embeddings=40960, rope_theta=ROPE_BASE, rms_norm_eps=EPS,
                    tie_word_embeddings=case["size"] == "0.6b", hidden_act="silu", attention_bias=False,
                    use_sliding_window=False)
    made = []
    for index in range(layers):
        mixer = dict(heads=heads, dim=dim, vdim=dim)
        if case["model"] == "gumapel":
            mixer.update(kv_heads=kv, scale=dim ** -0.5, v_mix=True, mask=dict(size=GUMAPEL_WINDOW))
            if index % 4 != 3:
                mixer["mask"]["keep_first"] = GUMAPEL_KEPT
                mixer["rot"] = dict(base=GUMAPEL_BASE, dims=dim)
            made.append(dict(type="attention" if index % 4 == 3 else "attention_2", mixer=mixer, mlp=dict(kind="dense", ff=ff)))
        elif index % 2 == 0:
            mixer.update(decay=_decay(heads), rot=dict(base=ROPE_BASE, dims=dim))
            made.append(dict(type="retention", mixer=mixer, mlp=dict(kind="dense", ff=ff)))
        else:
            mixer.update(kv_heads=kv, scale=dim ** -0.5, bias_max=float(BIMOLIX_CHUNK), mask=dict(size=BIMOLIX_CHUNK))
            made.append(dict(type="attention", mixer=mixer, mlp=dict(kind="dense", ff=ff)))
    return dict(architecture=case["model"].capitalize(), vocab=VOCAB, width=width, norm=dict(eps=EPS), layers=made)


def _decay(heads):
    return [1.0 - 2.0 ** -(5 + 4 * h / heads) for h in range(heads)]


# ----------------------------------------------------------------------------------------------------- the engine's side
class _State:
    pass


def prepare(case, seed):
    from tinyvllm_b200 import EngineConfig, SamplingParams
    from tinyvllm_b200.engine.engine import Engine
    from tinyvllm_b200.engine.step import StepEntry

    width, heads, kv, dim, ff = SIZES[case["size"]]
    requests = _requests(case, seed)
    longest = max(len(held) + len(new) for held, new in requests)
    room = sum((len(held) + len(new)) // PAGE + 2 for held, new in requests) * PAGE
    per_token = 2 * case["layers"] * kv * dim * (4 if case["dtype"] == "float32" else 2)
    rows = max(case["decodes"], 1)
    bucket = 1 << (rows - 1).bit_length()
    with tempfile.TemporaryDirectory() as folder:
        Path(folder, "config.json").write_text(json.dumps(_model_json(case)))
        engine = Engine.from_config(EngineConfig(
            model=folder, dtype=case["dtype"], weights="random", seed=int(seed), max_model_len=4096 if longest < 4096 else 16384,
            max_num_seqs=max(bucket, len(requests)), max_num_batched_tokens=16384, prefill_chunk_size=8192,
            prefill_reserve_tokens=0, prefill_reserve_requests=0, kv_block_size=PAGE,
            kv_cache_memory_bytes=per_token * room, graph_batch_sizes=(bucket,)))
    runner = engine.runner
    state = _State()
    state.engine, state.runner, state.decode_only = engine, runner, case["prompts"] == 0
    state.fresh = case["decodes"] == 0 and case["history"] == 0
    state.entries = [StepEntry(i, tuple(new), (len(new) - 1,)) for i, (_, new) in enumerate(requests)]
    if not state.fresh:
        waiting = []
        for index, (held, _) in enumerate(requests):
            runner.open(index)
            if held:
                waiting.append(StepEntry(index, tuple(held)))
            if waiting and (index + 1 == len(requests) or sum(len(e.tokens) for e in waiting) >= 4096):
                runner.run(waiting)
                waiting = []
    state.sampled = case["sampled"]
    state.params = [SamplingParams(max_new_tokens=64, ignore_eos=True) if not case["sampled"] or i % 2 == 0 else
                    SamplingParams(max_new_tokens=64, ignore_eos=True, temperature=0.8, seed=i, top_k=50 if i % 4 == 1 else 0,
                                   top_p=0.95 if i % 4 == 3 else 1.0) for i in range(len(requests))]
    state.draws = [1] * len(requests)
    return state


def run(state):
    """The step, and the cache as it was before: a decoding or continued request stands where it stood
    (the plan is given back), a fresh prompt's request is closed."""
    runner = state.runner
    if state.fresh:
        for entry in state.entries:
            runner.open(entry.request_id)
        logits = runner.run(state.entries)
        for entry in state.entries:
            runner.close(entry.request_id)
        return {"logits": logits}
    plan = runner.plan(state.entries)
    if state.decode_only:
        tokens, logits = state.engine.graphs.run(plan, state.entries, state.params, state.draws)
        made = {"logits": logits, "tokens": tokens} if state.sampled else {"logits": logits}
    else:
        made = {"logits": runner.forward(state.entries, plan)}
    runner.manager.rollback(plan)
    return made


# --------------------------------------------------------------------------------------------------- what it cannot avoid
def _layer_weights(case):
    """Values of one layer's matrices, a mean over the layers."""
    width, heads, kv, dim, ff = SIZES[case["size"]]
    attention = width * dim * (2 * heads + 2 * kv)
    if case["model"] == "bimolix":          # retention (q, k, v, gate, out) and attention (q, k = v, gate, out) in turn
        attention = width * dim * (5 * heads + 3 * heads + kv) / 2
    return attention + 3 * width * ff


def work(case):
    width, heads, kv, dim, ff = SIZES[case["size"]]
    layers, element = case["layers"], 4 if case["dtype"] == "float32" else 2
    matrices = _layer_weights(case)
    requests = [(length, 1) for length in _lengths(case["decodes"], case["context"], case["ragged"])]
    requests += [(case["history"], length) for length in _lengths(case["prompts"], case["tokens"], case["ragged"])]
    tokens = sum(new for _, new in requests)
    window = {"qwen3": None, "gumapel": GUMAPEL_WINDOW, "bimolix": BIMOLIX_CHUNK}[case["model"]]
    pairs = held = 0
    for before, new in requests:
        if window is None:
            pairs += new * before + new * (new + 1) // 2
            held += before
        else:
            pairs += sum(min(before + i + 1, window) if case["model"] == "gumapel" else (before + i) % window + 1
                         for i in range(new))
            held += min(before, window)
    attention_layers = layers if case["model"] != "bimolix" else layers / 2
    flops = 2.0 * tokens * layers * matrices + 4.0 * attention_layers * heads * dim * pairs + 2.0 * len(requests) * width * VOCAB
    if case["model"] == "bimolix":
        flops += 4.0 * (layers / 2) * heads * dim * dim * tokens          # the state: a product in, a product out
    cache = 2.0 * attention_layers * kv * dim * element * (held + tokens)
    bytes_ = element * (layers * matrices + VOCAB * width + tokens * width) + cache + 4.0 * len(requests) * VOCAB
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    if case["dtype"] == "float32":
        # four times the 2.5e-6 by which the path is off the 64-bit values (28 layers of 32-bit sums)
        return {"rel": 1e-5}
    # bfloat16 activations and products rounded in every layer: 0.7e-2 to 2.0e-2 off the 64-bit values, and two such
    # implementations differ from one another; a token flips where two logits lie that close
    made = {"rel": 6e-2}
    if case["sampled"]:
        made["differ"] = 0.3
    return made


# -------------------------------------------------------------------------------------------- the same in 64 bits, plainly
def _weights(case, seed):
    """The engine's random weights, as it documents them: one generator, checkpoint order, N(0, 0.02) or 1 + U(-0.1, 0.1)
    in 32 bits; matrices, tables and single numbers stored in the model's type, vectors in 32 bits."""
    device = "cuda" if torch.cuda.is_available() else "cpu"
    generator = torch.Generator(device=device)
    generator.manual_seed(int(seed))
    stored = {"bfloat16": torch.bfloat16, "float32": torch.float32}[case["dtype"]]
    w = {}

    def normal(name, *shape):
        t = torch.randn(shape, generator=generator, device=device) * 0.02
        w[name] = t if len(shape) == 1 else t.to(stored)

    def around_one(name, size):
        t = torch.rand((size,), generator=generator, device=device)
        w[name] = 1.0 + (2.0 * t - 1.0) * 0.1

    width, heads, kv, dim, ff = SIZES[case["size"]]
    q, k = heads * dim, kv * dim
    if case["model"] == "qwen3":
        normal("embed", VOCAB, width)
        for i in range(case["layers"]):
            around_one(f"{i}.norm1", width)
            normal(f"{i}.q", q, width), normal(f"{i}.k", k, width), normal(f"{i}.v", k, width), normal(f"{i}.o", width, q)
            around_one(f"{i}.q.norm", dim), around_one(f"{i}.k.norm", dim), around_one(f"{i}.norm2", width)
            normal(f"{i}.gate", ff, width), normal(f"{i}.up", ff, width), normal(f"{i}.down", width, ff)
        around_one("norm", width)
        if case["size"] == "0.6b":
            w["head"] = w["embed"]
        else:
            normal("head", VOCAB, width)
        return w
    if case["model"] == "gumapel":
        normal("embed", VOCAB, width)
        for i in range(case["layers"]):
            normal(f"{i}.q", q, width), normal(f"{i}.k", k, width), normal(f"{i}.v", k, width)
            if i % 4 == 3:
                normal(f"{i}.g", q, width)
            normal(f"{i}.gate", ff, width), normal(f"{i}.up", ff, width)
            normal(f"{i}.o", width, q), normal(f"{i}.down", width, ff)
            around_one(f"{i}.norm1", width)
            w[f"{i}.vmix"] = torch.rand((), generator=generator, device=device).to(stored)
        around_one("norm", width)
        normal("head", VOCAB, width)
        return w
    normal("embed", VOCAB, width), normal("embed.norm", width)
    for i in range(case["layers"]):
        normal(f"{i}.norm1", width)
        if i % 2 == 0:
            for name in "qkvg":
                normal(f"{i}.{name}", q, width)
            normal(f"{i}.o", width, q), normal(f"{i}.norm2", width)
            normal(f"{i}.gate", ff, width), normal(f"{i}.up", ff, width), normal(f"{i}.down", width, ff)
            continue
        normal(f"{i}.q", q, width), normal(f"{i}.k", k, width), normal(f"{i}.g", q, width), normal(f"{i}.o", width, q)
        around_one(f"{i}.q.norm", dim), around_one(f"{i}.k.norm", dim)
        normal(f"{i}.q.b", q), normal(f"{i}.k.b", k), normal(f"{i}.rel", BIMOLIX_ROWS, heads), normal(f"{i}.norm2", width)
        normal(f"{i}.gate", ff, width), normal(f"{i}.up", ff, width), normal(f"{i}.down", width, ff)
    normal("norm", width), normal("head", VOCAB, width)
    return w


def _over_rms(x):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS)


def _silu(z):
    return z * torch.sigmoid(z)


def _turn(x, base, halves):
    """x [tokens, heads, dim]: pair i turns by position * base^(-2 i / dim); a pair is (i, i + dim / 2) or (2 i, 2 i + 1)."""
    tokens, _, dim = x.shape
    rate = base ** (-2.0 * torch.arange(dim // 2, dtype=x.dtype, device=x.device) / dim)
    angle = torch.arange(tokens, dtype=x.dtype, device=x.device)[:, None, None] * rate
    c, s = torch.cos(angle), torch.sin(angle)
    a, b = (x[..., :dim // 2], x[..., dim // 2:]) if halves else (x[..., 0::2], x[..., 1::2])
    turned = (a * c - b * s, b * c + a * s)
    return torch.cat(turned, -1) if halves else torch.stack(turned, -1).flatten(-2)


def _attend(q, k, v, scale, seen_by, bias=None, one_more=False):
    """q [tokens, heads, dim] over k, v [tokens, kv heads, dim], a block of queries of a head at a time; ``seen_by(i, j)``:
    whether query i sees key j; ``bias(head, i, j)`` is added to the scores; ``one_more``: the denominator holds another
    term of score 0."""
    tokens, heads, _ = q.shape
    group = heads // k.shape[1]
    out = torch.empty(tokens, heads, v.shape[2], dtype=q.dtype, device=q.device)
    j = torch.arange(tokens, device=q.device)
    block = max(1, min(tokens, (1 << 26) // tokens))
    for at in range(0, tokens, block):
        i = j[at:at + block]
        seen = seen_by(i[:, None], j[None, :])
        for h in range(heads):
            s = (q[i, h] @ k[:, h // group].T) * scale
            if bias is not None:
                s = s + bias(h, i[:, None], j[None, :])
            s = s.masked_fill(~seen, -torch.inf)
            if one_more:
                top = torch.clamp(s.amax(-1, keepdim=True), min=0.0)
                e = torch.exp(s - top)
                p = e / (torch.exp(-top) + e.sum(-1, keepdim=True))
            else:
                p = torch.softmax(s, -1)
            out[i, h] = p @ v[:, h // group]
    return out


def _qwen3(case, w, ids):
    width, heads, kv, dim, ff = SIZES[case["size"]]
    x = w("embed")[ids].double()
    tokens = x.shape[0]
    for i in range(case["layers"]):
        h = _over_rms(x) * w(f"{i}.norm1")
        q = _over_rms((h @ w(f"{i}.q").T).view(tokens, heads, dim)) * w(f"{i}.q.norm")
        k = _over_rms((h @ w(f"{i}.k").T).view(tokens, kv, dim)) * w(f"{i}.k.norm")
        v = (h @ w(f"{i}.v").T).view(tokens, kv, dim)
        o = _attend(_turn(q, ROPE_BASE, True), _turn(k, ROPE_BASE, True), v, dim ** -0.5, lambda i, j: j <= i)
        x = x + o.reshape(tokens, -1) @ w(f"{i}.o").T
        h = _over_rms(x) * w(f"{i}.norm2")
        x = x + (_silu(h @ w(f"{i}.gate").T) * (h @ w(f"{i}.up").T)) @ w(f"{i}.down").T
    return (_over_rms(x[-1]) * w("norm")) @ w("head").T


def _gumapel(case, w, ids):
    width, heads, kv, dim, ff = SIZES[case["size"]]
    x = w("embed")[ids].double()
    tokens, first = x.shape[0], None
    for i in range(case["layers"]):
        h = _over_rms(x) * w(f"{i}.norm1")
        q, k, v = ((h @ w(f"{i}.{name}").T).view(tokens, -1, dim) for name in "qkv")
        gated = i % 4 == 3
        q, k = (_over_rms(q), _over_rms(k)) if gated else (_turn(q, GUMAPEL_BASE, False), _turn(k, GUMAPEL_BASE, False))
        if first is None:
            first = v
        else:
            v = (1.0 - w(f"{i}.vmix")) * v + w(f"{i}.vmix") * first
        kept = 0 if gated else GUMAPEL_KEPT
        o = _attend(q, k, v, dim ** -0.5, lambda i, j: (j <= i) & ((i - j < GUMAPEL_WINDOW) | (j < kept))).reshape(tokens, -1)
        if gated:
            o = o * torch.sigmoid(h @ w(f"{i}.g").T)
        z = h @ w(f"{i}.gate").T
        z = 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))
        x = x + o @ w(f"{i}.o").T + (z * (h @ w(f"{i}.up").T)) @ w(f"{i}.down").T
    return (_over_rms(x[-1]) * w("norm")) @ w("head").T


def _bimolix(case, w, ids):
    width, heads, kv, dim, ff = SIZES[case["size"]]
    x = _over_rms(w("embed")[ids].double()) * (1.0 + w("embed.norm"))
    tokens = x.shape[0]
    apart = torch.arange(tokens, device=x.device)
    half = BIMOLIX_ROWS // 2
    far = torch.clamp(apart.double(), min=half) / half
    bucket = torch.where(apart < half, apart, torch.clamp(
        half + torch.floor(torch.log(far) / math.log(BIMOLIX_CHUNK / half) * (BIMOLIX_ROWS - half)).long(), max=BIMOLIX_ROWS - 1))
    for i in range(case["layers"]):
        h = _over_rms(x) * (1.0 + w(f"{i}.norm1"))
        if i % 2 == 0:
            q, k, v = ((h @ w(f"{i}.{name}").T).view(tokens, heads, dim) for name in "qkv")
            q, k = _turn(q, ROPE_BASE, True), _turn(k, ROPE_BASE, True) * dim ** -0.5
            o = torch.empty_like(v)
            distance = (apart[:, None] - apart[None, :]).double()
            for head, decay in enumerate(_decay(heads)):
                kept = torch.where(distance >= 0, decay ** distance.clamp(min=0), 0.0)
                o[:, head] = ((q[:, head] @ k[:, head].T) * kept) @ v[:, head]
            x = x + (_over_rms(o).reshape(tokens, -1) * _silu(h @ w(f"{i}.g").T)) @ w(f"{i}.o").T
        else:
            q = _over_rms((h @ w(f"{i}.q").T + w(f"{i}.q.b")).view(tokens, heads, dim)) * w(f"{i}.q.norm")
            v = (h @ w(f"{i}.k").T + w(f"{i}.k.b")).view(tokens, kv, dim)
            k = _over_rms(v) * w(f"{i}.k.norm")
            rel = w(f"{i}.rel")
            o = _attend(q, k, v, dim ** -0.5, lambda i, j: (j <= i) & (i // BIMOLIX_CHUNK == j // BIMOLIX_CHUNK),
                        lambda head, i, j: rel[bucket[(i - j).clamp(min=0)], head], one_more=True)
            x = x + (o.reshape(tokens, -1) * torch.sigmoid(h @ w(f"{i}.g").T)) @ w(f"{i}.o").T
        h = _over_rms(x) * (1.0 + w(f"{i}.norm2"))
        x = x + (_silu(h @ w(f"{i}.gate").T) * (h @ w(f"{i}.up").T)) @ w(f"{i}.down").T
    return (_over_rms(x[-1]) * (1.0 + w("norm"))) @ w("head").T


def exact(case, seed):
    stored = _weights(case, seed)
    wide = {}

    def weight(name):
        """A layer's tensors in 64 bits (the embedding as it is stored: its rows are widened)."""
        if name == "embed":
            return stored[name]
        if name not in wide:
            if sum(t.numel() for t in wide.values()) > 3 << 30:
                wide.clear()
            wide[name] = stored[name].double()
        return wide[name]

    forward = {"qwen3": _qwen3, "gumapel": _gumapel, "bimolix": _bimolix}[case["model"]]
    with torch.no_grad():
        rows = [forward(case, weight, torch.tensor(held + new, device=stored["embed"].device))
                for held, new in _requests(case, seed)]
        made = {"logits": torch.stack(rows)}
    if case["sampled"]:
        made["tokens"] = None            # drawn with the engine's own noise
    return made
