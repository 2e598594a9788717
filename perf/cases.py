"""Cases by which this engine's speed is measured, and what they must compute.

The engine is stepped the way its scheduler and its replay step it: requests are opened in the cache, brought to
``ModelRunner.step`` as prompt portions and decoded tokens, and closed.  The sizes are the shapes that ``bench.py``
knows (Qwen3 0.6B whole, eight layers of 1.7B and of 8B, four Sogodra layers and the routed experts of the Gegepel
bench), weights are the engine's random ones, token ids are uniform.  Tokens to decode are given, not sampled, so that
two versions of the code compute the same positions.

Eight layers, and a vocabulary cut in that proportion: with random weights the roundings to bfloat16 add up, and two
correct orders of summation give logits of the 8B shape that differ by 1.4 % (2-norm) after 4 layers, 2.0 % after 8,
2.4 % after 12 and about 4 % after all 36; at 0.6B it is 0.7 % whatever the depth.  Every layer runs the same kernels.

Kinds of cases:

* ``decode``: ``steps`` captured decode steps of ``batch`` requests that share nothing, on contexts of ``context``
  tokens (``ragged``: lengths spread from a quarter of it up).  The contexts are prefilled once; every pass opens its
  requests on those pages, as a prefix hit does.
* ``prompt``: one prompt of ``tokens`` tokens in portions of 2,048, logits of its last token.
* ``mixed``: one step of ``batch`` decoded tokens beside ``portion`` prompt tokens of ``prompts`` requests, the first of
  which has ``behind`` tokens in the cache already: what continuous batching runs most of the time.
* ``life``: ``batch`` requests from their prompts (lengths from half of ``prompt`` up) through ``steps`` decoded tokens.
* ``sample``: one token for each of ``rows`` rows of logits, greedy, by temperature and with top-k / top-p / min-p mixed.
* ``experts``: a step's rows through a layer of routed experts.  (Whole models with experts are left out: in bfloat16 a
  close call of a router may fall either way, and then the logits of that row are another model's.)
"""
from __future__ import annotations

import itertools
import math
import random
import zlib

import torch

from sglang_rs_b200 import Engine, ops
from sglang_rs_b200.engine.runner import StepEntry
from sglang_rs_b200.sampling import RequestRandom, Sampler, SamplingParams

PORTION = 2048                       # prompt tokens of a step
PAGE = 16
SHAPES = {
    "qwen3-0.6b": dict(num_hidden_layers=28, hidden_size=1024, num_attention_heads=16, num_key_value_heads=8, head_dim=128,
                       intermediate_size=3072, vocab_size=151936, tie_word_embeddings=True),
    "qwen3-1.7b": dict(num_hidden_layers=8, hidden_size=2048, num_attention_heads=16, num_key_value_heads=8, head_dim=128,
                       intermediate_size=6144, vocab_size=43008, tie_word_embeddings=True),
    "qwen3-8b": dict(num_hidden_layers=8, hidden_size=4096, num_attention_heads=32, num_key_value_heads=8, head_dim=128,
                     intermediate_size=12288, vocab_size=32768, tie_word_embeddings=False),
}
THETA, EPS = 1000000.0, 1e-6
SOGODRA_EPS, SOGODRA_VOCAB, SOGODRA_WIDTH = 1e-5, 32768, 2048
EXPERT_SIZES = dict(width=2048, experts=64, ff=1408, top=6)


# ---------------------------------------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest call: one user of a small model; launches and gaps between them count as much as bytes
        dict(name="decode-0.6b-b1", kind="decode", shape="qwen3-0.6b", batch=1, context=512, ragged=False, steps=8),
        # the headline: decode at batch 1, 8 and 64 behind contexts of 2,048 tokens
        dict(name="decode-8b-b1", kind="decode", shape="qwen3-8b", batch=1, context=2048, ragged=False, steps=8),
        dict(name="decode-8b-b8", kind="decode", shape="qwen3-8b", batch=8, context=2048, ragged=False, steps=8),
        # a full server: many users whose conversations have different lengths
        dict(name="decode-8b-b64", kind="decode", shape="qwen3-8b", batch=64, context=2048, ragged=True, steps=8),
        # the headline's prompt
        dict(name="prompt-8b-2048", kind="prompt", shape="qwen3-8b", tokens=2048),
        # a long document in portions, of an odd length: attention over many keys
        dict(name="prompt-1.7b-8191", kind="prompt", shape="qwen3-1.7b", tokens=8191),
        # a short prompt arrives while others decode: few hundred rows, neither weight nor arithmetic bound
        dict(name="mixed-8b-b8-p256", kind="mixed", shape="qwen3-8b", batch=8, context=2048, portion=256, prompts=1, behind=0),
        # the step of the continuous-batching workload: portions of three prompts fill the step beside 48 decoding users
        dict(name="serve-1.7b-b48", kind="mixed", shape="qwen3-1.7b", batch=48, context=2048, portion=2000, prompts=3, behind=1536),
        # the true 32-bit path, prompt and decoding: what logits are compared with
        dict(name="float32-0.6b", kind="life", shape="qwen3-0.6b", dtype="float32", batch=2, prompt=300, steps=8),
        # sampling at the server's batch
        dict(name="sample-b64", kind="sample", rows=64, vocab=151936),
        # layers over a state per request: the gated delta rule, minGRU, windowed attention, clamped feed-forwards
        dict(name="sogodra-b4", kind="life", shape="sogodra", dtype="bfloat16", batch=4, prompt=1500, steps=8),
        # a portion's rows through a layer of routed experts
        dict(name="experts-2048", kind="experts", rows=2048, **EXPERT_SIZES),
    ]


def _log(rng: random.Random, low: int, high: int) -> int:
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng: random.Random):
    kind = rng.choice(["decode", "decode", "decode", "prompt", "prompt", "mixed", "mixed", "float32", "sample", "sogodra", "experts"])
    shape = rng.choice(sorted(SHAPES))
    if kind == "decode":
        batch = _log(rng, 1, 64)
        context = PAGE * _log(rng, 1, min(256, 131072 // PAGE // batch))
        return dict(kind="decode", shape=shape, batch=batch, context=context, ragged=rng.random() < 0.7, steps=8)
    if kind == "prompt":
        return dict(kind="prompt", shape=shape, tokens=_log(rng, 9, 2048 if shape == "qwen3-8b" else 8191))
    if kind == "mixed":
        batch = _log(rng, 1, 48)
        portion = _log(rng, 8, PORTION - batch)
        return dict(kind="mixed", shape=shape, batch=batch, context=PAGE * _log(rng, 2, 128), portion=portion,
                    prompts=rng.randint(1, min(4, portion)), behind=rng.choice([0, PAGE * _log(rng, 1, 128)]))
    if kind == "float32":
        return dict(kind="life", shape="qwen3-0.6b", dtype="float32", batch=rng.randint(1, 4), prompt=_log(rng, 8, 300), steps=8)
    if kind == "sample":
        return dict(kind="sample", rows=_log(rng, 1, 64), vocab=151936)
    if kind == "sogodra":
        return dict(kind="life", shape="sogodra", dtype="bfloat16", batch=rng.randint(1, 8), prompt=_log(rng, 8, 1500), steps=8)
    return dict(kind="experts", rows=_log(rng, 1, 2048), **EXPERT_SIZES)


# ---------------------------------------------------------------------------------------------- inputs from the seed
def _sogodra_config():
    heads = SOGODRA_WIDTH // 128
    rule = {"heads": heads, "kv_heads": heads, "dim": 128, "vdim": 128, "conv": 4}
    attention = {"heads": heads, "kv_heads": heads // 4, "dim": 128, "vdim": 128, "scale": 1.0 / math.sqrt(128), "mask": {"size": 1024},
                 "rot": {"base": 50000.0, "dims": 64, "scaling": {"factor": 8.0, "low": 1.0, "high": 6.0, "original": 4096}}}
    kinds = [("delta", rule), ("parallel", {"left": attention, "right": rule, "left_scale": 0.8, "right_scale": 1.2}),
             ("mingru", {"width": SOGODRA_WIDTH}), ("delta", rule)]
    return {"architecture": "Sogodra", "vocab": SOGODRA_VOCAB, "width": SOGODRA_WIDTH, "norm": {"eps": SOGODRA_EPS},
            "layers": [{"type": kind, "mixer": mixer, "mlp": {"kind": "dense", "ff": 3 * SOGODRA_WIDTH, "limit": 7.0}}
                       for kind, mixer in kinds]}


def _config(shape: str):
    if shape == "sogodra":
        return _sogodra_config()
    return {"architectures": ["Qwen3ForCausalLM"], "model_type": "qwen3", **SHAPES[shape], "rope_theta": THETA, "rms_norm_eps": EPS,
            "max_position_embeddings": 16384, "hidden_act": "silu", "attention_bias": False}


def _vocab(case) -> int:
    return SOGODRA_VOCAB if case["shape"] == "sogodra" else SHAPES[case["shape"]]["vocab_size"]


def _lengths(case, seed: int):
    """Of a decode or mixed case: the cached tokens of every decoding request (whole pages); of a life: the prompts' lengths."""
    rng = random.Random(seed * 31 + 7)
    if case["kind"] == "life":
        return [rng.randint((case["prompt"] + 1) // 2, case["prompt"]) for _ in range(case["batch"])]
    pages = case["context"] // PAGE
    if not case.get("ragged", True):
        return [case["context"]] * case["batch"]
    return [PAGE * rng.randint(max(1, pages // 4), pages) for _ in range(case["batch"])]


def _portions(case):
    """Rows of the prompts of a mixed step: uneven shares of ``portion``."""
    left, rows = case["portion"], []
    for i in range(case["prompts"] - 1):
        rows.append(max(1, min(left - (case["prompts"] - 1 - i), left // 2 - 1)))
        left -= rows[-1]
    return rows + [left]


def _token_lists(lengths, vocab: int, seed: int):
    g = torch.Generator().manual_seed(seed * 7919 + 13)
    return [torch.randint(0, vocab, (n,), generator=g).tolist() for n in lengths]


def _sequences(case, seed: int):
    """Per request: (tokens that are in the cache before the pass, tokens of the pass)."""
    vocab = _vocab(case)
    if case["kind"] == "prompt":
        return [([], _token_lists([case["tokens"]], vocab, seed)[0])]
    lengths = _lengths(case, seed)
    if case["kind"] == "life":
        return [([], t) for t in _token_lists([n + case["steps"] for n in lengths], vocab, seed)]
    own = case["steps"] if case["kind"] == "decode" else 1
    whole = [(n, own) for n in lengths]
    if case["kind"] == "mixed":
        whole += [(case["behind"] if i == 0 else 0, n) for i, n in enumerate(_portions(case))]
    return [(t[:n], t[n:]) for (n, _), t in zip(whole, _token_lists([a + b for a, b in whole], vocab, seed))]


# ---------------------------------------------------------------------------------------------- prepare
def _packed(lists):
    """(request, first, last) pieces of at most PORTION rows together, step by step."""
    steps, room = [[]], PORTION
    for index, tokens in enumerate(lists):
        first = 0
        while first < len(tokens):
            if room == 0:
                steps.append([])
                room = PORTION
            take = min(room, len(tokens) - first)
            steps[-1].append((index, first, first + take))
            first, room = first + take, room - take
    return [step for step in steps if step]


def _prepare_engine(case, seed: int):
    sequences = _sequences(case, seed)
    # the cached contexts once, and what a pass writes beside them
    tokens = sum(len(a) + 2 * len(b) + 2 * PAGE for a, b in sequences)
    engine = Engine(config=_config(case["shape"]), random_weights=True, seed=seed, dtype=case.get("dtype", "bfloat16"), page_size=PAGE,
                    max_total_tokens=tokens + PORTION, max_running_requests=2 * len(sequences) + 2, chunked_prefill_size=PORTION,
                    disable_radix_cache=True)        # the pass opens requests on its pages itself
    state = dict(case=case, engine=engine, own=[own for _, own in sequences], names=itertools.count(), pages=[None] * len(sequences))
    cached = [tokens for tokens, _ in sequences]
    if any(cached):
        handles = [engine.cache.open(f"context-{i}") if t else None for i, t in enumerate(cached)]
        for step in _packed(cached):
            engine.runner.step([StepEntry(handles[i], cached[i][a:b], []) for i, a, b in step])
        state["pages"] = [h.table(("kv", None)) if h else None for h in handles]
        state["contexts"] = handles              # they hold the pages
    return state


def _prepare_sample(case, seed: int):
    g = torch.Generator(device="cuda").manual_seed(seed)
    logits = torch.randn((case["rows"], case["vocab"]), generator=g, device="cuda") * 2.5
    kinds = [dict(), dict(temperature=0.7), dict(temperature=0.8, top_k=50, top_p=0.95), dict(temperature=1.0, top_p=0.9, min_p=0.05)]
    return dict(case=case, logits=logits, sampler=Sampler(logits.device, case["vocab"]),
                params=[SamplingParams(**kinds[r % 4]) for r in range(case["rows"])],
                randoms=[RequestRandom(r, seed * 1000 + r) for r in range(case["rows"])], ids=list(range(case["rows"])))


def _expert_tensors(case, seed: int):
    g = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape, std=0.02):
        return (torch.randn(shape, generator=g, device="cuda") * std).to(torch.bfloat16)
    width, experts, ff = case["width"], case["experts"], case["ff"]
    return dict(h=normal(case["rows"], width, std=1.0), router=normal(experts, width), up=normal(experts, 2 * ff, width),
                down=normal(experts, width, ff))


def prepare(case, seed):
    if case["kind"] == "sample":
        return _prepare_sample(case, seed)
    if case["kind"] == "experts":
        return dict(case=case, error=ops.new_error_word("cuda"), **_expert_tensors(case, seed))
    return _prepare_engine(case, seed)


# ---------------------------------------------------------------------------------------------- one pass
def _open(state):
    """The pass's requests, on the cached pages where they have some."""
    cache, handles = state["engine"].cache, []
    for pages in state["pages"]:
        handle = cache.open(f"pass-{next(state['names'])}")
        if pages is not None:
            cache.adopt_prefix(handle, ("kv", None), pages)
        handles.append(handle)
    return handles


def run(state):
    case = state["case"]
    if case["kind"] == "sample":
        return state["sampler"].pick_on_device(state["logits"], state["params"], state["randoms"], state["ids"])
    if case["kind"] == "experts":
        return ops.routed_experts(state["h"], state["router"], state["up"], state["down"], case["top"], "silu", False, state["error"])
    step, own, outputs = state["engine"].runner.step, state["own"], []
    handles = _open(state)
    if case["kind"] == "mixed":
        outputs.append(step([StepEntry(h, t, [len(t) - 1]) for h, t in zip(handles, own)]))
        done = [len(t) for t in own]
    elif case["kind"] == "decode":
        done = [0] * len(own)
    else:
        # prompts, in steps of at most PORTION rows; every request's last prompt row gives logits
        done = [len(t) - case.get("steps", 0) for t in own]
        for pieces in _packed([t[:n] for t, n in zip(own, done)]):
            logits = step([StepEntry(handles[i], own[i][a:b], [b - a - 1] if b == done[i] else []) for i, a, b in pieces])
            if logits is not None:
                outputs.append(logits.clone())
    for i in range(case.get("steps", 0)):
        # a captured step writes its logits where the next one will: they are taken along, as a sampler would take tokens
        outputs.append(step([StepEntry(h, [t[n + i]], [0]) for h, t, n in zip(handles, own, done)]).clone())
    for handle in handles:
        state["engine"].cache.close(handle)
    return outputs


# ---------------------------------------------------------------------------------------------- what a pass cannot do without
def _matrix_sizes(case):
    """(entries of the matrices that every row passes, entries of the head, kv entries per token, attention width) of a model."""
    if case["shape"] == "sogodra":
        w = SOGODRA_WIDTH
        delta, mlp = 5 * w * w + 2 * 16 * w, 9 * w * w
        parallel = (2 * w * w + 2 * (w // 4) * w) + (4 * w * w + 4 * 128 * w + 16 * w)
        return 2 * delta + parallel + 4 * w * w + 4 * mlp, SOGODRA_VOCAB * w, 2 * (w // 4), w
    s = SHAPES[case["shape"]]
    q, kv, h = s["num_attention_heads"] * s["head_dim"], s["num_key_value_heads"] * s["head_dim"], s["hidden_size"]
    layer = (q + 2 * kv) * h + h * q + 3 * s["intermediate_size"] * h
    return s["num_hidden_layers"] * layer, s["vocab_size"] * h, s["num_hidden_layers"] * 2 * kv, s["num_hidden_layers"] * q


def work(case):
    if case["kind"] == "sample":
        return {"bytes": 4.0 * case["rows"] * case["vocab"] + 4 * case["rows"], "flops": 0.0}
    if case["kind"] == "experts":
        used = min(case["experts"], case["rows"] * case["top"])
        entry = 3 * case["width"] * case["ff"]
        return {"bytes": 2.0 * used * entry + case["rows"] * case["width"] * 6.0, "flops": 2.0 * case["rows"] * case["top"] * entry}
    body, head, kv, attention = _matrix_sizes(case)
    size = 4 if case.get("dtype") == "float32" else 2
    sequences = [(len(a), len(b)) for a, b in _sequences(case, 1)]
    rows = sum(b for _, b in sequences)
    pairs = sum(b * a + b * (b + 1) / 2 for a, b in sequences)                 # (query, visible key)
    if case["shape"] == "sogodra":
        pairs = sum(sum(min(i + 1, 1024) for i in range(b)) for _, b in sequences)
    logit_rows = case.get("steps", 0) * len(sequences) + (0 if case["kind"] == "decode" else len(sequences))
    # a decode step reads every matrix and all keys of its requests; the prompts of a pass read the matrices once
    steps = case.get("steps", 0) + (0 if case["kind"] == "decode" else 1)
    kv_reads = kv * sum(a for a, _ in sequences) * (case["steps"] if case["kind"] == "decode" else 1)
    if case["kind"] == "life":
        kv_reads = kv * sum(min(b, 1024) if case["shape"] == "sogodra" else b for _, b in sequences) * case["steps"]
    return {"bytes": float(size) * (steps * (body + head) + kv_reads + kv * rows) + 4.0 * logit_rows * _vocab(case),
            "flops": 2.0 * rows * body + 2.0 * logit_rows * head + 4.0 * attention * pairs}


def tolerance(case):
    if case["kind"] == "sample":
        return "exact"
    if case["kind"] == "experts":
        return {"rel": 1e-2}
    return {"rel": 1e-4} if case.get("dtype") == "float32" else {"rel": 3e-2}


# ---------------------------------------------------------------------------------------------- the same in 64 bits
D = torch.float64


class _Weights:
    """The random-weights mode's tensors: N(0, 0.02) or 1 + U(-0.1, 0.1) from the seed and the tensor's name."""

    def __init__(self, seed: int, dtype: torch.dtype):
        self.seed, self.dtype = seed, dtype

    def _generator(self, name: str):
        return torch.Generator(device="cuda").manual_seed((int(self.seed) * 1_000_003 + zlib.crc32(name.encode("utf-8"))) % (2 ** 63 - 1))

    def normal(self, name: str, *shape) -> torch.Tensor:
        values = torch.randn(shape, generator=self._generator(name), device="cuda", dtype=torch.float32) * 0.02
        return values.to(self.dtype).to(D)           # vectors and convolution taps too are drawn in the compute type

    def scale(self, name: str, width: int) -> torch.Tensor:
        values = torch.rand((width,), generator=self._generator(name), device="cuda", dtype=torch.float32)
        return (1.0 + (values * 2 - 1) * 0.1).to(D)


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _turn(x, rates):
    """x [tokens, heads, dim] from position 0: the leading 2 * len(rates) entries turned in half-split pairs."""
    half = rates.numel()
    angle = (torch.arange(x.shape[0], device=x.device, dtype=D)[:, None] * rates[None, :])[:, None, :]
    a, b = x[..., :half], x[..., half:2 * half]
    return torch.cat([a * angle.cos() - b * angle.sin(), b * angle.cos() + a * angle.sin(), x[..., 2 * half:]], -1)


def _attend(q, k, v, scale, window=None, sink=None):
    """q [tokens, heads, dim], k and v [tokens, kv heads, dim] of one sequence."""
    tokens, heads, groups = q.shape[0], q.shape[1], k.shape[1]
    out = torch.empty_like(q)
    at = torch.arange(tokens, device=q.device)
    for first in range(0, tokens, 2048):
        rows = at[first:first + 2048]
        low = 0 if window is None else max(0, first - window + 1)
        keys = at[low:rows[-1] + 1]
        hidden = keys[None, :] > rows[:, None]
        if window is not None:
            hidden |= keys[None, :] <= rows[:, None] - window
        for head in range(heads):
            g = head // (heads // groups)
            s = (q[rows, head] @ k[keys, g].T * scale).masked_fill(hidden, float("-inf"))
            if sink is not None:
                s = torch.cat([s, sink[head].expand(s.shape[0], 1)], 1)
            out[rows, head] = torch.softmax(s, -1)[:, :keys.numel()] @ v[keys, g]
    return out


def _qwen3_exact(case, seed: int, sequences, wanted):
    s, w = SHAPES[case["shape"]], _Weights(seed, torch.float32 if case.get("dtype") == "float32" else torch.bfloat16)
    h, heads, kv, d, ff = (s[k] for k in ("hidden_size", "num_attention_heads", "num_key_value_heads", "head_dim", "intermediate_size"))
    bounds = list(itertools.accumulate([0] + [len(t) for t in sequences]))
    embed = w.normal("model.embed_tokens.weight", s["vocab_size"], h)
    x = embed[torch.tensor([t for tokens in sequences for t in tokens], device="cuda")]
    if not s["tie_word_embeddings"]:
        embed = None
    # the model's table of frequencies is a 32-bit constant
    rates = torch.pow(torch.tensor(THETA, dtype=D), -2.0 * torch.arange(d // 2, dtype=D) / d).to(torch.float32).to("cuda", D)
    for i in range(s["num_hidden_layers"]):
        p = f"model.layers.{i}."
        y = _rms(x, EPS) * w.scale(p + "input_layernorm.weight", h)
        q = (y @ w.normal(p + "self_attn.q_proj.weight", heads * d, h).T).view(-1, heads, d)
        k = (y @ w.normal(p + "self_attn.k_proj.weight", kv * d, h).T).view(-1, kv, d)
        v = (y @ w.normal(p + "self_attn.v_proj.weight", kv * d, h).T).view(-1, kv, d)
        q = _rms(q, EPS) * w.scale(p + "self_attn.q_norm.weight", d)
        k = _rms(k, EPS) * w.scale(p + "self_attn.k_norm.weight", d)
        y = torch.cat([_attend(_turn(q[a:b], rates), _turn(k[a:b], rates), v[a:b], d ** -0.5) for a, b in zip(bounds, bounds[1:])])
        x = x + y.view(-1, heads * d) @ w.normal(p + "self_attn.o_proj.weight", h, heads * d).T
        y = _rms(x, EPS) * w.scale(p + "post_attention_layernorm.weight", h)
        gate = y @ w.normal(p + "mlp.gate_proj.weight", ff, h).T
        y = torch.nn.functional.silu(gate) * (y @ w.normal(p + "mlp.up_proj.weight", ff, h).T)
        x = x + y @ w.normal(p + "mlp.down_proj.weight", h, ff).T
    rows = [bounds[i] + at for i, at in wanted]
    y = _rms(x[torch.tensor(rows, device="cuda")], EPS) * w.scale("model.norm.weight", h)
    return y @ (embed if embed is not None else w.normal("lm_head.weight", s["vocab_size"], h)).T


def _sogodra_rates(rot):
    i = torch.arange(rot["dims"] // 2, dtype=D)
    f, s = rot["base"] ** (-2.0 * i / rot["dims"]), rot["scaling"]
    wave = 2.0 * math.pi / f
    ramp = ((s["original"] / wave - s["low"]) / (s["high"] - s["low"])).clamp(0.0, 1.0)
    return ((1.0 - ramp) * f / s["factor"] + ramp * f).to(torch.float32).to("cuda", D)


def _delta_exact(x, w, p, m, channels: bool):
    """The gated delta rule over one sequence x [tokens, width]: S <- decay S, u = beta (v - S^T k), S <- S + k u^T, o = S^T q."""
    heads, d, width, tokens = m["heads"], m["dim"], x.shape[1], x.shape[0]

    def mixed(name):
        u = torch.cat([x.new_zeros(m["conv"] - 1, heads * d), x @ w.normal(p + name, heads * d, width).T])
        taps = w.normal(p + name + ".conv", heads * d, m["conv"])
        return torch.nn.functional.silu(sum(u[j:j + tokens] * taps[:, j] for j in range(m["conv"]))).view(tokens, heads, d)

    def unit(z):
        return z / torch.sqrt((z * z).sum(-1, keepdim=True) + 1e-6)
    q, k, v = unit(mixed("q")) * d ** -0.5, unit(mixed("k")), mixed("v")
    beta = torch.sigmoid(x @ w.normal(p + "b", heads, width).T)
    a_log = w.normal(p + "A_log", heads)
    if channels:
        z = (x @ w.normal(p + "a1", d, width).T) @ w.normal(p + "a2", heads * d, d).T + w.normal(p + "dt_bias", heads * d)
        decay = torch.exp(-torch.exp(a_log)[None, :, None] * torch.nn.functional.softplus(z).view(tokens, heads, d))
        gate = torch.sigmoid((x @ w.normal(p + "g1", d, width).T) @ w.normal(p + "g2", heads * d, d).T)
    else:
        z = x @ w.normal(p + "a", heads, width).T + w.normal(p + "dt_bias", heads)
        decay = torch.exp(-torch.exp(a_log) * torch.nn.functional.softplus(z))[:, :, None].expand(tokens, heads, d)
        gate = torch.nn.functional.silu(x @ w.normal(p + "g", heads * d, width).T)
    state, o = x.new_zeros(heads, d, d), torch.empty_like(v)
    for t in range(tokens):
        state = decay[t][:, :, None] * state
        u = beta[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", state, k[t]))
        state = state + k[t][:, :, None] * u[:, None, :]
        o[t] = torch.einsum("hdv,hd->hv", state, q[t])
    y = (_rms(o, SOGODRA_EPS) * w.scale(p + "norm", d)).reshape(tokens, heads * d) * gate
    return y @ w.normal(p + "o", width, heads * d).T


def _sogodra_exact(case, seed: int, sequences, wanted):
    w, config, width = _Weights(seed, torch.bfloat16), _sogodra_config(), SOGODRA_WIDTH
    embed = w.normal("embed", SOGODRA_VOCAB, width)
    xs = [embed[torch.tensor(tokens, device="cuda")] for tokens in sequences]
    for i, layer in enumerate(config["layers"]):
        p, m = f"l{i}.mix.", layer["mixer"]
        for n, x in enumerate(xs):
            if layer["type"] == "delta":
                y = _delta_exact(x, w, p, m, False)
            elif layer["type"] == "mingru":
                z = torch.sigmoid(x @ w.normal(p + "z", width, width).T + w.normal(p + "z.b", width))
                u = x @ w.normal(p + "x", width, width).T + w.normal(p + "x.b", width)
                u = torch.where(u >= 0, u + 0.5, torch.sigmoid(u))
                state, states = torch.zeros_like(z[0]), []
                for t in range(x.shape[0]):
                    state = (1.0 - z[t]) * state + z[t] * u[t]
                    states.append(state)
                y = torch.stack(states) * torch.nn.functional.silu(x @ w.normal(p + "g", width, width).T)
                y = y @ w.normal(p + "o", width, width).T
            else:
                a, at = m["left"], p + "left."
                q = (x @ w.normal(at + "q", a["heads"] * 128, width).T).view(-1, a["heads"], 128)
                k = (x @ w.normal(at + "k", a["kv_heads"] * 128, width).T).view(-1, a["kv_heads"], 128)
                v = (x @ w.normal(at + "v", a["kv_heads"] * 128, width).T).view(-1, a["kv_heads"], 128)
                rates = _sogodra_rates(a["rot"])
                q = _turn(_rms(q, SOGODRA_EPS) * w.scale(at + "q.norm", 128), rates)
                k = _turn(_rms(k, SOGODRA_EPS) * w.scale(at + "k.norm", 128), rates)
                sink = w.normal(at + "sink", a["heads"])
                y = _attend(q, k, v, a["scale"], a["mask"]["size"], sink).reshape(-1, a["heads"] * 128)
                y = m["left_scale"] * (y @ w.normal(at + "o", width, a["heads"] * 128).T)
                y = y + m["right_scale"] * _delta_exact(x, w, p + "right.", m["right"], True)
            x = x + _rms(y, SOGODRA_EPS) * w.scale(f"l{i}.norm1", width)
            f, ff, limit = f"l{i}.mlp.", layer["mlp"]["ff"], layer["mlp"]["limit"]
            g = (x @ w.normal(f + "gate", ff, width).T).clamp(max=limit)
            u = (x @ w.normal(f + "up", ff, width).T).clamp(-limit, limit)
            y = (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ w.normal(f + "down", width, ff).T
            xs[n] = x + _rms(y, SOGODRA_EPS) * w.scale(f"l{i}.norm2", width)
    y = torch.stack([xs[i][at] for i, at in wanted])
    return (_rms(y, SOGODRA_EPS) * w.scale("final.norm", width)) @ w.normal("head", SOGODRA_VOCAB, width).T


def _experts_exact(case, seed: int):
    t = {name: value.to(D) for name, value in _expert_tensors(case, seed).items()}
    scores = torch.softmax(t["h"] @ t["router"].T, -1)
    chosen = torch.topk(scores, case["top"], -1).indices
    out = torch.zeros_like(t["h"])
    for e in range(case["experts"]):
        rows = (chosen == e).any(-1).nonzero()[:, 0]
        z = t["h"][rows] @ t["up"][e].T
        y = (torch.nn.functional.silu(z[:, :case["ff"]]) * z[:, case["ff"]:]) @ t["down"][e].T
        out[rows] += scores[rows, e][:, None] * y
    return out


def exact(case, seed):
    if case["kind"] == "sample":
        return None                                  # whole numbers
    if case["kind"] == "experts":
        return _experts_exact(case, seed)
    sequences = _sequences(case, seed)
    rows = sum(len(a) + len(b) for a, b in sequences)
    if rows * _matrix_sizes(case)[0] > 2.5e14:
        return None                                  # tens of seconds in 64 bits
    # (request, position) of every row of logits, output by output
    outputs, steps = [], case.get("steps", 0)
    if case["kind"] == "mixed":
        outputs.append([(i, len(a) + len(b) - 1) for i, (a, b) in enumerate(sequences)])
    elif case["kind"] != "decode":
        ends = [len(b) - steps for _, b in sequences]
        for pieces in _packed([b[:n] for (_, b), n in zip(sequences, ends)]):
            rows_of_step = [(i, b - 1) for i, _, b in pieces if b == ends[i]]
            if rows_of_step:
                outputs.append(rows_of_step)
    for i in range(steps):
        outputs.append([(r, len(a) + len(b) - steps + i) for r, (a, b) in enumerate(sequences)])
    compute = _sogodra_exact if case["shape"] == "sogodra" else _qwen3_exact
    logits = compute(case, seed, [a + b for a, b in sequences], [place for places in outputs for place in places])
    return list(torch.split(logits, [len(places) for places in outputs]))
