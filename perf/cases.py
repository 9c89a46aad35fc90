"""What the speed of this library is measured on: the work that its users have it do with the models of its
benchmark, through `Engine.step` (the one way tokens reach a model) and the device sampler.

Three kinds of pass:

* ``decode``   one token for each sequence of a running batch, whose prompts lie in the cache: what a generation
               loop does hundreds of times a request.
* ``request``  prompts of unequal length into fresh slots (whole, or ``chunk`` tokens of each per step), then ``new``
               further tokens of each, one step after another, and the slots given back: time to the first token
               where ``new`` is 0, a short request or a trace replay where it is not.
* ``sample``   the choice of the next token from a batch's logits, with the filters of the default sampler.

The models are the shapes of Llama 3.2 1B and 3B and of Llama 3.1 8B and the two tiny ones of the tests, with random
weights as the benchmark has them.  A program loads a model once and then serves requests, so the engine and its
weights are kept between states; tokens, prompts and what the cache holds are made from the state's seed.
"""
import functools
import math
import random

import torch

from dlgo_b200.config import config_from_dict
from dlgo_b200.engine.engine import Engine
from dlgo_b200.sampling.sampler import DeviceSampler, SamplerConfig


def _llama3(factor, original=8192):
    return dict(rope_type="llama3", factor=factor, low_freq_factor=1.0, high_freq_factor=4.0,
                original_max_position_embeddings=original)


def _model(hidden, layers, ffn, heads, kv_heads, head_dim, vocab, theta, scaling, eps, positions, tied):
    return dict(architectures=["LlamaForCausalLM"], hidden_size=hidden, num_hidden_layers=layers, intermediate_size=ffn,
                num_attention_heads=heads, num_key_value_heads=kv_heads, head_dim=head_dim, vocab_size=vocab,
                rope_theta=theta, rope_scaling=scaling, rms_norm_eps=eps, max_position_embeddings=positions,
                tie_word_embeddings=tied)


MODELS = {
    "tiny_a": _model(64, 2, 160, 4, 2, 16, 256, 1e4, None, 1e-5, 128, True),
    "tiny_b": _model(96, 3, 256, 3, 1, 32, 384, 5e5, _llama3(4.0, 64), 1e-6, 256, False),
    "1b": _model(2048, 16, 8192, 32, 8, 64, 128256, 5e5, _llama3(32.0), 1e-5, 131072, True),
    "3b": _model(3072, 28, 8192, 24, 8, 128, 128256, 5e5, _llama3(32.0), 1e-5, 131072, True),
    "8b": _model(4096, 32, 14336, 32, 8, 128, 128256, 5e5, _llama3(8.0), 1e-5, 131072, False),
}
WEIGHT_SEEDS = {"tiny_a": 0, "tiny_b": 1, "1b": 2, "3b": 4, "8b": 5}
# positions that live sequences may hold together
CACHE_TOKENS = {"tiny_a": 1 << 14, "tiny_b": 1 << 14, "1b": 400_000, "3b": 150_000, "8b": 270_000}
NEW_TOKENS = 768        # a sequence of a running batch ends after as many new tokens, and the batch's next prompts begin


def listed():
    return [
        # the smallest calls: a tiny model in 32 bits, three unequal prompts and 16 steps; launches and host time are all of it
        dict(name="request_tiny_a_f32", kind="request", model="tiny_a", dtype="float32", prompts=3, low=5, high=32, lengths=1,
             chunk=0, new=16),
        # the exact path at a real size: a trace replay of two short odd prompts and eight steps in 32 bits
        dict(name="request_1b_f32", kind="request", model="1b", dtype="float32", prompts=2, low=65, high=301, lengths=2,
             chunk=0, new=8),
        # time to the first token of a chat message
        dict(name="prompt_1b_117", kind="request", model="1b", dtype="bfloat16", prompts=1, low=117, high=117, lengths=0,
             chunk=0, new=0),
        # the benchmark's prompt
        dict(name="prompt_1b_2048", kind="request", model="1b", dtype="bfloat16", prompts=1, low=2048, high=2048, lengths=0,
             chunk=0, new=0),
        # what a batch of eight requests begins with, at the largest model: unequal prompts, packed
        dict(name="prompt_8b_batch8", kind="request", model="8b", dtype="bfloat16", prompts=8, low=128, high=1024, lengths=3,
             chunk=0, new=0),
        # the benchmark's decode steps: one conversation, a small batch, a full batch
        dict(name="decode_1b_b1", kind="decode", model="1b", dtype="bfloat16", prompts=1, low=128, high=1024, lengths=3),
        dict(name="decode_1b_b8", kind="decode", model="1b", dtype="bfloat16", prompts=8, low=128, high=1024, lengths=3),
        dict(name="decode_1b_b64", kind="decode", model="1b", dtype="bfloat16", prompts=64, low=128, high=1024, lengths=3),
        # two long documents being asked about
        dict(name="decode_1b_long", kind="decode", model="1b", dtype="bfloat16", prompts=2, low=14001, high=17777, lengths=6),
        # the larger models' serving batches
        dict(name="decode_3b_b16", kind="decode", model="3b", dtype="bfloat16", prompts=16, low=64, high=2048, lengths=4),
        dict(name="decode_8b_b32", kind="decode", model="8b", dtype="bfloat16", prompts=32, low=256, high=4096, lengths=5),
        # the default sampler's choice for a full batch
        dict(name="sample_b64", kind="sample", rows=64, vocab=128256, temperature=0.7, top_k=40, top_p=0.9, penalty=1.1),
    ]


def _between(rng, low, high):
    """A whole number of [low, high], spread over the logarithm."""
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high + 0.5))))))


def draw(rng):
    kind = rng.choices(["decode", "request", "short_request", "exact", "tiny", "sample"], [34, 24, 12, 8, 12, 10])[0]
    lengths = rng.randrange(1 << 20)
    if kind == "sample":
        return dict(kind="sample", rows=_between(rng, 1, 64), vocab=_between(rng, 32000, 128256),
                    temperature=round(rng.uniform(0.5, 1.2), 2), top_k=rng.choice([0, 20, 40, 100]),
                    top_p=rng.choice([0.9, 0.95, 1.0]), penalty=rng.choice([1.0, 1.1]))
    if kind == "tiny":
        model = rng.choice(["tiny_a", "tiny_b"])
        high = _between(rng, 2, 100)
        return dict(kind="request", model=model, dtype=rng.choice(["float32", "bfloat16"]), prompts=_between(rng, 1, 8),
                    low=max(1, high // 4), high=high, lengths=lengths, chunk=rng.choice([0, 0, 7]), new=rng.randrange(0, 25))
    if kind == "exact":
        high = _between(rng, 8, 400)
        return dict(kind="request", model="1b", dtype="float32", prompts=_between(rng, 1, 4), low=max(1, high // 3), high=high,
                    lengths=lengths, chunk=0, new=rng.randrange(0, 9))
    model = rng.choices(["1b", "3b", "8b"], [60, 20, 20])[0]
    if kind == "decode":
        most, room = {"1b": (64, 60_000), "3b": (32, 30_000), "8b": (32, 50_000)}[model]     # sequences, prompt tokens of all
        prompts = _between(rng, 1, most)
        high = _between(rng, 64, max(64, min(17_000 if model == "1b" else 4096, room // prompts)))
        return dict(kind="decode", model=model, dtype="bfloat16", prompts=prompts, low=max(1, int(high * rng.uniform(0.1, 1.0))),
                    high=high, lengths=lengths)
    total = _between(rng, 16, 512) if kind == "short_request" else _between(rng, 400, {"1b": 16_000, "3b": 8000, "8b": 4000}[model])
    prompts = min(8, _between(rng, 1, max(1, total // 16)))
    high = max(2, total // prompts)
    return dict(kind="request", model=model, dtype="bfloat16", prompts=prompts,
                low=max(1, int(high * rng.uniform(0.2, 1.0))) if prompts > 1 else high, high=high, lengths=lengths,
                chunk=rng.choice([0, 0, 0, 1024]) if kind == "request" else 0,
                new=0 if kind == "request" else rng.choice([0, 0, 0, 4, 12]))


# ---------------------------------------------------------------------------------------------- inputs
def _weights(model, dtype):
    """The model's tensors by name on the GPU: N(0, 0.02), norms 1 + N(0, 0.02)."""
    m = MODELS[model]
    g = torch.Generator(device="cuda").manual_seed(WEIGHT_SEEDS[model])
    d, f, hd = m["hidden_size"], m["intermediate_size"], m["head_dim"]
    q, kv = m["num_attention_heads"] * hd, m["num_key_value_heads"] * hd

    def rand(*shape, mean=0.0):
        return torch.empty(shape, device="cuda", dtype=torch.float32).normal_(mean, 0.02, generator=g).to(dtype)

    w = {"model.embed_tokens.weight": rand(m["vocab_size"], d), "model.norm.weight": rand(d, mean=1.0)}
    if not m["tie_word_embeddings"]:
        w["lm_head.weight"] = rand(m["vocab_size"], d)
    for i in range(m["num_hidden_layers"]):
        p = "model.layers.%d." % i
        for name, shape in (("self_attn.q_proj", (q, d)), ("self_attn.k_proj", (kv, d)), ("self_attn.v_proj", (kv, d)),
                            ("self_attn.o_proj", (d, q)), ("mlp.gate_proj", (f, d)), ("mlp.up_proj", (f, d)),
                            ("mlp.down_proj", (d, f))):
            w[p + name + ".weight"] = rand(*shape)
        for name in ("input_layernorm", "post_attention_layernorm"):
            w[p + name + ".weight"] = rand(d, mean=1.0)
    return w


@functools.lru_cache(maxsize=2)
def _engine(model, dtype):
    kind = torch.float32 if dtype == "float32" else torch.bfloat16
    tokens = CACHE_TOKENS[model] if dtype == "bfloat16" or model.startswith("tiny") else CACHE_TOKENS[model] // 4
    return Engine(dtype=dtype, max_tokens=tokens, spec=config_from_dict(MODELS[model]).architecture_spec(),
                  tensors=_weights(model, kind))


def _lengths(case):
    r = random.Random(case["lengths"])
    return [r.randint(case["low"], case["high"]) for _ in range(case["prompts"])]


def _tokens(case, seed, new):
    """Prompts and the tokens that follow them, as a program holds them: lists of ids."""
    g = torch.Generator().manual_seed(seed)
    vocab = MODELS[case["model"]]["vocab_size"]
    prompts = [torch.randint(0, vocab, (n,), generator=g).tolist() for n in _lengths(case)]
    follow = torch.randint(0, vocab, (new, case["prompts"]), generator=g).tolist()
    return prompts, follow


class _Batch:
    """A running batch: sequences with their prompts in the cache, which take one token a step."""

    def __init__(self, case, seed):
        self.engine = _engine(case["model"], case["dtype"])
        self.prompts, self.follow = _tokens(case, seed, NEW_TOKENS)
        self.slots = []
        self.begin()
        # the first step of a batch size is recorded once per engine; a program has that behind it
        self.step()
        self.close()
        self.begin()

    def begin(self):
        self.slots = [self.engine.take_slot() for _ in self.prompts]
        self.engine.step(self.slots, self.prompts)
        self.done = 0

    def step(self):
        if self.done == len(self.follow):
            self.close()
            self.begin()
        tokens = [[t] for t in self.follow[self.done]]
        self.done += 1
        return self.engine.step(self.slots, tokens)

    def close(self):
        for s in self.slots:
            self.engine.free_slot(s)
        self.slots = []

    def __del__(self):
        self.close()


class _Request:
    """Prompts into fresh slots, then given tokens step by step."""

    def __init__(self, case, seed):
        self.engine = _engine(case["model"], case["dtype"])
        self.prompts, self.follow = _tokens(case, seed, case["new"])
        self.chunk = case["chunk"]
        if case["new"]:
            self.step()         # the first step of a batch size is recorded once per engine

    def step(self):
        eng, out = self.engine, []
        slots = [eng.take_slot() for _ in self.prompts]
        if not self.chunk:
            out.append(eng.step(slots, self.prompts))
        else:
            for at in range(0, max(map(len, self.prompts)), self.chunk):
                part = [(s, p[at:at + self.chunk], len(p) <= at + self.chunk) for s, p in zip(slots, self.prompts) if len(p) > at]
                logits = eng.step([s for s, _, _ in part], [t for _, t, _ in part],
                                  [[len(t) - 1] if last else [] for _, t, last in part])
                if logits is not None:
                    out.append(logits.clone())      # a step of one token each returns the engine's own buffer
        for tokens in self.follow:
            out.append(eng.step(slots, [[t] for t in tokens]).clone())
        for s in slots:
            eng.free_slot(s)
        return out[0] if len(out) == 1 else torch.cat(out)


class _Sample:
    """Logits as a trained model leaves them: a broad floor and a few candidates above it."""

    def __init__(self, case, seed):
        g = torch.Generator(device="cuda").manual_seed(seed)
        rows, vocab = case["rows"], case["vocab"]
        self.logits = torch.randn(rows, vocab, generator=g, device="cuda") * 2.5
        at = torch.randint(0, vocab, (rows, 24), generator=g, device="cuda")
        self.logits.scatter_(1, at, torch.rand(rows, 24, generator=g, device="cuda") * 8 + 9)
        self.recent = torch.cat([at[:, :8], torch.randint(0, vocab, (rows, 56), generator=g, device="cuda")], 1).tolist()
        self.config = SamplerConfig(temperature=case["temperature"], top_k=case["top_k"], top_p=case["top_p"],
                                    repetition_penalty=case["penalty"])
        self.sampler = DeviceSampler(seed)
        self.requests, self.draws = list(range(rows)), [(seed + 3 * i) % 251 for i in range(rows)]

    def step(self):
        return self.sampler.sample(self.logits, self.config, self.requests, self.draws, self.recent)


def prepare(case, seed):
    return {"decode": _Batch, "request": _Request, "sample": _Sample}[case["kind"]](case, seed)


def run(state):
    return state.step()


# ------------------------------------------------------------------------------------- work and exactness
def work(case):
    if case["kind"] == "sample":
        n = case["rows"] * case["vocab"]
        return {"bytes": 4 * n + case["rows"] * 260, "flops": 2 * n}
    m = MODELS[case["model"]]
    size = 4 if case["dtype"] == "float32" else 2
    d, f, hd, layers, vocab = m["hidden_size"], m["intermediate_size"], m["head_dim"], m["num_hidden_layers"], m["vocab_size"]
    hq, hkv = m["num_attention_heads"], m["num_key_value_heads"]
    per_layer = d * (hq + 2 * hkv) * hd + hq * hd * d + 3 * d * f
    cache = 2 * layers * hkv * hd * size            # keys and values of one position
    lens = _lengths(case)
    n = len(lens)

    def step(contexts, brought, wanted):
        """One step: the weights once, what the attention reads and writes of the cache, the logits."""
        tokens = sum(brought)
        byte = (layers * (per_layer + 2 * d) + d + vocab * d) * size + min(tokens, vocab) * d * size
        byte += cache * sum(c + t for c, t in zip(contexts, brought)) + 4 * wanted * vocab
        pairs = sum(t * c + t * (t + 1) // 2 for c, t in zip(contexts, brought))
        return byte, 2 * layers * tokens * per_layer + 2 * wanted * d * vocab + 4 * layers * hq * hd * pairs

    if case["kind"] == "decode":
        b, fl = step(lens, [1] * n, n)
        return {"bytes": b, "flops": fl}
    total = [0, 0]
    chunk = case["chunk"] or max(lens)
    for at in range(0, max(lens), chunk):
        part = [(at, min(chunk, ln - at)) for ln in lens if ln > at]
        b, fl = step([c for c, _ in part], [t for _, t in part], sum(1 for ln in lens if at < ln <= at + chunk))
        total = [total[0] + b, total[1] + fl]
    for k in range(case["new"]):
        b, fl = step([ln + k for ln in lens], [1] * n, n)
        total = [total[0] + b, total[1] + fl]
    return {"bytes": total[0], "flops": total[1]}


def tolerance(case):
    if case["kind"] == "sample":
        return "exact"
    if case["dtype"] == "float32":
        # measured against 64 bits: 2e-7 at the tiny sizes, 8e-6 at 1b, whose sums run over up to 8192 products
        return {"rel": 1e-6} if case["model"].startswith("tiny") else {"rel": 3e-5}
    # measured: two runs of the same step differ by 0.006 to 0.012 (the order of bfloat16 products' sums over 16 to 32
    # layers), and a step is 0.013 to 0.043 away from 64 bits
    return {"rel": 0.03}


def _exact_logits(case, w, tokens, places):
    """Logits in 64 bits of one whole sequence at some places: [places, vocab]."""
    m = MODELS[case["model"]]
    hq, hkv, hd, eps = m["num_attention_heads"], m["num_key_value_heads"], m["head_dim"], m["rms_norm_eps"]
    t = len(tokens)
    freq = 1.0 / m["rope_theta"] ** (torch.arange(0, hd, 2, dtype=torch.float64, device="cuda") / hd)
    s = m["rope_scaling"]
    if s:
        wave = 2 * math.pi / freq
        low, high, orig = s["low_freq_factor"], s["high_freq_factor"], s["original_max_position_embeddings"]
        mix = ((orig / wave - low) / (high - low)).clamp(0, 1)
        freq = mix * freq + (1 - mix) * freq / s["factor"]
    angle = torch.arange(t, dtype=torch.float64, device="cuda")[:, None] * freq[None]
    cos, sin = angle.cos()[:, None], angle.sin()[:, None]

    def tensor(name):
        return w[name].double()

    def norm(x, name):
        return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * tensor(name)

    def rotate(x):
        a, b = x[..., :hd // 2], x[..., hd // 2:]
        return torch.cat([a * cos - b * sin, a * sin + b * cos], -1)

    def attend(q, k, v):
        k, v = (x.transpose(0, 1).repeat_interleave(hq // hkv, 0) for x in (k, v))
        out, q = [], q.transpose(0, 1)
        for at in range(0, t, 512):
            to = min(t, at + 512)
            score = q[:, at:to] @ k[:, :to].transpose(1, 2) / math.sqrt(hd)
            seen = torch.arange(to, device="cuda")[None] <= torch.arange(at, to, device="cuda")[:, None]
            out.append(score.masked_fill(~seen, -math.inf).softmax(-1) @ v[:, :to])
        return torch.cat(out, 1).transpose(0, 1).reshape(t, hq * hd)

    x = w["model.embed_tokens.weight"][torch.tensor(tokens, device="cuda")].double()
    for i in range(m["num_hidden_layers"]):
        p = "model.layers.%d." % i
        h = norm(x, p + "input_layernorm.weight")
        q, k, v = ((h @ tensor(p + "self_attn.%s_proj.weight" % n).t()).view(t, -1, hd) for n in "qkv")
        x = x + attend(rotate(q), rotate(k), v) @ tensor(p + "self_attn.o_proj.weight").t()
        h = norm(x, p + "post_attention_layernorm.weight")
        gate = h @ tensor(p + "mlp.gate_proj.weight").t()
        x = x + (gate * torch.sigmoid(gate) * (h @ tensor(p + "mlp.up_proj.weight").t())) @ tensor(p + "mlp.down_proj.weight").t()
    head = "model.embed_tokens.weight" if m["tie_word_embeddings"] else "lm_head.weight"
    return norm(x[places], "model.norm.weight") @ tensor(head).t()


def exact(case, seed):
    if case["kind"] == "sample":
        return None
    if work(dict(case, kind="request", chunk=0, new=1))["flops"] > 1.5e14:
        return None         # over about 20 seconds in 64 bits
    prompts, follow = _tokens(case, seed, NEW_TOKENS if case["kind"] == "decode" else case["new"])
    if case["kind"] == "decode":
        follow = follow[:1]
    w = _weights(case["model"], torch.float32 if case["dtype"] == "float32" else torch.bfloat16)
    each = [_exact_logits(case, w, p + [row[i] for row in follow], list(range(len(p) - 1, len(p) + len(follow))))
            for i, p in enumerate(prompts)]
    if case["kind"] == "decode":
        return torch.stack([e[1] for e in each])
    chunk, order = case["chunk"] or max(map(len, prompts)), []
    for at in range(0, max(map(len, prompts)), chunk):
        order += [(i, 0) for i, p in enumerate(prompts) if at < len(p) <= at + chunk]
    order += [(i, k + 1) for k in range(len(follow)) for i in range(len(prompts))]
    return torch.stack([each[i][k] for i, k in order])
