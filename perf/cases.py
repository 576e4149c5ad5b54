"""What the engine's speed is measured on: steps of the model runner, whole short requests and the sampler, at the
sizes this package is used at.

A case is one of three kinds.

``step``     one step of ``ModelRunner.step`` over requests whose earlier tokens lie in the paged cache: any number
             of sequences that decode one token each, beside at most one portion of a prompt.  A step may be run
             again on the same state: it writes the same keys and values to the same places.
``request``  whole requests of a design that keeps a state per request: their prompts in one step, then ``new`` steps
             that decode a given token for each of them; the requests come and go inside the pass.
``sample``   the draw of every row's next token from a step's logits.

The engine (weights, page pools, captured graphs) is what a serving program keeps while requests come and go: it is
made once for a kind of model and holds every state that is alive.  Weights are random (seed 0) in the checkpoint's
layout, tokens are uniform over the vocabulary, as in ``bench.py``.
"""

from __future__ import annotations

import math
import weakref

import numpy as np
import torch

from deterministic_inference_b200 import EngineConfig, SamplingParams, preset
from deterministic_inference_b200.config import GamilornConfig, NedupelConfig
from deterministic_inference_b200.engine.batch import SequenceInput
from deterministic_inference_b200.engine.runner import ModelRunner
from deterministic_inference_b200.sampling import sample
from deterministic_inference_b200.weights.random_init import random_tensors_on_device

WEIGHT_SEED = 0
STEP_TOKENS = 8192           # the engine's token budget of a step


# ---- the cases ----------------------------------------------------------------------------------

def listed() -> list:
    def step(name, model="qwen3_0_6b", dtype="bfloat16", decode=0, context=0, ragged=False, portion=0, prefix=0):
        return {"name": name, "kind": "step", "model": model, "layers": LAYERS[model], "dtype": dtype, "decode": decode,
                "context": context, "ragged": ragged, "portion": portion, "prefix": prefix}

    return [
        # one user in a conversation: the latency of a token
        step("decode_1", decode=1, context=2048),
        # the benchmark's default: a few users, long contexts of one length
        step("decode_8", decode=8, context=2048),
        # a busy server: many requests of all lengths up to 2,048
        step("decode_64_ragged", decode=64, context=2048, ragged=True),
        # a question of two sentences, to its first token
        step("prompt_83", portion=83),
        # the benchmark's prompt
        step("prompt_2048", portion=2048),
        # continuous batching: decoding requests beside a later portion of a long prompt
        step("mixed_24_and_1000", decode=24, context=1500, ragged=True, portion=1000, prefix=700),
        # a larger model (the benchmark's second one), decoding and reading a prompt
        step("decode_8_large", model="qwen3_8b", decode=8, context=2048),
        step("prompt_3000_large", model="qwen3_8b", portion=3000),
        # the 32-bit path, which traces are replayed and compared with
        step("float32_4_and_200", dtype="float32", decode=4, context=600, ragged=True, portion=200, prefix=100),
        # the designs with a state per request: a long prompt of the one (sigmoid attention beside a delta rule), and
        # short conversations of the other (latent attention, retention, routed experts)
        {"name": "gamilorn_prompt_2048", "kind": "request", "design": "gamilorn", "layers": 4, "batch": 1,
         "prompt": 2048, "ragged": False, "new": 0},
        {"name": "nedupel_8_conversations", "kind": "request", "design": "nedupel", "layers": 4, "batch": 8,
         "prompt": 200, "ragged": True, "new": 16},
        # a server's sampling step: rows with temperatures, some with top-k and top-p, some greedy
        {"name": "sample_64", "kind": "sample", "rows": 64, "vocab": 151936, "filtered": True},
    ]


LAYERS = {"qwen3_0_6b": 28, "qwen3_8b": 12}      # the second model is cut as the benchmark cuts it


def _log_uniform(rng, lo: int, hi: int) -> int:
    return min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))


def draw(rng) -> dict:
    kind = rng.choice(["decode", "decode", "prompt", "prompt", "mixed", "float32", "request", "request", "request",
                       "sample"])
    if kind == "sample":
        return {"kind": "sample", "rows": _log_uniform(rng, 1, 64),
                "vocab": rng.choice([151936, rng.randrange(20000, 152000)]), "filtered": rng.random() < 0.6}
    if kind == "request":
        batch = _log_uniform(rng, 1, 16)
        return {"kind": "request", "design": rng.choice(["gamilorn", "nedupel"]), "layers": 4, "batch": batch,
                "prompt": _log_uniform(rng, 16, min(3000, 4000 // batch)), "ragged": batch > 1 and rng.random() < 0.7,
                "new": rng.choice([0, 0, _log_uniform(rng, 1, 16)])}
    model = "qwen3_8b" if kind in ("decode", "prompt") and rng.random() < 0.3 else "qwen3_0_6b"
    case = {"kind": "step", "model": model, "layers": LAYERS[model], "dtype": "bfloat16", "decode": 0, "context": 0,
            "ragged": False, "portion": 0, "prefix": 0}
    if kind in ("decode", "mixed"):
        case["decode"] = _log_uniform(rng, 1, 64 if kind == "decode" else 32)
        case["context"] = _log_uniform(rng, 64, min(4096, 65536 // case["decode"]))
        case["ragged"] = case["decode"] > 1 and rng.random() < 0.7
    if kind == "prompt":
        case["portion"] = _log_uniform(rng, 16, 3000)
    if kind == "mixed":
        case["portion"] = _log_uniform(rng, 32, 2000)
        case["prefix"] = rng.choice([0, _log_uniform(rng, 16, 2000)])
    if kind == "float32":
        case.update(dtype="float32", decode=rng.randrange(1, 9), context=_log_uniform(rng, 32, 1000), ragged=True,
                    portion=_log_uniform(rng, 2, 300), prefix=rng.choice([0, _log_uniform(rng, 16, 300)]))
    return case


# ---- configurations -------------------------------------------------------------------------------

def _gamilorn(layers: int):
    """The benchmark's Gamilorn at the layer sizes of Qwen3-0.6B."""
    q = preset("qwen3_0_6b")
    layer = {"type": "parallel",
             "mixer": {"left": {"heads": q.num_attention_heads, "kv_heads": q.num_key_value_heads, "dim": q.head_dim,
                                "vdim": q.head_dim, "scale": q.head_dim ** -0.5, "mask": {"size": 1024, "keep_first": 4}},
                       "left_scale": 1.0, "right": {"heads": 16, "dim": 64, "decay_rank": 64}, "right_scale": 1.0},
             "mlp": {"kind": "dense", "ff": q.intermediate_size}}
    return GamilornConfig.from_dict({
        "architecture": "Gamilorn", "vocab": q.vocab_size, "width": q.hidden_size, "max_positions": 8192,
        "norm": {"eps": 1e-6}, "logit_softcap": 30.0, "layers": [layer] * layers})


def _nedupel(layers: int):
    """The benchmark's Nedupel at the layer sizes of Qwen3-0.6B."""
    q = preset("qwen3_0_6b")
    d, entries = q.head_dim, []
    for i in range(layers):
        mlp = {"kind": "dense", "ff": q.intermediate_size * 3 // 2} if i == 0 else \
            {"kind": "moe", "expert": {"ff": 1536, "limit": 7.0}, "router": {"experts": 16, "top": 2}}
        if i % 2 == 0:
            m = {"heads": q.num_attention_heads, "dim": d - 64, "rot_dim": 64, "vdim": d, "kv_rank": 192,
                 "scale": d ** -0.5, "rot": {"base": 500000.0, "dims": 64, "scaling": {
                     "factor": 4.0, "original": 2048, "fast": 32.0, "slow": 1.0}}}
            if i:
                m["kv_from"] = 0
            entries.append({"type": "latent_attention", "mixer": m, "mlp": mlp})
        else:
            entries.append({"type": "retention", "mlp": mlp, "mixer": {
                "heads": 8, "dim": 128, "vdim": 256, "decay": [1.0 - 2.0 ** (-5 - h) for h in range(8)],
                "rot": {"base": 10000.0, "dims": 128}}})
    return NedupelConfig.from_dict({
        "architecture": "Nedupel", "vocab": q.vocab_size, "width": q.hidden_size, "max_positions": 8192,
        "norm": {"eps": 1e-6}, "embedding": {"scale": 4.0}, "residual_mult": 0.25, "logit_scale": 0.5,
        "layers": entries})


def _config(case: dict):
    if case["kind"] == "request":
        return {"gamilorn": _gamilorn, "nedupel": _nedupel}[case["design"]](case["layers"])
    return preset(case["model"], num_hidden_layers=case["layers"], max_window_layers=case["layers"])


# ---- the engine and a state in it -------------------------------------------------------------------

_kept: list = []             # the engine of the kind of model in use, as [key, runner]


def _runner(case: dict, tokens: int) -> ModelRunner:
    """The running engine for the case's model, with pools for at least six states of ``tokens`` tokens."""
    key = (case.get("design") or case["model"], case["layers"], case.get("dtype", "bfloat16"))
    pool = 1 << max(15, (6 * tokens - 1).bit_length())
    if not _kept or _kept[0] != key or _kept[1].cfg.kv_pool_tokens < pool:
        _kept[:] = []
        _kept[:] = [key, ModelRunner(EngineConfig(
            model_config=_config(case), random_seed=WEIGHT_SEED, dtype=case.get("dtype", "bfloat16"),
            kv_pool_tokens=pool, max_reqs=512, max_seq_len=8192, max_prefill_tokens=STEP_TOKENS))]
    return _kept[1]


class State:
    pass


def _lengths(case: dict, n: int, most: int, rng) -> list:
    """Token counts of ``n`` sequences; ragged ones are spread evenly between an eighth of ``most`` and ``most`` (the
    same sum for every seed), in an order of the seed's."""
    if not case["ragged"] or n < 2:
        return [most] * n
    low = max(1, most // 8)
    return [int(x) for x in rng.permutation(np.linspace(low, most, n).astype(np.int64))]


def _tokens_of(case: dict, seed: int) -> tuple:
    """(lengths, token lists) of a case's sequences: what lies in the cache and the step's own tokens behind it."""
    rng = np.random.RandomState(seed % (1 << 31))
    vocab = _config(case).vocab_size
    if case["kind"] == "request":
        lengths = _lengths(case, case["batch"], case["prompt"], rng)
        return lengths, [rng.randint(0, vocab, n + case["new"]).tolist() for n in lengths]
    lengths = _lengths(case, case["decode"], case["context"], rng)
    own = [1] * len(lengths)
    if case["portion"]:
        lengths, own = lengths + [case["prefix"]], own + [case["portion"]]
    return lengths, [rng.randint(0, vocab, n + o).tolist() for n, o in zip(lengths, own)]


def _release(cache, slots: list) -> None:
    for s in slots:
        cache.release_slot(s)


def _prepare_sample(case: dict, seed: int) -> State:
    st = State()
    g = torch.Generator(device="cuda").manual_seed(seed)
    rng = np.random.RandomState(seed % (1 << 31))
    # a model's logits: a bulk of unlikely tokens and some hundred that stand out
    st.logits = 1.5 * torch.randn(case["rows"], case["vocab"], generator=g, device="cuda")
    at = torch.randint(0, case["vocab"], (case["rows"], 200), generator=g, device="cuda")
    st.logits.scatter_add_(1, at, 3.0 + 3.0 * torch.randn(at.shape, generator=g, device="cuda"))
    st.params, st.positions = [], []
    for i in range(case["rows"]):
        kind = ("greedy", "plain", "top_k", "top_p", "both")[i % 5] if case["filtered"] else "plain"
        st.params.append(SamplingParams(
            temperature=0.0 if kind == "greedy" else float(rng.choice([0.6, 0.7, 1.0])), seed=int(rng.randint(1 << 30)),
            top_k=int(rng.choice([20, 50])) if kind in ("top_k", "both") else -1,
            top_p=float(rng.choice([0.8, 0.95])) if kind in ("top_p", "both") else 1.0))
        st.positions.append(int(rng.randint(1, 4096)))
    return st


def prepare(case: dict, seed: int):
    if case["kind"] == "sample":
        st = _prepare_sample(case, seed)
        st.case = case
        return st
    lengths, tokens = _tokens_of(case, seed)
    runner = _runner(case, sum(-(-len(t) // 16) * 16 for t in tokens))
    st = State()
    st.case, st.runner, st.lengths, st.tokens = case, runner, lengths, tokens
    if case["kind"] == "request":
        return st
    st.slots = [runner.cache.allocate_slot() for _ in lengths]
    weakref.finalize(st, _release, runner.cache, list(st.slots))
    # the earlier tokens of every sequence, in steps of the engine's budget of tokens
    batch, used = [], 0
    for slot, n, toks in zip(st.slots, lengths, tokens):
        if n and used + n > STEP_TOKENS:
            runner.step(batch)
            batch, used = [], 0
        if n:
            batch.append(SequenceInput(slot, toks[:n], 0, []))
            used += n
    if batch:
        runner.step(batch)
    st.entries = [SequenceInput(slot, toks[n:], n, [len(toks) - n - 1])
                  for slot, n, toks in zip(st.slots, lengths, tokens)]
    return st


def run(state):
    case = state.case
    if case["kind"] == "sample":
        return sample(state.logits, state.params, state.positions)
    runner = state.runner
    if case["kind"] == "step":
        return runner.step(state.entries)[0]
    cache = runner.cache
    slots = [cache.allocate_slot() for _ in state.lengths]
    logits = [runner.step([SequenceInput(s, t[:n], 0, [n - 1])
                           for s, n, t in zip(slots, state.lengths, state.tokens)])[0]]
    for i in range(case["new"]):
        # (a decode step's logits hold until the next one)
        logits.append(runner.step([SequenceInput(s, [t[n + i]], n + i, [0])
                                   for s, n, t in zip(slots, state.lengths, state.tokens)])[0].clone())
    _release(cache, slots)
    return logits


# ---- what a pass cannot do without ---------------------------------------------------------------------

def _visible(first: int, n: int, window=None) -> float:
    """Keys that the queries at positions first .. first + n - 1 see, in all."""
    if window is None or first + n <= window:
        return n * first + n * (n + 1) / 2
    return float(sum(min(p + 1, window) for p in range(first, first + n)))


def _work_qwen3(case: dict) -> dict:
    c = _config(case)
    lengths, tokens = _tokens_of(case, 0)
    size = 4 if case["dtype"] == "float32" else 2
    h, d, hq, hkv, inter, v = (c.hidden_size, c.head_dim, c.num_attention_heads, c.num_key_value_heads,
                               c.intermediate_size, c.vocab_size)
    params = (hq + 2 * hkv) * d * h + hq * d * h + 3 * h * inter
    own = [len(t) - n for n, t in zip(lengths, tokens)]
    rows = len(own)
    layers = case["layers"]
    pairs = sum(_visible(n, o) for n, o in zip(lengths, own))
    kept = sum(lengths) + sum(own)
    return {"bytes": size * (layers * params + v * h + sum(own) * h + layers * 2 * hkv * d * kept) + 4 * rows * v,
            "flops": 2 * sum(own) * layers * params + layers * 4 * d * hq * pairs + 2 * rows * v * h}


def _work_request(case: dict) -> dict:
    lengths, _ = _tokens_of(case, 0)
    q = preset("qwen3_0_6b")
    h, v, d, hq, hkv = q.hidden_size, q.vocab_size, q.head_dim, q.num_attention_heads, q.num_key_value_heads
    b, size, total_bytes, total_flops = len(lengths), 2, 0.0, 0.0
    steps = [(sum(lengths), [(0, n) for n in lengths])] + [(b, [(n + i, 1) for n in lengths]) for i in range(case["new"])]
    for t, spans in steps:
        read = flops = 0.0
        for i in range(case["layers"]):
            if case["design"] == "gamilorn":
                pairs = sum(_visible(a, n, 1024) for a, n in spans)
                kept = sum(min(a + n, 1024 + n) for a, n in spans)
                dense = (hq + 2 * hkv) * d * h + hq * d * h + 6 * h * 1024 + 2 * 64 * h + 2 * h * q.intermediate_size
                read += size * (dense + 2 * hkv * d * kept) + 2 * 4 * b * 16 * 64 * 64
                flops += 2 * t * dense + 4 * d * hq * pairs + 8 * t * 16 * 64 * 64
                continue
            if i % 2 == 0:
                pairs, kept = sum(_visible(a, n) for a, n in spans), sum(a + n for a, n in spans)
                mixer = 2 * hq * d * h + (256 * h if i == 0 else 0) + hq * 192 * (d - 64 + d)
                read += size * (mixer + 256 * kept)
                flops += 2 * t * mixer + 4 * d * hq * pairs
            else:
                mixer = 2 * 1024 * h + 3 * 2048 * h
                read += size * mixer + 2 * 4 * b * 8 * 128 * 256
                flops += 2 * t * mixer + 4 * t * 8 * 128 * 256
            if i == 0:
                ff = ff_row = 2 * h * (q.intermediate_size * 3 // 2)
            else:      # every expert some token asks for is read once, a token meets two
                ff, ff_row = 3 * h * 1536 * 16 * (1 - (1 - 2 / 16) ** t), 2 * 3 * h * 1536
            read += size * ff
            flops += 2 * t * ff_row
        total_bytes += read + size * (v * h + t * h) + 4 * b * v
        total_flops += flops + 2 * b * v * h
    return {"bytes": total_bytes, "flops": total_flops}


def work(case: dict) -> dict:
    if case["kind"] == "sample":
        n = case["rows"] * case["vocab"]
        return {"bytes": 4 * n, "flops": 10 * n}
    return _work_request(case) if case["kind"] == "request" else _work_qwen3(case)


def tolerance(case: dict):
    if case["kind"] == "sample":
        return "exact"
    # about four times the distance from the 64-bit results (2e-6; 0.005 of four layers with a 32-bit stream; 0.012 of
    # 28 layers with a 16-bit one, 0.026 at the larger width: there the limit is what a comparison can use)
    if case.get("dtype") == "float32":
        return {"rel": 1e-5, "max": 1e-4}
    return {"rel": 0.02, "max": 0.2} if case["kind"] == "request" else {"rel": 0.03, "max": 0.3}


# ---- the same in 64 bits ---------------------------------------------------------------------------------

def _weights(case: dict) -> dict:
    """The engine's weights (they are inputs here), read as 64-bit numbers when they are used."""
    from deterministic_inference_b200.models.decoder import DecoderModel
    specs = DecoderModel(_config(case).plan(), torch.bfloat16, "cuda").tensor_specs()
    return random_tensors_on_device(specs, WEIGHT_SEED, torch.bfloat16, "cuda")


def _unit(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _frequencies(dims: int, base: float):
    return base ** (-torch.arange(0, dims, 2, dtype=torch.float64, device="cuda") / dims)


def _halves(x, pos, freqs):
    """Rotation of element i with element i + half; x [n, heads, dims], pos [n]."""
    a = (pos.double()[:, None] * freqs)[:, None, :]
    u, v = x.chunk(2, dim=-1)
    return torch.cat([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()], dim=-1)


def _causal(n: int, window=None, keep: int = 0):
    i = torch.arange(n, device="cuda")
    seen = i[None, :] <= i[:, None]
    if window is not None:
        seen &= (i[:, None] - i[None, :] < window) | (i[None, :] < keep)
    return seen


def _exact_qwen3(case: dict, seed: int):
    c, w = _config(case), _weights(case)
    get = lambda name: w[name].double()
    lengths, tokens = _tokens_of(case, seed)
    order = sorted(range(len(tokens)), key=lambda i: (len(tokens[i]) - lengths[i] != 1, i))     # the step's order
    tokens = [tokens[i] for i in order]
    ends = np.cumsum([len(t) for t in tokens]).tolist()
    starts = [e - len(t) for e, t in zip(ends, tokens)]
    h, d, hq, hkv, eps = c.hidden_size, c.head_dim, c.num_attention_heads, c.num_key_value_heads, c.rms_norm_eps
    ids = torch.tensor([t for s in tokens for t in s], device="cuda")
    pos = torch.cat([torch.arange(len(t), device="cuda") for t in tokens])
    # (angles as the checkpoint's own code forms them: 32-bit frequencies and products)
    half = d // 2
    inv = 1.0 / (c.rope_theta ** (torch.arange(half, dtype=torch.float32) / half))
    angle = torch.outer(pos.float().cpu(), inv).double().cuda()[:, None, :]

    def turn(x):
        u, v = x.chunk(2, dim=-1)
        return torch.cat([u * angle.cos() - v * angle.sin(), v * angle.cos() + u * angle.sin()], dim=-1)

    x = w["model.embed_tokens.weight"][ids].double()
    step = 16384                               # rows of a feed-forward at a time
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        y = _unit(x, eps) * get(p + "input_layernorm.weight")
        q = (y @ get(p + "self_attn.q_proj.weight").T).view(-1, hq, d)
        k = (y @ get(p + "self_attn.k_proj.weight").T).view(-1, hkv, d)
        v = (y @ get(p + "self_attn.v_proj.weight").T).view(-1, hkv, d)
        q = turn(_unit(q, eps) * get(p + "self_attn.q_norm.weight"))
        k = turn(_unit(k, eps) * get(p + "self_attn.k_norm.weight"))
        out = torch.empty_like(q)
        for a, e in zip(starts, ends):
            hidden = ~_causal(e - a)
            for g in range(hkv):
                heads = slice(g * (hq // hkv), (g + 1) * (hq // hkv))
                s = torch.einsum("ihd,jd->hij", q[a:e, heads], k[a:e, g]) * d ** -0.5
                s = torch.softmax(s.masked_fill_(hidden, -math.inf), dim=-1)
                out[a:e, heads] = torch.einsum("hij,jd->ihd", s, v[a:e, g])
        x = x + out.reshape(-1, hq * d) @ get(p + "self_attn.o_proj.weight").T
        del q, k, v, out, y
        gate, up, down = (get(p + f"mlp.{n}_proj.weight").T for n in ("gate", "up", "down"))
        for a in range(0, x.shape[0], step):
            y = _unit(x[a:a + step], eps) * get(p + "post_attention_layernorm.weight")
            x[a:a + step] += (torch.nn.functional.silu(y @ gate) * (y @ up)) @ down
    x = _unit(x[[e - 1 for e in ends]], eps) * get("model.norm.weight")
    return x @ get("model.embed_tokens.weight" if c.tie_word_embeddings else "lm_head.weight").T


def _delta_rule(r, k, v, w, a):
    """[n, heads, d] each: S <- diag(w) S - (a u) (u^T S) + k v^T with u = k / |k|; o = S^T r."""
    n, heads, d = r.shape
    u = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    au, s, out = a * u, torch.zeros(heads, d, d, dtype=r.dtype, device=r.device), torch.empty_like(r)
    for t in range(n):
        read = torch.bmm(u[t][:, None], s)
        s = w[t][..., None] * s - au[t][..., None] * read + k[t][..., None] * v[t][:, None]
        out[t] = torch.bmm(r[t][:, None], s)[:, 0]
    return out


def _gamilorn_logits(cfg: dict, get, table, ids, wanted):
    n, eps = ids.shape[0], cfg["norm"]["eps"]
    x = table("embed")[ids].double() + table("pos")[:n].double()
    norm = lambda x, name: _unit(x, eps) * (1.0 + get(name))
    plus = torch.nn.functional.softplus
    for i, layer in enumerate(cfg["layers"]):
        p, m = f"l{i}.", layer["mixer"]
        h, c, q = norm(x, p + "norm1"), m["left"], p + "mix.left."
        query = (h @ get(q + "q").T + get(q + "q.b")).view(n, c["kv_heads"], -1, c["dim"])
        key = (h @ get(q + "k").T + get(q + "k.b")).view(n, c["kv_heads"], c["dim"])
        value = (h @ get(q + "v").T + get(q + "v.b")).view(n, c["kv_heads"], c["vdim"])
        seen = _causal(n, c["mask"]["size"], c["mask"].get("keep_first", 0))
        s = torch.einsum("ighd,jgd->ghij", query, key) * c["scale"] + get(q + "pb").view(c["kv_heads"], -1, 1, 1)
        o = torch.einsum("ghij,jgd->ighd", torch.sigmoid(s) * seen, value).reshape(n, -1)
        left = o @ get(q + "o").T
        c, q = m["right"], p + "mix.right."
        shape = (n, c["heads"], c["dim"])
        r, k, v = ((h @ get(q + s).T).view(shape) for s in "rkv")
        decay = torch.exp(-math.exp(-0.5) * torch.sigmoid(torch.tanh(h @ get(q + "w1").T) @ get(q + "w2").T + get(q + "w0")))
        rate = torch.sigmoid(h @ get(q + "a").T + get(q + "a.b"))
        o = _unit(_delta_rule(r, k, v, decay.view(shape), rate.view(shape)), eps).reshape(n, -1)
        right = (o * get(q + "norm") * torch.sigmoid(h @ get(q + "g").T)) @ get(q + "o").T
        x = x + m["left_scale"] * left + m["right_scale"] * right
        z, (a, b) = norm(x, p + "norm2") @ get(p + "mlp.up").T, get(p + "mlp.act")
        low = z.clamp(max=0.0)
        x = x + (torch.where(z > 0, plus(a) * z * z, (0.5 + plus(b)) * (torch.expm1(low) - low)) + z / 2) \
            @ get(p + "mlp.down").T
    cap = cfg["logit_softcap"]
    return cap * torch.tanh(norm(x[wanted], "final.norm") @ get("head").T / cap)


def _stretched(dims: int, base: float, s: dict):
    """(frequencies, factor on both parts of the rotation) of stretched positions: pairs that turn often keep their
    frequency, slow ones have it divided, between them the pair's index decides."""
    at = lambda turns: dims * math.log(s["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))
    lo, hi = max(math.floor(at(s["fast"])), 0), min(math.ceil(at(s["slow"])), dims - 1)
    f = _frequencies(dims, base)
    r = ((torch.arange(dims // 2, device="cuda").double() - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    return f / s["factor"] * r + f * (1 - r), 0.1 * math.log(s["factor"]) + 1.0


def _nedupel_logits(cfg: dict, get, table, ids, wanted):
    n, eps, m = ids.shape[0], cfg["norm"]["eps"], cfg["residual_mult"]
    pos = torch.arange(n, device="cuda")
    x = table("embed")[ids].double() * cfg["embedding"]["scale"]
    norm = lambda x, name: _unit(x, eps) * (1.0 + get(name))
    rows = {}
    for i, layer in enumerate(cfg["layers"]):
        p, c = f"l{i}.", layer["mixer"]
        h, q = norm(x, p + "norm1"), p + "mix."
        if layer["type"] == "latent_attention":
            freqs, size = _stretched(c["rot"]["dims"], c["rot"]["base"], c["rot"]["scaling"])
            ang = (pos.double()[:, None] * freqs)[:, None, :]

            def pairs(y):
                a, b = y[..., 0::2], y[..., 1::2]
                return size * torch.stack([a * ang.cos() - b * ang.sin(), b * ang.cos() + a * ang.sin()], -1).flatten(-2)

            if c.get("kv_from") is None:
                down = h @ get(q + "dkv").T
                rows[i] = (_unit(down[:, :c["kv_rank"]], eps) * get(q + "dkv.norm"), pairs(down[:, None, c["kv_rank"]:])[:, 0])
            latent, key_rot = rows[i if c.get("kv_from") is None else c["kv_from"]]
            query = (h @ get(q + "q").T).view(n, c["heads"], -1)
            key = (latent @ get(q + "uk").T).view(n, c["heads"], -1)
            value = (latent @ get(q + "uv").T).view(n, c["heads"], -1)
            s = torch.einsum("ihd,jhd->hij", query[..., :c["dim"]], key) + \
                torch.einsum("ihd,jd->hij", pairs(query[..., c["dim"]:]), key_rot)
            s = torch.softmax((s * c["scale"]).masked_fill(~_causal(n), -math.inf), dim=-1)
            o = torch.einsum("hij,jhd->ihd", s, value).reshape(n, -1)
        else:
            freqs = _frequencies(c["rot"]["dims"], c["rot"]["base"])
            shape = (n, c["heads"], -1)
            query = _halves((h @ get(q + "q").T).view(shape), pos, freqs)
            key = _halves((h @ get(q + "k").T).view(shape), pos, freqs) * c["dim"] ** -0.5
            decay = torch.tensor(c["decay"], dtype=torch.float64, device="cuda").log()[:, None, None]
            # the state's sum, written out: o_i = sum over j <= i of decay^(i - j) (q_i . k_j) v_j
            far = (pos[:, None] - pos[None, :]).clamp(min=0).double()
            s = torch.einsum("ihd,jhd->hij", query, key) * torch.exp(decay * far) * _causal(n)
            o = torch.einsum("hij,jhd->ihd", s, (h @ get(q + "v").T).view(shape))
            o = _unit(o, eps).reshape(n, -1) * torch.nn.functional.silu(h @ get(q + "g").T)
        x = x + m * (o @ get(q + "o").T)
        h, q, mlp = norm(x, p + "norm2"), p + "mlp.", layer["mlp"]
        if mlp["kind"] == "dense":
            y = torch.relu(h @ get(q + "up").T) ** 2 @ get(q + "down").T
        else:
            y, chosen, limit = torch.zeros_like(h), table(q + "table")[ids].long(), mlp["expert"]["limit"]
            for e in range(mlp["router"]["experts"]):
                at = (chosen == e).any(-1).nonzero()[:, 0]
                if at.numel():
                    g = (h[at] @ get(f"{q}e{e}.gate").T).clamp(max=limit)
                    u = (h[at] @ get(f"{q}e{e}.up").T).clamp(-limit, limit)
                    y[at] += (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ get(f"{q}e{e}.down").T / mlp["router"]["top"]
        x = x + m * y
    return cfg["logit_scale"] * (norm(x[wanted], "final.norm") @ get("head").T)


def _exact_request(case: dict, seed: int):
    cfg, w = _config(case).to_dict(), _weights(case)
    lengths, tokens = _tokens_of(case, seed)
    model = {"gamilorn": _gamilorn_logits, "nedupel": _nedupel_logits}[case["design"]]
    steps: list = [[] for _ in range(1 + case["new"])]
    order = sorted(range(len(tokens)), key=lambda i: (lengths[i] != 1, i))      # the prompts' step runs in this order
    for i in range(len(tokens)):
        ids = torch.tensor(tokens[i], device="cuda")
        wanted = torch.arange(lengths[i] - 1, len(tokens[i]), device="cuda")
        for s, row in zip(steps, model(cfg, lambda name: w[name].double(), lambda name: w[name], ids, wanted)):
            s.append(row)
    return [torch.stack([steps[0][i] for i in order])] + [torch.stack(s) for s in steps[1:]]


def _exact_sample(case: dict, seed: int):
    st = _prepare_sample(case, seed)
    cols = torch.arange(case["vocab"], dtype=torch.int64, device="cuda")
    out = []
    for row, p, position in zip(st.logits, st.params, st.positions):
        if p.temperature == 0:
            out.append(int(row.argmax()))
            continue
        probs = torch.softmax(row.double() / p.temperature, dim=-1)
        ranked, index = probs.sort(descending=True, stable=True)
        kept = (ranked.cumsum(0) - ranked) <= p.top_p
        if p.top_k > 0:
            kept &= torch.arange(kept.numel(), device="cuda") < p.top_k
        kept[0] = True
        step = torch.tensor(p.seed, device="cuda") * 19349663 ^ torch.tensor(position, device="cuda") * 73856093
        u = ((step * 8589934591 ^ cols * 479001599) % (1 << 24)).double() / (1 << 24)
        score = torch.log(probs + 1e-10) - torch.log(-torch.log(u + 1e-10) + 1e-10)
        keep = torch.zeros_like(kept).scatter_(0, index, kept)
        out.append(int(score.masked_fill(~keep, -math.inf).argmax()))
    return torch.tensor(out, dtype=torch.int32)


def exact(case: dict, seed: int):
    with torch.inference_mode():
        if case["kind"] == "sample":
            return _exact_sample(case, seed)
        return _exact_request(case, seed) if case["kind"] == "request" else _exact_qwen3(case, seed)
