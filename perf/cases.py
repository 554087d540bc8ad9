"""The work that a user of the engine has it do, as cases that can be timed and compared.

Three kinds of pass:

* ``step`` -- one ``ModelRunner.step`` over a batch of requests: single tokens (decoding), prompt portions, or both,
  on the layer sizes of Qwen3-4B, 8B and 14B with random weights, in bfloat16 or in true 32-bit.  Returns the logits
  of every request's last token.  The requests' contexts were processed by earlier steps of the same runner, their
  pages handed out in shuffled order as a pool in use has them.
* ``sample`` -- ``Sampler.sample_records`` over a step's logits: one token a row, with the options of the request.
* ``generate`` -- ``LLM.generate``: prompts in, tokens out, through the scheduler, for a model so small that launches
  and host work are all there is.
"""
import math

import numpy as np
import torch

from vllm_cpp_b200 import LLM, EngineConfig, ModelRunner, Qwen3Config, StepEntry, build_model
from vllm_cpp_b200.sampling import Sampler, SamplingOptions
from vllm_cpp_b200.weights.loader import WeightStore

DEVICE = "cuda:0"
PAGE = 16
STEP_TOKENS = 2048          # the engine's default token budget of a step
VOCAB = 151936
MODELS = {
    "4b": dict(hidden_size=2560, intermediate_size=9728, num_hidden_layers=36, num_attention_heads=32, tie_word_embeddings=True),
    "8b": dict(hidden_size=4096, intermediate_size=12288, num_hidden_layers=36, num_attention_heads=32, tie_word_embeddings=False),
    "14b": dict(hidden_size=5120, intermediate_size=17408, num_hidden_layers=40, num_attention_heads=40, tie_word_embeddings=False),
}
KV_HEADS, HEAD_DIM, EPS, THETA = 8, 128, 1e-6, 1e6
DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}
SAMPLING = {      # temperature, top_p, repetition penalty
    "default": (0.7, 0.8, 1.1),     # the engine's own defaults
    "nucleus": (0.8, 0.95, 1.0),
    "temperature": (0.8, 1.0, 1.0),
    "greedy": (0.0, 1.0, 1.0),
}
TINY = dict(vocab_size=256, hidden_size=64, intermediate_size=128, num_hidden_layers=2, num_attention_heads=4,
            num_key_value_heads=2, head_dim=16, max_position_embeddings=128, rope_theta=1e4, tie_word_embeddings=True)


def _step(name, model, singles=0, low=0, high=0, prompts=0, tokens=0, start=0, dtype="bfloat16"):
    """``singles`` requests that decode one token at contexts spread over [low, high], and ``prompts`` prompt portions
    of ``tokens`` tokens together, each behind ``start`` tokens that earlier steps processed."""
    case = dict(kind="step", model=model, dtype=dtype, singles=singles, low=low, high=high, prompts=prompts, tokens=tokens,
                start=start)
    return dict(case, name=name) if name else case


def listed():
    return [
        # one person talking to the model: the latency of a token half-way through an answer to a 2,048-token prompt
        _step("decode_1", "8b", 1, 2176, 2176),
        # the benchmark's batch: eight requests at different places of their 256 new tokens
        _step("decode_8", "8b", 8, 2049, 2304),
        # a busy server: many requests of very different lengths, not a round number of them
        _step("decode_61", "4b", 61, 120, 1500),
        # the benchmark's prompt, alone in its step
        _step("prompt_2048", "8b", prompts=1, tokens=2048),
        # a short question: latency, and launches beside little work
        _step("prompt_77", "8b", prompts=1, tokens=77),
        # several ragged prompts admitted at once
        _step("prompts_9", "4b", prompts=9, tokens=911),
        # continuous batching: decoding beside a prompt portion that fills the rest of the step's budget
        _step("mixed_24", "4b", 24, 200, 3000, prompts=1, tokens=2024, start=1000),
        # the last portion of an 8,192-token prompt on the largest model
        _step("long_prompt_14b", "14b", prompts=1, tokens=2048, start=6144),
        # the true 32-bit engine, which checks of the serving engine decode and replay with
        _step("float32_decode", "4b", 3, 100, 400, dtype="float32"),
        _step("float32_prompt", "4b", prompts=1, tokens=201, dtype="float32"),
        # next tokens of a full batch with the engine's default options (penalty over what each request has seen,
        # temperature, nucleus)
        dict(name="sample_64", kind="sample", rows=64, options="default", history=600),
        # a tiny model end to end: three prompts, eight tokens each
        dict(name="generate_tiny", kind="generate", shortest=5, longest=17, requests=3, new=8),
    ]


def _spread(rng, low, high):
    """A whole number between low and high, evenly over the logarithm."""
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high + 1)) - 1e-9))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "prompt", "prompt", "mixed", "mixed", "float32", "sample", "sample", "generate"])
    if kind == "decode":
        singles = _spread(rng, 1, 256)
        high = _spread(rng, 32, min(4000, 40000 // singles))
        return _step(None, rng.choice(["4b", "8b"]) if singles > 8 else rng.choice(["4b", "8b", "14b"]), singles,
                     rng.randint(max(1, high // 10), high), high)
    if kind == "prompt":
        tokens = _spread(rng, 2, 2048)
        prompts = rng.randint(1, min(12, tokens // 2))
        return _step(None, rng.choice(["4b", "8b"]), prompts=prompts, tokens=tokens, start=rng.choice([0, 0, rng.randint(1, 2000)]))
    if kind == "mixed":
        singles = _spread(rng, 1, 64)
        high = _spread(rng, 32, min(4000, 40000 // singles))
        tokens = _spread(rng, 2, 2048 - singles)
        return _step(None, rng.choice(["4b", "8b"]), singles, rng.randint(max(1, high // 10), high), high,
                     rng.randint(1, min(4, tokens // 2)), tokens, rng.choice([0, rng.randint(1, 2000)]))
    if kind == "float32":
        if rng.random() < 0.5:
            high = rng.randint(20, 400)
            return _step(None, "4b", rng.randint(1, 8), rng.randint(1, high), high, dtype="float32")
        return _step(None, "4b", prompts=1, tokens=_spread(rng, 2, 200), start=rng.choice([0, rng.randint(1, 300)]), dtype="float32")
    if kind == "sample":
        return dict(kind="sample", rows=_spread(rng, 1, 256), options=rng.choice(["default", "default", "nucleus", "temperature", "greedy"]),
                    history=_spread(rng, 1, 4000))
    return dict(kind="generate", shortest=rng.randint(1, 8), longest=rng.randint(9, 40), requests=rng.randint(1, 8), new=rng.randint(2, 12))


# ------------------------------------------------------------------------------------------------ a step's shape
def _between(low, high, n):
    """n whole numbers spread unevenly over [low, high]: the golden ratio's multiples, so none follows from the last."""
    return [low + int((high - low + 1) * ((0.5 + 0.6180339887498949 * i) % 1.0)) for i in range(n)]


def _requests(case):
    """(tokens already processed, tokens of this step) of every request."""
    shape = [(c, 1) for c in _between(case["low"], case["high"], case["singles"])]
    if case["prompts"]:
        weights = _between(50, 150, case["prompts"])
        lengths = [max(1, case["tokens"] * w // sum(weights)) for w in weights]
        lengths[0] += case["tokens"] - sum(lengths)
        shape += [(case["start"], n) for n in lengths]
    return shape


def _config(case):
    return Qwen3Config(vocab_size=VOCAB, num_key_value_heads=KV_HEADS, head_dim=HEAD_DIM, max_position_embeddings=40960,
                       rms_norm_eps=EPS, rope_theta=THETA, **MODELS[case["model"]])


def _generator(seed, index):
    g = torch.Generator(device=DEVICE)
    g.manual_seed((int(seed) * 1000003 + index) & 0x7FFFFFFFFFFFFFFF)
    return g


def _layer_shapes(m):
    q, kv = m["num_attention_heads"] * HEAD_DIM, KV_HEADS * HEAD_DIM
    h, i = m["hidden_size"], m["intermediate_size"]
    return {"input_layernorm.weight": (h,), "self_attn.q_proj.weight": (q, h), "self_attn.k_proj.weight": (kv, h),
            "self_attn.v_proj.weight": (kv, h), "self_attn.o_proj.weight": (h, q), "self_attn.q_norm.weight": (HEAD_DIM,),
            "self_attn.k_norm.weight": (HEAD_DIM,), "post_attention_layernorm.weight": (h,), "mlp.gate_proj.weight": (i, h),
            "mlp.up_proj.weight": (i, h), "mlp.down_proj.weight": (h, i)}


def _tensor(shape, dtype, seed, index):
    """Matrices N(0, 0.02), gains 1 + N(0, 0.1)."""
    t = torch.empty(shape, dtype=dtype, device=DEVICE).normal_(0.0, 0.02 if len(shape) == 2 else 0.1, generator=_generator(seed, index))
    return t if len(shape) == 2 else t + 1


def _layer(case, seed, layer):
    return {name: _tensor(shape, DTYPES[case["dtype"]], seed, 16 * (layer + 1) + k)
            for k, (name, shape) in enumerate(_layer_shapes(MODELS[case["model"]]).items())}


def _ends(case, seed):
    m, dt = MODELS[case["model"]], DTYPES[case["dtype"]]
    t = {"model.embed_tokens.weight": _tensor((VOCAB, m["hidden_size"]), dt, seed, 1), "model.norm.weight": _tensor((m["hidden_size"],), dt, seed, 2)}
    if not m["tie_word_embeddings"]:
        t["lm_head.weight"] = _tensor((VOCAB, m["hidden_size"]), dt, seed, 3)
    return t


def _tokens(case, seed):
    """All tokens of every request, the processed ones and this step's."""
    rng = np.random.default_rng([int(seed), 7])
    return [rng.integers(0, VOCAB, past + n).tolist() for past, n in _requests(case)]


# ------------------------------------------------------------------------------------------------ step
def _prepare_step(case, seed):
    m, dtype = MODELS[case["model"]], DTYPES[case["dtype"]]
    tensors = _ends(case, seed)
    for layer in range(m["num_hidden_layers"]):
        tensors.update({f"model.layers.{layer}.{k}": t for k, t in _layer(case, seed, layer).items()})
    model = build_model(_config(case), dtype, DEVICE)
    store = WeightStore(tensors, dtype, DEVICE)
    del tensors
    model.load(store)
    store.release()

    shape, tokens = _requests(case), _tokens(case, seed)
    blocks = [-(-(past + n) // PAGE) for past, n in shape]
    order = np.random.default_rng([int(seed), 11]).permutation(sum(blocks)).tolist()
    tables = [order[sum(blocks[:i]):sum(blocks[:i + 1])] for i in range(len(blocks))]
    runner = ModelRunner(model, PAGE, sum(blocks), len(shape), dtype, DEVICE, max_model_len=max(64, PAGE * max(blocks)),
                         max_step_tokens=STEP_TOKENS)
    # the processed tokens, in steps of up to the budget
    batch, room = [], STEP_TOKENS
    for slot, (past, _) in enumerate(shape):
        at = 0
        while at < past:
            n = min(past - at, room)
            batch.append(StepEntry(slot, at, tokens[slot][at:at + n], [tables[slot]], []))
            at, room = at + n, room - n
            if room == 0:
                runner.step(batch, check=False)
                batch, room = [], STEP_TOKENS
    if batch:
        runner.step(batch, check=False)
    entries = [StepEntry(slot, past, tokens[slot][past:], [tables[slot]], [n - 1]) for slot, (past, n) in enumerate(shape)]
    runner.step(entries)        # a step of this shape ran before: what the runner captures once is there
    return dict(kind="step", runner=runner, entries=entries)


def _rope(x, positions):
    half = HEAD_DIM // 2
    angle = positions.double()[:, None] * (THETA ** (-torch.arange(half, dtype=torch.float64, device=x.device) / half))[None, :]
    cos, sin = angle.cos()[:, None, :], angle.sin()[:, None, :]
    a, b = x[..., :half], x[..., half:]
    return torch.cat([a * cos - b * sin, b * cos + a * sin], dim=-1)


def _rms(x, gain):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS) * gain


def _exact_step(case, seed):
    w = work(case)
    m, shape = MODELS[case["model"]], _requests(case)
    total = sum(p + n for p, n in shape)
    heads = m["num_attention_heads"]
    per_token = 2.0 * m["num_hidden_layers"] * sum(s[0] * s[1] for s in _layer_shapes(m).values() if len(s) == 2)
    scores = 4.0 * m["num_hidden_layers"] * heads * HEAD_DIM * sum((p + n) ** 2 for p, n in shape)
    if per_token * total + scores > 4e14 or w["flops"] <= 0:
        return None
    ids = _tokens(case, seed)
    ends = _ends(case, seed)
    table = ends["model.embed_tokens.weight"]
    x = table[torch.tensor([t for r in ids for t in r], device=DEVICE)].double()
    lengths = [len(r) for r in ids]
    starts = np.concatenate([[0], np.cumsum(lengths)]).tolist()
    positions = torch.cat([torch.arange(n, device=DEVICE) for n in lengths])
    group = heads // KV_HEADS
    for layer in range(m["num_hidden_layers"]):
        t = {k: v.double() for k, v in _layer(case, seed, layer).items()}
        y = _rms(x, t["input_layernorm.weight"])
        q = (y @ t["self_attn.q_proj.weight"].T).view(total, heads, HEAD_DIM)
        k = (y @ t["self_attn.k_proj.weight"].T).view(total, KV_HEADS, HEAD_DIM)
        v = (y @ t["self_attn.v_proj.weight"].T).view(total, KV_HEADS, HEAD_DIM)
        q = _rope(_rms(q, t["self_attn.q_norm.weight"]), positions)
        k = _rope(_rms(k, t["self_attn.k_norm.weight"]), positions)
        mixed = torch.empty_like(q)
        for i, n in enumerate(lengths):
            s = slice(starts[i], starts[i] + n)
            for a in range(0, n, 2048):     # query rows of one request, a stretch at a time
                b = min(n, a + 2048)
                qs = q[s][a:b].view(b - a, KV_HEADS, group, HEAD_DIM).permute(1, 2, 0, 3).reshape(KV_HEADS, group * (b - a), HEAD_DIM)
                ks, vs = k[s][:b].permute(1, 2, 0), v[s][:b].permute(1, 0, 2)
                hidden = torch.arange(b, device=DEVICE)[None, :] > torch.arange(a, b, device=DEVICE)[:, None]
                for h in range(KV_HEADS):
                    score = (qs[h] @ ks[h] / math.sqrt(HEAD_DIM)).view(group, b - a, b).masked_fill_(hidden, -math.inf)
                    out = torch.softmax(score, -1) @ vs[h]
                    mixed[s][a:b].view(b - a, KV_HEADS, group, HEAD_DIM)[:, h] = out.permute(1, 0, 2)
        x = x + mixed.view(total, -1) @ t["self_attn.o_proj.weight"].T
        y = _rms(x, t["post_attention_layernorm.weight"])
        for a in range(0, total, 8192):
            part = y[a:a + 8192]
            up = torch.nn.functional.silu(part @ t["mlp.gate_proj.weight"].T) * (part @ t["mlp.up_proj.weight"].T)
            x[a:a + 8192] += up @ t["mlp.down_proj.weight"].T
    last = x[torch.tensor(starts[1:], device=DEVICE) - 1]
    head = ends.get("lm_head.weight", table)
    y = _rms(last, ends["model.norm.weight"].double())
    return torch.cat([y @ head[a:a + 16384].double().T for a in range(0, VOCAB, 16384)], dim=1)


# ------------------------------------------------------------------------------------------------ sample
def _prepare_sample(case, seed):
    rows, g = case["rows"], _generator(seed, 5)
    # a model's scores: a broad bulk and a few tokens that stand out
    logits = torch.empty(rows, VOCAB, device=DEVICE).normal_(0.0, 2.5, generator=g)
    best = torch.randint(0, VOCAB, (rows, 24), generator=g, device=DEVICE)
    logits.scatter_add_(1, best, torch.empty(rows, 24, device=DEVICE).uniform_(4.0, 14.0, generator=g))
    sampler = Sampler(VOCAB, rows, DEVICE)
    temperature, top_p, penalty = SAMPLING[case["options"]]
    flat, use_counts, no_nucleus = Sampler.records([SamplingOptions(temperature, top_p, penalty, int(seed) * 1000 + r) for r in range(rows)],
                                                   [(7 * r) % 256 for r in range(rows)], list(range(rows)))
    if use_counts:      # what each request has seen so far, among it some of the tokens that stand out now
        seen = torch.randint(0, VOCAB, (rows, case["history"]), generator=g, device=DEVICE, dtype=torch.int32)
        few = min(8, case["history"])
        seen[:, :few] = best[:, :few].int()
        slots = (torch.arange(rows, device=DEVICE, dtype=torch.int32) + 1)[:, None].expand_as(seen)
        sampler.observe(seen.reshape(-1).contiguous(), slots.reshape(-1).contiguous(), seen.numel())
    params = torch.tensor(flat, dtype=torch.int32, device=DEVICE).view(-1, 8)
    return dict(kind="sample", sampler=sampler, args=(logits, params, use_counts, no_nucleus))


# ------------------------------------------------------------------------------------------------ generate
def _prepare_generate(case, seed):
    llm = LLM(config=Qwen3Config(**TINY), random_seed=int(seed), engine=EngineConfig(
        dtype="float32", page_size=4, max_tokens=1024, max_num_seqs=8, max_step_tokens=64))
    rng = np.random.default_rng([int(seed), 13])
    prompts = [rng.integers(0, TINY["vocab_size"], n).tolist() for n in _between(case["shortest"], case["longest"], case["requests"])]
    state = dict(kind="generate", llm=llm, prompts=prompts, new=case["new"])
    run(state)          # an engine that has served such requests before
    return state


# ------------------------------------------------------------------------------------------------ the interface
def prepare(case, seed):
    return {"step": _prepare_step, "sample": _prepare_sample, "generate": _prepare_generate}[case["kind"]](case, seed)


def run(state):
    if state["kind"] == "step":
        return state["runner"].step(state["entries"], check=False)
    if state["kind"] == "sample":
        return state["sampler"].sample_records(*state["args"])
    return [torch.tensor(t) for t in state["llm"].generate(state["prompts"], state["new"], 0.0, 1.0, repeat_penalty=1.0)]


def exact(case, seed):
    return _exact_step(case, seed) if case["kind"] == "step" else None


def work(case):
    if case["kind"] == "sample":
        counted = SAMPLING[case["options"]][2] != 1.0
        return {"bytes": case["rows"] * (VOCAB * (8 if counted else 4) + 36.0), "flops": 0.0}
    if case["kind"] == "generate":
        m, vocab, requests = TINY, TINY["vocab_size"], case["requests"]
        layer = sum(a * b for a, b in ((64, 64), (32, 64), (32, 64), (64, 64), (128, 64), (128, 64), (64, 128)))
        params = m["num_hidden_layers"] * layer + vocab * m["hidden_size"]
        fed = sum(_between(case["shortest"], case["longest"], requests)) + requests * (case["new"] - 1)
        return {"bytes": float(4 * case["new"] * params), "flops": 2.0 * fed * params}
    m, shape, size = MODELS[case["model"]], _requests(case), 4 if case["dtype"] == "float32" else 2
    layers, heads = m["num_hidden_layers"], m["num_attention_heads"]
    params = layers * sum(s[0] * s[1] for s in _layer_shapes(m).values() if len(s) == 2)
    new, keys = sum(n for _, n in shape), sum(p + n for p, n in shape)
    pairs = sum(n * p + n * (n + 1) / 2 for p, n in shape)      # (query, key) pairs that causality leaves
    return {
        # every matrix and the head once, the tokens' embedding rows, all keys and values once (read, or written by
        # this step), the logits out
        "bytes": float(size * (params + VOCAB * m["hidden_size"] + new * m["hidden_size"] + layers * keys * 2 * KV_HEADS * HEAD_DIM)
                       + 4 * len(shape) * VOCAB),
        "flops": 2.0 * params * new + 2.0 * VOCAB * m["hidden_size"] * len(shape) + 4.0 * layers * heads * HEAD_DIM * pairs,
    }


def tolerance(case):
    if case["kind"] != "step":
        return "exact"          # tokens
    if case["dtype"] == "float32":
        return {"rel": 5e-5}    # 36 layers of 32-bit sums: 1.3e-5 from 64 bits, as far as another order of the sums may be off
    # activations rounded to bfloat16 at every hand-over of 36 layers: 2e-2 (a single logit 0.1) between two orders of
    # the products' 32-bit sums, 3.3e-2 from 64 bits
    return {"rel": 0.03, "max": 0.4}
