"""The work that users have the engine do, as cases that can be timed and compared.

A case is one batch of requests from their prompts to their last token, through the engine's by-hand entry points
(`submit`, `plan`, `build_batch`, the step function, `commit`, `poll`): prompts enter in portions of up to `budget` rows a
step beside the decoded tokens of the requests that have started, then all decode. The tokens that follow a prompt are
given (a replay, as `bin/trace_run` does it), so that two runs can be compared by their logits: those from which every
request's first and last token are drawn. The model, its engine and its pool are kept from pass to pass; every pass
submits its requests anew.

Models have the sizes that bench.py has (GPT-2 at 124M, 355M and 1.5B; the six other designs with the layers of one of
these sizes), random weights drawn name by name, rounded to bfloat16. The 64-bit statements of the seven designs below
share no code with the package.
"""

from __future__ import annotations

import math
import zlib

import numpy as np
import torch

# ---- configurations -----------------------------------------------------------------------------

SIZES = {"124M": (12, 768, 12), "355M": (24, 1024, 16), "1.5B": (48, 1600, 25)}   # layers, width, heads
VOCAB, POSITIONS, PAGE = 50257, 1024, 16
BIAS_ROWS, DECAY_RANK = 16, 16    # sizes that a configuration leaves to the checkpoint


def _divisor(h: int, most: int) -> int:
    return max(k for k in range(1, max(1, most) + 1) if h % k == 0)


def config_of(case: dict) -> dict:
    """config.json of a case's model."""
    layers, d, h = SIZES[case["size"]]
    hd, kv, design = d // h, _divisor(h, h // 4), case["design"]
    ff = max(128, round(8 * d / 3 / 128) * 128)   # a gated unit with as many weights as GPT-2's two matrices
    if design == "gpt2":
        return {"architectures": ["GPT2LMHeadModel"], "model_type": "gpt2", "n_layer": layers, "n_embd": d, "n_head": h, "n_inner": 4 * d,
                "vocab_size": VOCAB, "n_positions": POSITIONS, "activation_function": "gelu_new", "layer_norm_epsilon": 1e-5,
                "scale_attn_weights": True, "scale_attn_by_inverse_layer_idx": False, "tie_word_embeddings": True, "eos_token_id": None}
    data = {"architecture": design.capitalize(), "vocab": VOCAB, "width": d, "norm": {"eps": 1e-5}}
    yarn = {"factor": 4.0, "original": 256, "fast": 32.0, "slow": 1.0}
    if design == "zirunex":
        mixer = {"heads": h, "kv_heads": kv, "dim": hd, "vdim": hd, "scale": hd ** -0.5, "mask": {"size": 256, "keep_first": 4}}
        data.update(embedding={"scale": 1.0},
                    layers=[{"type": "attention", "mixer": mixer, "mlp": {"kind": "dense", "ff": ff, "limit": 7.0}} for _ in range(layers)])
    elif design == "bosenex":
        memory = {"heads": h, "dim": hd // 2, "vdim": hd, "gate_cap": 15.0}
        pair = {"left": {"heads": h, "kv_heads": kv, "dim": hd, "vdim": hd, "scale": hd ** -0.5, "softcap": 30.0, "mask": {"size": 256},
                         "rot": {"dims": hd, "base": 10000.0}},
                "right": {"heads": 2 * h, "vdim": hd, "state": 64, "groups": 1, "conv": 4, "norm_groups": 1}}
        moe = {"kind": "moe", "router": {"experts": 8, "top": 2}, "expert": {"ff": ff // 4, "limit": 7.0}, "shared": {"ff": ff // 4, "limit": 7.0}}
        data.update(embedding={"scale": 1.0}, logit_scale=1.0,
                    layers=[{"type": "parallel" if i % 3 == 2 else "mlstm", "mixer": pair if i % 3 == 2 else memory,
                             "mlp": {"kind": "dense", "ff": ff} if i == 0 else moe} for i in range(layers)])
    elif design == "zudalorn":
        retention = {"heads": h, "dim": hd // 2, "vdim": hd, "decay": [1.0 - 2.0 ** (-5.0 - 3.0 * i / (h - 1)) for i in range(h)],
                     "rot": {"dims": hd // 2, "base": 10000.0}}
        latent = {"heads": h, "dim": hd, "rot_dim": hd // 2, "vdim": hd, "kv_rank": 2 * hd, "scale": (hd + hd // 2) ** -0.5, "mask": {"size": 256},
                  "rot": {"dims": hd // 2, "base": 10000.0, "scaling": yarn}}
        moe = {"kind": "moe", "router": {"experts": 8, "top": 2, "groups": {"count": 4, "keep": 2}}, "expert": {"ff": ff // 4}, "shared": {"ff": ff // 4}}
        data.update(layers=[{"type": "latent_attention" if i % 3 == 2 else "retention", "mixer": latent if i % 3 == 2 else retention,
                             "mlp": {"kind": "dense", "ff": 3 * ff // 2} if i == 0 else moe} for i in range(layers)])
    elif design == "pidodra":
        latent = {"heads": h, "dim": hd, "rot_dim": hd // 2, "vdim": hd, "kv_rank": 2 * hd, "q_rank": d // 2, "scale": (hd + hd // 2) ** -0.5,
                  "rot": {"dims": hd // 2, "base": 10000.0}}
        grouped = {"heads": h, "kv_heads": kv, "dim": hd, "vdim": hd, "scale": hd ** -0.5, "rot": {"dims": hd, "base": 10000.0, "scaling": yarn}}
        moe = {"kind": "moe", "router": {"experts": 8, "top": 2, "groups": {"count": 4, "keep": 2}, "scale": 2.0}, "expert": {"ff": ff // 4}}
        data.update(embedding={"scale": 2.0}, postln_alpha=2.0,
                    layers=[{"type": "attention" if i % 2 else "latent_attention",
                             "mixer": latent if i % 2 == 0 else dict(grouped, kv_from=i - 2) if i % 4 == 3 else grouped, "mlp": moe} for i in range(layers)])
    elif design == "lagelorn":
        delta = {"heads": h, "kv_heads": _divisor(h, h // 2), "dim": hd, "vdim": hd, "conv": 4}
        pair = {"left": {"heads": h, "kv_heads": kv, "dim": hd, "vdim": hd, "scale": hd ** -0.5, "bias_max": 128, "mask": {"size": 256}},
                "left_scale": 1.5, "right": {"heads": h, "dim": hd}, "right_scale": 0.8}
        data.update(max_positions=POSITIONS, postln_alpha=2.0, token_side={"dim": 64}, logit_softcap=25.0,
                    layers=[{"type": "parallel" if i % 3 == 2 else "delta", "mixer": pair if i % 3 == 2 else delta, "mlp": {"kind": "dense", "ff": ff}}
                            for i in range(layers)])
    else:
        half = _divisor(h, h // 2)
        pair = {"left": {"heads": half, "kv_heads": _divisor(half, half // 4), "dim": hd, "vdim": hd, "scale": hd ** -0.5, "bias_max": 128,
                         "q_temp": {"coef": 0.1, "every": 256}}, "left_scale": 0.7,
                "right": {"heads": half, "dim": hd, "vdim": hd, "decay": [1.0 - 2.0 ** (-3.0 - 6.0 * i / (half - 1)) for i in range(half)]}, "right_scale": 0.7}
        window = {"heads": h, "kv_heads": kv, "dim": hd, "vdim": hd, "scale": 1.0, "mask": {"size": 256}, "rot": {"dims": hd, "base": 10000.0}}
        moe = {"kind": "moe", "router": {"experts": 8, "identity": 2, "top": 3, "groups": {"count": 2, "keep": 1}, "scale": 1.5}, "expert": {"ff": 3 * ff // 8}}
        data.update(streams=4, residual_mult=0.7,
                    layers=[{"type": "attention" if i % 2 else "parallel", "mixer": window if i % 2 else pair, "mlp": moe} for i in range(layers)])
    return data


# ---- weights ------------------------------------------------------------------------------------

JOINS = 0.1   # the size of a sublayer's output beside a stream of ones


def tensor(name: str, shape, gpt2: bool) -> torch.Tensor:
    """The weight of that name, float32 values that bfloat16 holds: matrices that keep a row's size (GPT-2's by its own 0.02), what
    joins the stream a few times smaller than it (as trained models and their usual initialisation have it; with sublayers as large
    as the stream, a router's close calls would move the logits by more than all rounding), gains around one, gates, steps and decays in
    the range where they matter."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(zlib.crc32(name.encode()))
    x = torch.randn(tuple(shape), generator=gen, device="cuda")
    last = name.rsplit(".", 1)[-1]
    if gpt2:
        if ".ln_" in name or name.startswith("ln_f"):
            x = 0.02 * x + (1.0 if last == "weight" else 0.0)
        else:
            x = x * (0.01 if last == "bias" else 0.02)
    elif ".hc" in name:
        s = shape[0]
        x = torch.eye(s, device="cuda") + 0.1 * x if last == "mix" else (1.0 + 0.3 * x) / (s if last == "in" else 1)
    elif name in ("embed", "side.embed", "pos"):
        x = x * (0.5 if name == "pos" else 1.0)
    elif last == "conv":
        x = 0.4 * x
    elif last in ("rel", "u", "sink"):
        x = 0.7 * x
    elif ".mu." in name:
        x = torch.sigmoid(x)
    elif len(shape) == 2:
        x = x * shape[1] ** -0.5 * (JOINS if last in ("o", "down") else 1.0)
    elif last in ("norm", "norm1", "norm2"):
        x = (1.0 + 0.1 * x) * (JOINS if name.endswith("side.norm") else 1.0)
    elif last in ("out", "norm1b", "norm2b"):
        x = (1.0 + 0.1 * x) * (JOINS if last == "out" else 0.3 * JOINS)   # (after the latter nothing else makes a choice's difference smaller)
    elif last == "A_log":
        x = 0.8 * x - 0.5
    elif last == "D":
        x = 1.0 + 0.3 * x
    elif last == "w0":
        x = x - 1.5
    elif name.endswith(".f.b"):
        x = 2.0 + x
    elif last == "correction":
        x = 0.01 * x
    else:
        x = 0.3 * x
    return x.to(torch.bfloat16).float()


# ---- cases --------------------------------------------------------------------------------------

def _case(name, design, size, dtype, requests, shortest, longest, new, budget=1024, temperature=0.0, top_k=0):
    case = {"design": design, "size": size, "dtype": dtype, "requests": requests, "shortest": shortest, "longest": longest, "new": new,
            "budget": budget, "temperature": temperature, "top_k": top_k}
    return case if name is None else {"name": name, **case}


def listed() -> list[dict]:
    return [
        # somebody tries a prompt: one request, a few tokens in and out
        _case("gpt2 one request", "gpt2", "124M", "bfloat16", 1, 11, 11, 16),
        # the benchmark's batch: eight requests with prompts of 512 tokens decode side by side
        _case("gpt2 eight requests", "gpt2", "124M", "bfloat16", 8, 512, 512, 32, budget=2048),
        # scoring: whole contexts in, one token out
        _case("gpt2 two whole contexts", "gpt2", "124M", "bfloat16", 2, 1023, 1023, 1, budget=2048),
        # the true 32-bit path: a replay of a few sequences
        _case("gpt2 float32 replay", "gpt2", "124M", "float32", 3, 21, 200, 8),
        # a serving batch with sampling: prompts of very different lengths enter beside the others' decoded tokens
        _case("gpt2 355M sixty-four requests", "gpt2", "355M", "bfloat16", 64, 16, 768, 16, budget=512, temperature=0.8, top_k=40),
        # the largest model, long prompts
        _case("gpt2 1.5B eight requests", "gpt2", "1.5B", "bfloat16", 8, 900, 1000, 8, budget=2048),
        # each of the other designs with the traffic of a small service
        _case("zirunex 355M sixteen requests", "zirunex", "355M", "bfloat16", 16, 100, 900, 16),
        _case("bosenex four requests", "bosenex", "124M", "bfloat16", 4, 50, 500, 16),
        _case("zudalorn eight requests", "zudalorn", "124M", "bfloat16", 8, 30, 700, 16),
        _case("pidodra twelve requests", "pidodra", "124M", "bfloat16", 12, 100, 600, 16),
        _case("lagelorn six requests", "lagelorn", "124M", "bfloat16", 6, 40, 900, 16, temperature=0.7),
        _case("tagulix thirty-two requests", "tagulix", "124M", "bfloat16", 32, 20, 400, 16),
    ]


def draw(rng) -> dict:
    def log_uniform(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    design = rng.choice(["gpt2"] * 6 + ["zirunex", "bosenex", "zudalorn", "pidodra", "lagelorn", "tagulix"])
    float32 = design == "gpt2" and rng.random() < 0.2
    size = "124M" if float32 else rng.choice(["124M", "124M", "355M", "1.5B"] if design == "gpt2" else ["124M", "124M", "355M"])
    most = 4 if float32 else {"124M": 64, "355M": 32, "1.5B": 6}[size]
    requests = log_uniform(1, most)
    longest = log_uniform(5, 300 if float32 else 900)
    shortest = log_uniform(3, longest)
    new = rng.randint(1, 8) if float32 else rng.randint(1, {"124M": 24, "355M": 16, "1.5B": 8}[size])
    temperature, top_k = rng.choice([(0.0, 0), (0.0, 0), (0.8, 40), (1.0, 0)])
    return _case(None, design, size, "float32" if float32 else "bfloat16", requests, shortest, longest, new, budget=rng.choice([512, 1024, 2048]),
                 temperature=temperature, top_k=top_k)


def lengths(case: dict) -> list[int]:
    """The requests' prompt lengths: from the shortest to the longest, in an order in which long and short ones alternate."""
    n, lo, hi = case["requests"], case["shortest"], case["longest"]
    if n == 1:
        return [hi]
    spread = [lo + round((hi - lo) * i / (n - 1)) for i in range(n)]
    return spread[0::2][::-1] + spread[1::2]


def token_lists(case: dict, seed: int) -> tuple[list[np.ndarray], list[np.ndarray]]:
    """(prompts, the tokens that follow each)."""
    rng = np.random.default_rng([seed & 0x7FFFFFFF, 17])
    prompts = [rng.integers(0, VOCAB, n, dtype=np.int32) for n in lengths(case)]
    return prompts, [rng.integers(0, VOCAB, case["new"], dtype=np.int32) for _ in prompts]


# ---- preparing and running ----------------------------------------------------------------------

_engine: dict = {}   # the engine of the case at hand, kept as a service keeps it


def engine_of(case: dict):
    key = tuple(case[k] for k in ("design", "size", "dtype", "requests", "budget"))
    if key in _engine:
        return _engine[key]
    _engine.clear()
    torch.cuda.empty_cache()
    from research_2_b200 import run as run_engine
    from research_2_b200.config.registry import architecture_of
    from research_2_b200.models import loading
    from research_2_b200.parts import Runtime

    data = config_of(case)
    arch = architecture_of(data)
    cfg = arch.parse_config(data)
    tensors = {}
    for spec in arch.weight_spec(cfg).tensors:
        shape = [(BIAS_ROWS if n.endswith("bias rows") else DECAY_RANK) if isinstance(n, str) else n for n in spec.shape]
        tensors[spec.name] = tensor(spec.name, shape, case["design"] == "gpt2").to(torch.bfloat16)
    model = arch.build(cfg, tensors, Runtime(torch.device("cuda:0"), loading.compute_dtype(case["dtype"])))
    _engine[key] = run_engine(model, dtype=case["dtype"], max_requests=case["requests"], max_seq_len=POSITIONS, block_size=PAGE,
                              max_batch_tokens=case["budget"])
    return _engine[key]


def prepare(case: dict, seed: int) -> dict:
    prompts, replies = token_lists(case, seed)
    return {"engine": engine_of(case), "prompts": prompts, "replies": replies, "case": case, "seed": seed}


@torch.no_grad()
def run(state: dict):
    """-> {"first": the logits that each request's first new token is drawn from [requests, vocab], "last": its last one's}."""
    engine, case, n_new = state["engine"], state["case"], state["case"]["new"]
    index = {}
    for i, prompt in enumerate(state["prompts"]):
        rid = engine.submit(prompt, n_new, case["temperature"], (), case["top_k"], seed=state["seed"] | (i << 32))
        index[rid] = i
    first, last = [None] * len(index), [None] * len(index)
    while (plan := engine.plan()) is not None:
        logits = engine.step_fn(engine.build_batch(plan))
        tokens = np.zeros(plan.n_entries, dtype=np.int32)
        kept = None
        for e in range(plan.n_entries):
            if not plan.emits[e]:
                continue
            i = index[int(plan.req[e])]
            at = int(plan.start[e] + plan.rows[e]) - len(state["prompts"][i])   # this step draws the request's token `at`
            tokens[e] = state["replies"][i][at]
            if at == 0 or at == n_new - 1:
                kept = logits.clone() if kept is None else kept   # the step's own buffer is the next step's too
                if at == 0:
                    first[i] = kept[e]
                if at == n_new - 1:
                    last[i] = kept[e]
        engine.commit(tokens)
    for rid in index:
        engine.poll(rid)
    return {"first": torch.stack(first), "last": torch.stack(last)}


# ---- what a pass cannot do without --------------------------------------------------------------

def _cached_numbers(case: dict) -> list[tuple[int, int]]:
    """Per layer with a cache: (numbers read per key seen, the most keys a position sees; 0: all)."""
    layers, d, h = SIZES[case["size"]]
    hd, kv = d // h, _divisor(h, h // 4)
    grouped, latent = 2 * kv * hd, 2 * hd + hd // 2
    half = _divisor(h, h // 2)
    return {"gpt2": [(2 * d, 0)] * layers, "zirunex": [(grouped, 260)] * layers, "bosenex": [(grouped, 256)] * (layers // 3),
            "zudalorn": [(latent, 256)] * (layers // 3), "pidodra": [(latent, 0)] * (layers // 2) + [(grouped, 0)] * (layers // 2),
            "lagelorn": [(grouped, 256)] * (layers // 3),
            "tagulix": [(2 * _divisor(half, half // 4) * hd, 0)] * (layers // 2) + [(grouped, 256)] * (layers // 2)}[case["design"]]


def work(case: dict) -> dict:
    """Bytes: every step's weights once (of routed experts as many as its tokens can choose), the keys and values that its tokens
    see, the logits. Flops: the products of every token with the weights it uses, and of the heads with the keys seen."""
    from research_2_b200.config.registry import architecture_of
    from research_2_b200.models import loading  # noqa: F401  (registers the designs)

    layers, d, h = SIZES[case["size"]]
    data = config_of(case)
    arch = architecture_of(data)
    dense = routed = table = 0
    for spec in arch.weight_spec(arch.parse_config(data)).tensors:
        n = math.prod(BIAS_ROWS if isinstance(x, str) else x for x in spec.shape)
        if spec.name in ("wte.weight", "wpe.weight", "embed", "pos", "side.embed", "head"):
            table += n if spec.name in ("wte.weight", "head") else 0
        elif ".mlp.e" in spec.name:
            routed += n
        else:
            dense += n
    top = {"bosenex": 2, "zudalorn": 2, "pidodra": 2, "tagulix": 3}.get(case["design"], 0)
    size = 4 if case["dtype"] == "float32" else 2
    prompts, new = lengths(case), case["new"]
    cached = _cached_numbers(case)

    def seen(n, most):   # keys that n tokens from a sequence's start see, summed
        full = min(n, most) if most else n
        return full * (full + 1) / 2 + (n - full) * most

    n_prompt, n_decoded = sum(prompts), len(prompts) * (new - 1)
    steps = [case["budget"]] * (n_prompt // case["budget"]) + ([n_prompt % case["budget"]] if n_prompt % case["budget"] else []) + [len(prompts)] * (new - 1)
    total = sum(dense + table + routed * min(1.0, t * top / 8) for t in steps)
    for numbers, most in cached:
        total += sum(numbers * (seen(n + new - 1, most) - seen(n, most)) for n in prompts) + 2 * numbers * sum(prompts)
    flops = 2.0 * (n_prompt + n_decoded) * (dense + routed * top / 8) + 2.0 * len(prompts) * new * table
    flops += sum(4.0 * d * seen(n + new - 1, most) for n in prompts for _, most in cached)
    return {"bytes": total * size + 4.0 * len(prompts) * new * VOCAB, "flops": flops}


def tolerance(case: dict):
    """About four times the error against 64 bits that was measured (float32: 1.6e-6; bfloat16 without routers: 0.002 to 0.0055, single
    logits six times that); where routers choose, a close call that goes the other way moves a row's logits by a few hundredths."""
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-4}
    if case["design"] in ("gpt2", "zirunex", "lagelorn"):
        return {"rel": 0.02, "max": 0.15}
    return {"rel": 0.03, "max": 0.6}


# ---- the designs in 64 bits ---------------------------------------------------------------------

def exact(case: dict, seed: int):
    """The same logits from whole sequences in 64 bits: rows [requests, longest, width], the shorter ones followed by zeros that
    nothing before them sees."""
    prompts, replies = token_lists(case, seed)
    new = case["new"]
    rows = torch.zeros(len(prompts), max(map(len, prompts)) + new - 1, dtype=torch.int64, device="cuda")
    for i, (p, r) in enumerate(zip(prompts, replies)):
        rows[i, : len(p) + new - 1] = torch.from_numpy(np.concatenate([p, r[: new - 1]])).long().cuda()
    ends = torch.tensor([len(p) - 1 for p in prompts], device="cuda")

    def w(name, *shape):
        return tensor(name, shape, case["design"] == "gpt2").double()

    config = config_of(case)
    x, head = PLAIN[case["design"]](config, w, rows)
    who = torch.arange(len(prompts), device="cuda")
    out = {}
    for name, at in (("first", ends), ("last", ends + new - 1)):
        logits = head(x[who, at])
        out[name] = logits
    return out


def lin(x, w, b=None):
    y = x @ w.T
    return y if b is None else y + b


def unit(x, eps=1e-5):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def silu(x):
    return x * torch.sigmoid(x)


def gelu_tanh(x):
    return 0.5 * x * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (x + 0.044715 * x ** 3)))


def heads_of(x, n):
    return x.unflatten(-1, (n, -1))


def attend(q, k, v, scale, window=0, keep=0, chunk=0, cap=0.0, bias=None, sink=None, shared_v_heads=None):
    """q [B, T, H, d], k and v [B, T, G, .] -> [B, T, H, dv]. bias [H, T] by distance; sink [H]: exp(sink) joins the denominator."""
    b, t, h, _ = q.shape
    i, j = torch.arange(t, device=q.device)[:, None], torch.arange(t, device=q.device)[None, :]
    see = j <= i
    if window:
        see = see & ((i - j < window) | (j < keep))
    if chunk:
        see = see & (i // chunk == j // chunk)
    out = torch.empty(b, t, h, v.shape[-1], dtype=q.dtype, device=q.device)
    for n in range(h):
        g = n // (h // k.shape[2])
        s = (q[:, :, n] @ k[:, :, g].transpose(1, 2)) * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        if bias is not None:
            s = s + bias[n][(i - j).clamp(min=0)]
        s = s.masked_fill(~see, -math.inf)
        top = s.amax(-1, keepdim=True)
        if sink is not None:
            top = torch.maximum(top, sink[n])
        e = torch.exp(s - top)
        total = e.sum(-1, keepdim=True)
        if sink is not None:
            total = total + torch.exp(sink[n] - top)
        out[:, :, n] = (e / total) @ v[:, :, g]
    return out


def frequencies(rot):
    """(the angle per position of every pair, the factor on cos and sin)."""
    dims, base, scaling = rot["dims"], rot["base"], rot.get("scaling")
    plain = [base ** (-2.0 * i / dims) for i in range(dims // 2)]
    if not scaling:
        return plain, 1.0
    lo, hi = (dims * math.log(scaling["original"] / (2.0 * math.pi * scaling[k])) / (2.0 * math.log(base)) for k in ("fast", "slow"))
    lo, hi = max(math.floor(lo), 0), min(math.ceil(hi), dims - 1)
    ramp = [min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0) for i in range(dims // 2)]
    return [f / scaling["factor"] * r + f * (1.0 - r) for f, r in zip(plain, ramp)], 0.1 * math.log(scaling["factor"]) + 1.0


def rotate(x, rot, interleaved):
    """x [B, T, heads, d]: the first rot["dims"] numbers of a head turn pair by pair."""
    freqs, size = frequencies(rot)
    n, t = len(freqs), x.shape[1]
    angle = (torch.arange(t, device=x.device, dtype=x.dtype)[:, None] * torch.tensor(freqs, device=x.device, dtype=x.dtype))[None, :, None, :]
    c, s = torch.cos(angle) * size, torch.sin(angle) * size
    out = x.clone()
    a, b = (slice(0, 2 * n, 2), slice(1, 2 * n, 2)) if interleaved else (slice(0, n), slice(n, 2 * n))
    u, v = x[..., a], x[..., b]
    out[..., a], out[..., b] = u * c - v * s, v * c + u * s
    return out


def distance_bias(table, t, most):
    """table [rows, H] -> [H, t]: half the rows are distances of their own, the rest steps of the logarithm up to `most`."""
    rows, half = table.shape[0], table.shape[0] // 2
    at = [n if n < half else min(rows - 1, half + math.floor(math.log(n / half) / math.log(most / half) * (rows - half))) for n in range(t)]
    return table[at].T


def fold(q, k, v, decay):
    """S <- decay_t S + k_t v_t^T, o_t = S^T q_t. q, k [B, T, H, d], v [B, T, H, dv], decay [B or 1, T or 1, H, d or 1]."""
    b, t, h, d = k.shape
    s = torch.zeros(b, h, d, v.shape[-1], dtype=k.dtype, device=k.device)
    decay = decay.expand(b, t, h, decay.shape[-1])
    out = torch.empty_like(v)
    for i in range(t):
        s = s * decay[:, i, :, :, None] + k[:, i, :, :, None] * v[:, i, :, None, :]
        out[:, i] = (s * q[:, i, :, :, None]).sum(2)
    return out


def short_conv(x, taps, bias=0.0):
    """silu of the causal convolution; the last of `taps` [C, n] is the current row's."""
    n = taps.shape[1]
    padded = torch.nn.functional.pad(x, (0, 0, n - 1, 0))
    return silu(sum(padded[:, i: i + x.shape[1]] * taps[:, i] for i in range(n)) + bias)


def mix_experts(x, weights, unit_of):
    """x [N, D], weights [N, experts]: the chosen experts' outputs times their weights."""
    out = torch.zeros_like(x)
    for e in range(weights.shape[1]):
        at = weights[:, e].nonzero()[:, 0]
        if at.numel():
            out[at] += weights[at, e: e + 1] * unit_of(e, x[at])
    return out


def choose(score, marks_of, count, keep, top):
    """[N, n] True where chosen: the `top` largest scores inside the `keep` groups with the largest marks."""
    n = score.shape[1]
    grouped = score.unflatten(1, (count, n // count))
    kept = torch.zeros(score.shape[0], count, dtype=torch.bool, device=score.device)
    kept.scatter_(1, marks_of(grouped).topk(keep, dim=1).indices, True)
    open_to = score.masked_fill(~kept.repeat_interleave(n // count, dim=1), -math.inf)
    return torch.zeros_like(kept[:, :1]).repeat(1, n).scatter_(1, open_to.topk(top, dim=1).indices, True)


def plain_gpt2(c, w, rows):
    d, h, f = c["n_embd"], c["n_head"], c["n_inner"]

    def norm(x, p):
        x = x - x.mean(-1, keepdim=True)
        return unit(x) * w(p + ".weight", d) + w(p + ".bias", d)

    def product(x, p, n_in, n_out):
        return x @ w(p + ".weight", n_in, n_out) + w(p + ".bias", n_out)

    x = w("wte.weight", VOCAB, d)[rows] + w("wpe.weight", POSITIONS, d)[: rows.shape[1]]
    for i in range(c["n_layer"]):
        p = f"h.{i}."
        q, k, v = (heads_of(t, h) for t in product(norm(x, p + "ln_1"), p + "attn.c_attn", d, 3 * d).split(d, dim=-1))
        x = x + product(attend(q, k, v, (d // h) ** -0.5).flatten(2), p + "attn.c_proj", d, d)
        x = x + product(gelu_tanh(product(norm(x, p + "ln_2"), p + "mlp.c_fc", d, f)), p + "mlp.c_proj", f, d)
    return norm(x, "ln_f"), lambda x: lin(x, w("wte.weight", VOCAB, d))


def plain_zirunex(c, w, rows):
    d = c["width"]
    x = w("embed", VOCAB, d)[rows]
    for i, layer in enumerate(c["layers"]):
        p, m, f = f"l{i}.", layer["mixer"], layer["mlp"]["ff"]
        h = unit(x) * (1.0 + w(p + "norm1", d))
        q = unit(heads_of(lin(h, w(p + "mix.q", m["heads"] * m["dim"], d)), m["heads"])) * w(p + "mix.q.norm", m["dim"])
        k = unit(heads_of(lin(h, w(p + "mix.k", m["kv_heads"] * m["dim"], d)), m["kv_heads"])) * w(p + "mix.k.norm", m["dim"])
        v = heads_of(lin(h, w(p + "mix.v", m["kv_heads"] * m["vdim"], d)), m["kv_heads"])
        y = attend(q, k, v, m["scale"], m["mask"]["size"], m["mask"]["keep_first"], sink=torch.zeros(m["heads"], dtype=x.dtype, device=x.device))
        n = m["heads"] * m["vdim"]
        y = lin(y.flatten(2) * torch.sigmoid(lin(h, w(p + "mix.g", n, d))), w(p + "mix.o", d, n))
        g, u = lin(h, w(p + "mlp.gate", f, d)).clamp(max=7.0), lin(h, w(p + "mlp.up", f, d)).clamp(-7.0, 7.0)
        x = x + y + lin(g * torch.sigmoid(1.702 * g) * (u + 1.0), w(p + "mlp.down", d, f))
    return unit(x) * (1.0 + w("final.norm", d)), lambda x: lin(x, w("head", VOCAB, d))


def plain_bosenex(c, w, rows):
    d = c["width"]

    def memory(x, p, m):
        h, dk, dv = m["heads"], m["dim"], m["vdim"]
        q, k = heads_of(lin(x, w(p + "q", h * dk, d)), h) * dk ** -0.5, heads_of(lin(x, w(p + "k", h * dk, d)), h)
        v = heads_of(lin(x, w(p + "v", h * dv, d)), h)
        cap = m["gate_cap"]
        log_i = cap * torch.tanh(lin(x, w(p + "i", h, d), w(p + "i.b", h)) / cap)
        log_f = torch.nn.functional.logsigmoid(cap * torch.tanh(lin(x, w(p + "f", h, d), w(p + "f.b", h)) / cap))
        b, t = x.shape[:2]
        s = torch.zeros(b, h, dk, dv, dtype=x.dtype, device=x.device)
        n, top = torch.zeros(b, h, dk, dtype=x.dtype, device=x.device), torch.zeros(b, h, dtype=x.dtype, device=x.device)
        out = torch.empty_like(v)
        for i in range(t):
            after = torch.maximum(log_f[:, i] + top, log_i[:, i])
            keep, take, top = torch.exp(log_f[:, i] + top - after), torch.exp(log_i[:, i] - after), after
            s = keep[..., None, None] * s + take[..., None, None] * k[:, i, :, :, None] * v[:, i, :, None, :]
            n = keep[..., None] * n + take[..., None] * k[:, i]
            den = torch.maximum((n * q[:, i]).sum(-1).abs(), torch.exp(-top)) + 1e-6
            out[:, i] = (s * q[:, i, :, :, None]).sum(2) / den[..., None]
        out = unit(out).flatten(2) * w(p + "norm", h * dv) * torch.sigmoid(lin(x, w(p + "g", h * dv, d)))
        return lin(out, w(p + "o", d, h * dv))

    def attention(x, p, m):
        h, g, dk, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        q, k = (rotate(heads_of(lin(x, w(p + s, n * dk, d)), n), m["rot"], False) for s, n in (("q", h), ("k", g)))
        v = heads_of(lin(x, w(p + "v", g * dv, d)), g)
        y = attend(q, k, v, m["scale"], m["mask"]["size"], cap=m["softcap"], sink=w(p + "sink", h))
        return lin((y * torch.sigmoid(lin(x, w(p + "g", h, d)))[..., None]).flatten(2), w(p + "o", d, h * dv))

    def space(x, p, m):
        h, dv, n = m["heads"], m["vdim"], m["state"]
        inner = h * dv
        z, xbc, dt = lin(x, w(p + "in", 2 * inner + 2 * n + h, d)).split([inner, inner + 2 * n, h], dim=-1)
        xs, bs, cs = short_conv(xbc, w(p + "conv", inner + 2 * n, m["conv"]), w(p + "conv.b", inner + 2 * n)).split([inner, n, n], dim=-1)
        xs = heads_of(xs, h)
        dt = torch.nn.functional.softplus(dt + w(p + "dt_bias", h))
        keep = torch.exp(-torch.exp(w(p + "A_log", h)) * dt)[..., None]
        spread = [t[:, :, None, :].expand(-1, -1, h, -1) for t in (bs, cs)]
        y = fold(spread[1], spread[0], xs * dt[..., None], keep) + w(p + "D", h)[:, None] * xs
        return lin(unit(y.flatten(2) * silu(z)) * w(p + "norm", inner), w(p + "o", d, inner))

    def expert(x, p, f, limit):
        g, u = lin(x, w(p + "gate", f, d)).clamp(max=limit), lin(x, w(p + "up", f, d)).clamp(-limit, limit)
        return lin(g * torch.sigmoid(1.702 * g) * (u + 1.0), w(p + "down", d, f))

    x = w("embed", VOCAB, d)[rows]
    for i, layer in enumerate(c["layers"]):
        p, m, f = f"l{i}.", layer["mixer"], layer["mlp"]
        h = unit(x) * w(p + "norm1", d)
        if layer["type"] == "mlstm":
            x = x + memory(h, p + "mix.", m)
        else:
            left, right = attention(h, p + "mix.left.", m["left"]), space(h, p + "mix.right.", m["right"])
            x = x + 0.5 * (unit(left) * w(p + "mix.left.out", d) + unit(right) * w(p + "mix.right.out", d))
        h = unit(x) * w(p + "norm2", d)
        p += "mlp."
        if f["kind"] == "dense":
            x = x + lin(torch.relu(lin(h, w(p + "gate", f["ff"], d))) * lin(h, w(p + "up", f["ff"], d)), w(p + "down", d, f["ff"]))
            continue
        h = h.flatten(0, 1)
        e, ff = f["router"]["experts"], f["expert"]["ff"]
        best = lin(h, w(p + "router", e, d), w(p + "router.b", e)).topk(f["router"]["top"], dim=1)
        share = torch.zeros(h.shape[0], e, dtype=h.dtype, device=h.device).scatter_(1, best.indices, torch.softmax(best.values, dim=1))
        y = mix_experts(h, share, lambda n, r: expert(r, f"{p}e{n}.", ff, f["expert"]["limit"]))
        x = x + (y + expert(h, p + "shared.", f["shared"]["ff"], f["shared"]["limit"])).view_as(x)
    return unit(x) * w("final.norm", d), lambda x: lin(x, w("head", VOCAB, d))


def silu_unit(x, w, p, f, d):
    return lin(silu(lin(x, w(p + "gate", f, d))) * lin(x, w(p + "up", f, d)), w(p + "down", d, f))


def plain_zudalorn(c, w, rows):
    d = c["width"]

    def latent(x, p, m):
        h, dk, r, dv, n = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
        q = heads_of(lin(x, w(p + "q", h * (dk + r), d)), h)
        down = lin(x, w(p + "dkv", n + r, d))
        kept = unit(down[..., :n]) * w(p + "dkv.norm", n)
        turned = rotate(down[..., None, n:], m["rot"], True).expand(-1, -1, h, -1)
        k = torch.cat([heads_of(lin(kept, w(p + "uk", h * dk, n)), h), turned], dim=-1)
        q = torch.cat([q[..., :dk], rotate(q[..., dk:], m["rot"], True)], dim=-1)
        y = attend(q, k, heads_of(lin(kept, w(p + "uv", h * dv, n)), h), m["scale"], m["mask"]["size"])
        return lin(y.flatten(2), w(p + "o", d, h * dv))

    def retention(x, p, m):
        h, dk, dv = m["heads"], m["dim"], m["vdim"]
        q, k = (rotate(heads_of(lin(x, w(p + s, h * dk, d)), h), m["rot"], False) for s in "qk")
        decay = torch.tensor(m["decay"], dtype=x.dtype, device=x.device)[None, None, :, None]
        y = fold(q, k * dk ** -0.5, heads_of(lin(x, w(p + "v", h * dv, d)), h), decay)
        return lin(unit(y).flatten(2) * silu(lin(x, w(p + "g", h * dv, d))), w(p + "o", d, h * dv))

    def dense(x, p, f):
        a, b = (torch.nn.functional.softplus(t) for t in w(p + "act", 2))
        z = lin(x, w(p + "up", f, d))
        neg = z.clamp(max=0.0)
        return lin(torch.where(z > 0, a * z * z + 0.5 * z, (0.5 + b) * (torch.expm1(neg) - neg) + 0.5 * z), w(p + "down", d, f))

    def experts(x, p, f):
        e, r, ff = f["router"]["experts"], f["router"], f["expert"]["ff"]
        s = torch.sigmoid(lin(x, w(p + "router", e, d)))
        chosen = choose(s + w(p + "correction", e), lambda g: g.topk(2, dim=2).values.sum(2), r["groups"]["count"], r["groups"]["keep"], r["top"])
        share = s * chosen
        y = mix_experts(x, share / share.sum(1, keepdim=True), lambda n, t: silu_unit(t, w, f"{p}e{n}.", ff, d))
        return y + torch.sigmoid(lin(x, w(p + "shared.sg", 1, d))) * silu_unit(x, w, p + "shared.", f["shared"]["ff"], d)

    x = w("embed", VOCAB, d)[rows]
    for i, layer in enumerate(c["layers"]):
        p, f = f"l{i}.", layer["mlp"]
        h = unit(x) * w(p + "norm1")
        y = (latent if layer["type"] == "latent_attention" else retention)(h, p + "mix.", layer["mixer"])
        x = x + unit(y) * w(p + "norm1b")
        h = (unit(x) * w(p + "norm2")).flatten(0, 1)
        y = dense(h, p + "mlp.", f["ff"]) if f["kind"] == "dense" else experts(h, p + "mlp.", f)
        x = x + (unit(y) * w(p + "norm2b")).view_as(x)
    return unit(x) * w("final.norm"), lambda x: lin(x, w("head", VOCAB, d))


def plain_pidodra(c, w, rows):
    d, alpha = c["width"], c["postln_alpha"]

    def latent(x, p, m):
        h, dk, r, dv, n, nq = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"], m["q_rank"]
        q = heads_of(lin(unit(lin(x, w(p + "dq", nq, d))) * w(p + "dq.norm", nq), w(p + "uq", h * (dk + r), nq)), h)
        down = lin(x, w(p + "dkv", n + r, d))
        kept = unit(down[..., :n]) * w(p + "dkv.norm", n)
        turned = rotate(down[..., None, n:], m["rot"], True).expand(-1, -1, h, -1)
        k = torch.cat([heads_of(lin(kept, w(p + "uk", h * dk, n)), h), turned], dim=-1)
        q = torch.cat([q[..., :dk], rotate(q[..., dk:], m["rot"], True)], dim=-1)
        y = attend(q, k, heads_of(lin(kept, w(p + "uv", h * dv, n)), h), m["scale"], sink=w(p + "sink", h))
        return lin(y.flatten(2) * torch.sigmoid(lin(x, w(p + "g", h * dv, d))), w(p + "o", d, h * dv))

    def grouped(x, p, m, held):
        h, g, dk, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        q = rotate(unit(heads_of(lin(x, w(p + "q", h * dk, d)), h)) * w(p + "q.norm", dk), m["rot"], False)
        if held is None:
            k = rotate(unit(heads_of(lin(x, w(p + "k", g * dk, d)), g)) * w(p + "k.norm", dk), m["rot"], False)
            held = k, heads_of(lin(x, w(p + "v", g * dv, d)), g)
        y = attend(q, *held, m["scale"]) * torch.sigmoid(lin(x, w(p + "g", h, d)))[..., None]
        return lin(y.flatten(2), w(p + "o", d, h * dv)), held

    def experts(x, p, f):
        r = f["router"]
        s = torch.softmax(lin(x, w(p + "router", r["experts"], d)), dim=1)
        share = s * choose(s, lambda g: g.amax(2), r["groups"]["count"], r["groups"]["keep"], r["top"]) * r["scale"]
        return mix_experts(x, share, lambda n, t: silu_unit(t, w, f"{p}e{n}.", f["expert"]["ff"], d))

    x, held = w("embed", VOCAB, d)[rows] * c["embedding"]["scale"], {}
    for i, layer in enumerate(c["layers"]):
        p, m = f"l{i}.", layer["mixer"]
        if layer["type"] == "latent_attention":
            y = latent(x, p + "mix.", m)
        else:
            y, held[i] = grouped(x, p + "mix.", m, held.get(m.get("kv_from")))
        x = unit(alpha * x + y) * w(p + "norm1", d)
        x = unit(alpha * x + experts(x.flatten(0, 1), p + "mlp.", layer["mlp"]).view_as(x)) * w(p + "norm2", d)
    return unit(x) * w("final.norm", d), lambda x: lin(x, w("head", VOCAB, d))


def plain_lagelorn(c, w, rows):
    d, alpha, cap = c["width"], c["postln_alpha"], c["logit_softcap"]

    def delta(x, p, m):
        h, g, dk, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]

        def length_one(t):
            return t * torch.rsqrt((t * t).sum(-1, keepdim=True) + 1e-6)

        q, k = (length_one(heads_of(short_conv(lin(x, w(p + s, g * dk, d)), w(f"{p}{s}.conv", g * dk, m["conv"])), g)).repeat_interleave(h // g, dim=2)
                for s in "qk")
        q = q * dk ** -0.5
        v = heads_of(short_conv(lin(x, w(p + "v", h * dv, d)), w(p + "v.conv", h * dv, m["conv"])), h)
        beta = torch.sigmoid(lin(x, w(p + "b", h, d)))
        keep = torch.exp(-torch.exp(w(p + "A_log", h)) * torch.nn.functional.softplus(lin(x, w(p + "a", h, d)) + w(p + "dt_bias", h)))
        s = torch.zeros(x.shape[0], h, dk, dv, dtype=x.dtype, device=x.device)
        out = torch.empty_like(v)
        for i in range(x.shape[1]):
            s = s * keep[:, i, :, None, None]
            change = beta[:, i, :, None] * (v[:, i] - (s * k[:, i, :, :, None]).sum(2))
            s = s + k[:, i, :, :, None] * change[:, :, None, :]
            out[:, i] = (s * q[:, i, :, :, None]).sum(2)
        out = (unit(out) * w(p + "norm", dv)).flatten(2)
        return lin(out * silu(lin(x, w(p + "g", h * dv, d))), w(p + "o", d, h * dv))

    def chunks(x, p, m):
        h, g, dk = m["heads"], m["kv_heads"], m["dim"]
        q = heads_of(unit(lin(x, w(p + "q", h * dk, d), w(p + "q.b", h * dk))) * w(p + "q.norm", h * dk), h)
        raw = lin(x, w(p + "k", g * dk, d), w(p + "k.b", g * dk))
        k = heads_of(unit(raw) * w(p + "k.norm", g * dk), g)
        bias = distance_bias(w(p + "rel", BIAS_ROWS, h), x.shape[1], m["bias_max"])
        y = attend(q, k, heads_of(raw, g), m["scale"], chunk=m["mask"]["size"], bias=bias, sink=w(p + "sink", h))
        return lin(y.flatten(2), w(p + "o", d, h * dk))

    def time_mix(x, p, m):
        h, n = m["heads"], m["heads"] * m["dim"]
        before = torch.nn.functional.pad(x, (0, 0, 1, 0))[:, :-1]
        mixed = {s: x + (before - x) * w(f"{p}mu.{s}", d) for s in "rkvgw"}
        r, k, v = (heads_of(lin(mixed[s], w(p + s, n, d)), h) for s in "rkv")
        inner = lin(torch.tanh(lin(mixed["w"], w(p + "w1", DECAY_RANK, d))), w(p + "w2", n, DECAY_RANK)) + w(p + "w0", n)
        decay = heads_of(torch.exp(-torch.exp(inner)), h)
        bonus = w(p + "u", h, m["dim"])
        s = torch.zeros(x.shape[0], h, m["dim"], m["dim"], dtype=x.dtype, device=x.device)
        out = torch.empty_like(v)
        for i in range(x.shape[1]):
            write = k[:, i, :, :, None] * v[:, i, :, None, :]
            out[:, i] = ((s + bonus[:, :, None] * write) * r[:, i, :, :, None]).sum(2)
            s = s * decay[:, i, :, :, None] + write
        return lin(unit(out).flatten(2) * w(p + "norm", n) * silu(lin(mixed["g"], w(p + "g", n, d))), w(p + "o", d, n))

    x = w("embed", VOCAB, d)[rows] + w("pos", POSITIONS, d)[: rows.shape[1]]
    n = c["token_side"]["dim"]
    side = w("side.embed", VOCAB, len(c["layers"]) * n)[rows]
    for i, layer in enumerate(c["layers"]):
        p, m, f = f"l{i}.", layer["mixer"], layer["mlp"]["ff"]
        if layer["type"] == "delta":
            y = delta(x, p + "mix.", m)
        else:
            y = m["left_scale"] * chunks(x, p + "mix.left.", m["left"]) + m["right_scale"] * time_mix(x, p + "mix.right.", m["right"])
        x = unit(alpha * x + y) * w(p + "norm1", d)
        inner = gelu_tanh(lin(x, w(p + "mlp.gate", f, d), w(p + "mlp.gate.b", f))) * lin(x, w(p + "mlp.up", f, d), w(p + "mlp.up.b", f))
        x = unit(alpha * x + lin(inner, w(p + "mlp.down", d, f), w(p + "mlp.down.b", d))) * w(p + "norm2", d)
        y = gelu_tanh(lin(x, w(p + "side.gate", n, d))) * side[..., i * n: (i + 1) * n]
        x = x + unit(lin(y, w(p + "side.proj", d, n))) * w(p + "side.norm", d)
    return unit(x) * w("final.norm", d), lambda x: cap * torch.tanh(lin(x, w("head", VOCAB, d)) / cap)


def plain_tagulix(c, w, rows):
    d, streams, m_res = c["width"], c["streams"], c["residual_mult"]

    def window(x, p, m):
        h, g, dk = m["heads"], m["kv_heads"], m["dim"]
        q, k = (unit(rotate(heads_of(lin(x, w(p + s, n * dk, d), w(f"{p}{s}.b", n * dk)), n), m["rot"], True)) for s, n in (("q", h), ("k", g)))
        y = attend(q, k, heads_of(lin(x, w(p + "v", g * dk, d), w(p + "v.b", g * dk)), g), m["scale"], m["mask"]["size"])
        return lin(y.flatten(2), w(p + "o", d, h * dk), w(p + "o.b", d))

    def biased(x, p, m):
        h, g, dk, t = m["heads"], m["kv_heads"], m["dim"], x.shape[1]
        q, k = (unit(heads_of(lin(x, w(p + s, n * dk, d)), n)) * w(f"{p}{s}.norm", dk) for s, n in (("q", h), ("k", g)))
        grow = torch.tensor([1.0 + m["q_temp"]["coef"] * math.log((i + 1) // m["q_temp"]["every"] + 1) for i in range(t)], dtype=x.dtype, device=x.device)
        bias = distance_bias(w(p + "rel", BIAS_ROWS, h), t, m["bias_max"])
        y = attend(q * grow[:, None, None], k, heads_of(lin(x, w(p + "v", g * dk, d)), g), m["scale"], bias=bias, sink=w(p + "sink", h))
        return lin(y.flatten(2), w(p + "o", d, h * dk))

    def decaying(x, p, m):
        h, n = m["heads"], m["heads"] * m["dim"]
        q, k, v = (heads_of(silu(lin(x, w(p + s, n, d))), h) for s in "qkv")
        y = fold(q, k, v, torch.tensor(m["decay"], dtype=x.dtype, device=x.device)[None, None, :, None])
        return lin(unit(y.flatten(2)) * w(p + "norm", n) * torch.sigmoid(lin(x, w(p + "g", n, d))), w(p + "o", d, n))

    def mixture(x, p, f):
        r, ff = f["router"], f["expert"]["ff"]
        n = r["experts"] + r["identity"]
        s = torch.softmax(lin(x, w(p + "router", n, d)), dim=1)
        share = s * choose(s + w(p + "correction", n), lambda g: g.amax(2), r["groups"]["count"], r["groups"]["keep"], r["top"])
        share = share / share.sum(1, keepdim=True) * r["scale"]

        def expert(e, t):
            z = lin(t, w(f"{p}e{e}.up", ff, d))
            return lin(0.5 * z * (1.0 + torch.erf(z / math.sqrt(2.0))), w(f"{p}e{e}.down", d, ff))

        return mix_experts(x, share[:, : r["experts"]], expert) + share[:, r["experts"]:].sum(1, keepdim=True) * x

    def join(x, p, sublayer):
        u = torch.einsum("a,btad->btd", w(p + "in", streams), x)
        return torch.einsum("ac,btad->btcd", w(p + "mix", streams, streams), x) + m_res * w(p + "out", streams)[:, None] * sublayer(u)[:, :, None, :]

    x = w("embed", VOCAB, d)[rows][:, :, None, :].expand(-1, -1, streams, -1)
    for i, layer in enumerate(c["layers"]):
        p, m = f"l{i}.", layer["mixer"]

        def mixer(u):
            h = unit(u) * w(p + "norm1", d)
            if layer["type"] == "attention":
                return window(h, p + "mix.", m)
            return m["left_scale"] * biased(h, p + "mix.left.", m["left"]) + m["right_scale"] * decaying(h, p + "mix.right.", m["right"])

        x = join(x, p + "hc1.", mixer)
        x = join(x, p + "hc2.", lambda u: mixture((unit(u) * w(p + "norm2", d)).flatten(0, 1), p + "mlp.", layer["mlp"]).view_as(u))
    return unit(x.sum(2)) * w("final.norm", d), lambda x: lin(x, w("head", VOCAB, d))


PLAIN = {"gpt2": plain_gpt2, "zirunex": plain_zirunex, "bosenex": plain_bosenex, "zudalorn": plain_zudalorn, "pidodra": plain_pidodra,
         "lagelorn": plain_lagelorn, "tagulix": plain_tagulix}
