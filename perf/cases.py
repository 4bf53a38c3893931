"""The work that the engine's performance is measured on: single layers over prompts (attention in its forms, recurrent
mixers, feed-forwards) and whole passes from a request's arrival to its last token.

``listed()`` names the fixed cases and ``draw(rng)`` makes more of the same ranges; ``prepare`` builds what a program has in
hand before the call (weights, a layer or a model runner, inputs), ``run`` makes one call, ``work`` counts the bytes and
operations that the call cannot do without, ``tolerance`` states how far another correct implementation may be off, and
``exact`` is the same call in plain float64 torch, without this package.

Two families of cases:

* ``what`` = "serve": requests are admitted, their prompts run in steps of up to 2048 tokens, then every request decodes a
  given number of given tokens, and the requests are given back: ``ModelRunner.add_request`` / ``step`` / ``free_request``,
  as the scheduler drives them.  The logits of every step come back.  Each pass is whole, so that it can be repeated.
* everything else is one layer part over a step's tokens, ``lengths`` giving every request's share ("2048", "1024,700,90",
  "1*64" for 64 requests with one token each).  Recurrent parts carry their state on from pass to pass, as a prompt's
  portions do; the state comes back beside the output.

The sizes are those of ``bench.py``: the Qwen3 0.6B and 8B widths, and its layer sizes of the other architectures.
"""

from __future__ import annotations

import math
import zlib

import torch

F64 = torch.float64
EPS = 1e-6
PAGE = 16
STEP_TOKENS = 2048          # the most tokens a prompt step brings

# Heads, key/value heads and feed-forward widths by model width.
HEADS = {1024: (16, 8), 2048: (16, 8), 4096: (32, 8)}
FF = {1024: 3072, 2048: 6144, 4096: 12288}


# ------------------------------------------------------------------------------------------------- cases
def listed() -> list[dict]:
    return [
        # One user's chat turn on the small model: a short prompt, then single tokens. Latency and launches count.
        dict(name="serve one request", what="serve", model="qwen3", width=1024, layers=4, vocab=151936, rows=1, prompt=300, new=24),
        # The benchmark's batch: eight requests with contexts of thousands, decoded together.
        dict(name="serve eight requests", what="serve", model="qwen3", width=1024, layers=4, vocab=32768, rows=8, prompt=2600, new=40),
        # The same pass on a model that alternates gated linear attention with attention and Mamba-2 side by side.
        dict(name="serve recurrent", what="serve", model="legelix", width=2048, layers=2, vocab=32768, rows=12, prompt=150, new=24),
        # A prompt step's attention layer at the 8B width: three requests' portions of unequal, odd lengths.
        dict(name="attention ragged", what="attention", width=4096, lengths="1531,500,17", dtype="bfloat16"),
        # The true 32-bit engine, used to check models: an attention layer over one prompt.
        dict(name="attention float32", what="attention", width=1024, lengths="700", dtype="float32"),
        # The dense feed-forward at the 8B width, for a step with a few hundred tokens.
        dict(name="feed-forward", what="feed_forward", width=4096, lengths="333", dtype="bfloat16"),
        # Attention and Mamba-2 side by side on one input: a whole prompt and the tail of another.
        dict(name="parallel mixers", what="parallel", width=2048, lengths="2048,77", dtype="bfloat16"),
        # The gated delta rule over a prompt.
        dict(name="delta rule", what="delta", width=2048, lengths="2048", dtype="bfloat16"),
        # Retention over two prompts' portions at the largest width.
        dict(name="retention", what="retention", width=4096, lengths="1500,548", dtype="bfloat16"),
        # Attention over a window that keeps the first tokens, with one in the softmax's denominator: a long prompt.
        dict(name="kept window", what="kept_window", width=2048, lengths="3000", dtype="bfloat16"),
        # Latent attention (a position keeps one row of 160 values for all heads) over a prompt.
        dict(name="latent attention", what="latent", width=2048, lengths="2048", dtype="bfloat16"),
        # A routed feed-forward, 16 experts of which a token takes 4.
        dict(name="routed", what="routed", width=2048, lengths="777", dtype="bfloat16"),
    ]


LAYERS = ("attention", "feed_forward", "gla", "parallel", "delta", "retention", "kept_window", "latent", "routed")


def _spread(rng, low: int, high: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng) -> dict:
    if rng.random() < 0.2:
        if rng.random() < 0.3:
            return dict(what="serve", model="legelix", width=2048, layers=2, vocab=32768, rows=rng.randint(1, 16),
                        prompt=_spread(rng, 8, 200), new=rng.randint(8, 32))
        rows = _spread(rng, 1, 16)
        return dict(what="serve", model="qwen3", width=1024, layers=rng.randint(2, 4), vocab=32768, rows=rows,
                    prompt=_spread(rng, 20, min(4000, 20000 // rows)), new=rng.randint(8, 40))
    what = rng.choice(LAYERS)
    widths = {"attention": (1024, 2048, 4096), "feed_forward": (1024, 2048, 4096), "parallel": (2048,), "gla": (2048,), "routed": (1024, 2048)}
    width = rng.choice(widths.get(what, (1024, 2048, 4096) if what == "retention" else (2048,)))
    dtype = "float32" if what in ("attention", "feed_forward") and width == 1024 and rng.random() < 0.5 else "bfloat16"
    if rng.random() < 0.2:                                   # a decode step's share of the layer
        lengths = f"1*{_spread(rng, 1, 64)}"
    else:
        most = 900 if dtype == "float32" else 2100
        tokens, cuts = _spread(rng, 32, most), rng.choice((1, 1, 2, 3))
        parts = []
        for left in range(cuts, 1, -1):
            parts.append(max(1, min(tokens - left, int(tokens * rng.uniform(0.1, 0.9)))))
            tokens -= parts[-1]
        lengths = ",".join(str(n) for n in (*parts, max(1, tokens)))
    return dict(what=what, width=width, lengths=lengths, dtype=dtype)


def lengths_of(case: dict) -> list[int]:
    if "*" in case["lengths"]:
        n, count = case["lengths"].split("*")
        return [int(n)] * int(count)
    return [int(n) for n in case["lengths"].split(",")]


# ------------------------------------------------------------------------------------- sizes of the layers
def _rot_scaling_llama() -> dict:
    return {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}


def _legelix(width: int, layers: int, vocab: int) -> dict:
    heads, kv = HEADS[width]
    gla = {"type": "gla", "mixer": dict(tau=16.0, heads=8, dim=128, vdim=256), "mlp": {"kind": "dense", "ff": FF[width]}}
    left = dict(heads=heads, kv_heads=kv, dim=128, vdim=128, scale=128 ** -0.5, mask={"size": 1024},
                rot={"base": 500000.0, "dims": 128, "scaling": _rot_scaling_llama()})
    right = dict(heads=32, vdim=64, state=128, groups=2, conv=4, norm_groups=2)
    both = {"type": "parallel", "mlp": {"kind": "dense", "ff": FF[width]},
            "mixer": {"left": left, "right": right, "left_scale": 1.0, "right_scale": 1.0}}
    return dict(vocab=vocab, width=width, layers=tuple([gla, both][i % 2] for i in range(layers)), norm_eps=EPS, residual_mult=0.5,
                decay_rank=16)


def _rizovik_delta(width: int) -> dict:
    heads, kv = HEADS[width]
    return dict(heads=heads, kv_heads=kv, dim=128, vdim=128, conv=4)


def _tedulorn_retention(width: int) -> dict:
    heads = {1024: 8, 2048: 16, 4096: 32}[width]
    return dict(heads=heads, dim=128, vdim=128, rot={"base": 10000.0, "dims": 128},
                decay=[1.0 - 2.0 ** -(5 + h % 8) for h in range(heads)])


def _tedulorn_window(width: int) -> dict:
    heads, kv = HEADS[width]
    return dict(heads=heads, kv_heads=kv, dim=128, vdim=128, scale=128 ** -0.5, v_mix=False, rot={"base": 150000.0, "dims": 64},
                mask={"size": 1024, "keep_first": 64})


def _fekotar_latent(width: int) -> dict:
    return dict(heads=16, dim=128, rot_dim=32, vdim=128, kv_rank=128, q_rank=768, scale=160 ** -0.5,
                rot={"base": 10000.0, "dims": 32, "scaling": {"factor": 40.0, "original": 4096, "fast": 32.0, "slow": 1.0}})


def _gefovik_routed(width: int) -> dict:
    return {"kind": "moe", "expert": {"ff": FF[width] // 4}, "router": {"experts": 16, "identity": 2, "top": 4}}


def _config(case: dict):
    """The configuration of the model that the case's layer belongs to (one layer, but for whole passes)."""
    from zephyr_b200.config import FekotarConfig, GefovikConfig, LegelixConfig, Qwen3Config, RizovikConfig, TedulornConfig

    what, width = case["what"], case["width"]
    if what in ("attention", "feed_forward") or case.get("model") == "qwen3":
        heads, kv = HEADS[width]
        return Qwen3Config(vocab_size=case.get("vocab", 256), hidden_size=width, intermediate_size=FF[width],
                           num_hidden_layers=case.get("layers", 1), num_attention_heads=heads, num_key_value_heads=kv, head_dim=128,
                           max_position_embeddings=4352, rms_norm_eps=EPS, rope_theta=1000000.0, tie_word_embeddings=True)
    if case.get("model") == "legelix":
        return LegelixConfig(**_legelix(width, case["layers"], case["vocab"]))
    if what in ("gla", "parallel"):
        both = _legelix(width, 2, 256)
        return LegelixConfig(**dict(both, layers=(both["layers"][0 if what == "gla" else 1],)))
    if what == "delta":
        return RizovikConfig(vocab=256, width=width, norm_eps=EPS, residual_mult=0.6,
                             layers=({"type": "delta", "mixer": _rizovik_delta(width), "mlp": None},))
    if what in ("retention", "kept_window"):
        kind = "retention" if what == "retention" else "attention"
        mixer = _tedulorn_retention(width) if what == "retention" else _tedulorn_window(width)
        return TedulornConfig(vocab=256, width=width, norm_eps=EPS, embedding_scale=8.0, side_dim=0,
                              layers=({"type": kind, "mixer": mixer, "mlp": None},))
    if what == "latent":
        return FekotarConfig(vocab=256, width=width, norm_eps=EPS, logit_scale=0.25, bigram=None,
                             layers=({"type": "latent_attention", "mixer": _fekotar_latent(width), "mlp": None},))
    heads, kv = HEADS[width]
    keyed = dict(heads=heads, kv_heads=kv, dim=128, vdim=128, scale=128 ** -0.5, softcap=50.0)
    return GefovikConfig(vocab=256, width=width, norm_eps=EPS, embedding_scale=1.0,
                         layers=({"type": "attention", "mixer": keyed, "mlp": _gefovik_routed(width)},))


# --------------------------------------------------------------------------------------- inputs and weights
def _generator(seed: int, name: str, device="cuda") -> torch.Generator:
    generator = torch.Generator(device=device)
    generator.manual_seed((int(seed) * 1000003 + zlib.crc32(name.encode())) & (2 ** 62 - 1))
    return generator


def _uniform(shape, low: float, high: float, generator) -> torch.Tensor:
    return torch.rand(shape, generator=generator, device=generator.device) * (high - low) + low


def _tensor(seed: int, name: str, shape, role: str, dtype: torch.dtype) -> torch.Tensor:
    """Matrices N(0, 0.02), norm scales around one, shifts around zero; the recurrences' rates as such models start them:
    rates exp(A_log) in 1..16, step sizes softplus(dt_bias) in 0.001..0.1."""
    g = _generator(seed, name)
    if name.endswith("A_log"):
        values = _uniform(shape, 1.0, 16.0, g).log()
    elif name.endswith("dt_bias"):
        step = _uniform(shape, math.log(1e-3), math.log(1e-1), g).exp()
        values = step + torch.log(-torch.expm1(-step))
    else:
        values = torch.randn(shape, generator=g, device="cuda") * (0.01 if role == "norm" else 0.02) + (1.0 if role == "norm" else 0.0)
    return values.to(dtype)


class _Weights:
    """A weight store of seeded tensors."""

    def __init__(self, expected: dict, seed: int, dtype: torch.dtype):
        self.expected, self.seed, self.kind = expected, seed, dtype

    def names(self):
        return tuple(self.expected)

    def shape(self, name):
        return tuple(self.expected[name].shape)

    def dtype(self, name):
        return self.kind

    def read(self, name):
        return _tensor(self.seed, name, self.shape(name), self.expected[name].role, self.kind)


def _dtype(case: dict) -> torch.dtype:
    return getattr(torch, case.get("dtype", "bfloat16"))


def _hidden(case: dict, seed: int) -> torch.Tensor:
    """What a norm hands to a layer: rows of unit root mean square."""
    return torch.randn((sum(lengths_of(case)), case["width"]), generator=_generator(seed, "hidden"), device="cuda").to(_dtype(case))


def _tokens(case: dict, seed: int) -> list[list[int]]:
    """Every request's prompt and the tokens that it decodes."""
    g = _generator(seed, "tokens", "cpu")
    return torch.randint(case["vocab"], (case["rows"], case["prompt"] + case["new"]), generator=g).tolist()


def _prompt_steps(case: dict, tokens: list[list[int]]) -> list[list[tuple[int, int, int]]]:
    """The prompts cut into steps of up to ``STEP_TOKENS`` tokens: (request, first token, one past the last)."""
    steps, step, room = [], [], STEP_TOKENS
    for row in range(case["rows"]):
        at = 0
        while at < case["prompt"]:
            count = min(room, case["prompt"] - at)
            step.append((row, at, at + count))
            at, room = at + count, room - count
            if room == 0:
                steps.append(step)
                step, room = [], STEP_TOKENS
    return steps + ([step] if step else [])


# --------------------------------------------------------------------------------------------- prepare, run
def prepare(case: dict, seed: int) -> dict:
    from zephyr_b200.engine import ModelRunner, StepEntry
    from zephyr_b200.parts import Model, expected_weights

    spec = _config(case).to_model_spec()
    model = Model.load(spec, _Weights(expected_weights(spec), seed, _dtype(case)), _dtype(case), "cuda")
    if case["what"] == "serve":
        longest = case["prompt"] + case["new"]
        runner = ModelRunner(model, PAGE, case["rows"] * -(-longest // PAGE) + 1, case["rows"], max_seq_len=longest)
        tokens = _tokens(case, seed)
        steps = [[StepEntry(row, tokens[row][a:b], (b - a - 1,) if b == case["prompt"] else ()) for row, a, b in step]
                 for step in _prompt_steps(case, tokens)]
        steps += [[StepEntry(row, tokens[row][at:at + 1], (0,)) for row in range(case["rows"])]
                  for at in range(case["prompt"], longest)]
        return {"what": "serve", "runner": runner, "rows": case["rows"], "reserve": longest, "steps": steps}
    lengths, x = lengths_of(case), _hidden(case, seed)
    if case["what"] in ("feed_forward", "routed"):
        return {"what": "feed_forward", "layer": model.layers[0].feed_forward, "x": x}
    pages = sum(-(-n // PAGE) for n in lengths) + 1
    runner = ModelRunner(model, PAGE, pages, len(lengths))
    for row, n in enumerate(lengths):
        runner.add_request(row, n)
    ctx = runner.build_context([StepEntry(row, [0] * n) for row, n in enumerate(lengths)])
    call = spec.run_order[0]
    state = {"gla": call.cache, "delta": call.cache, "retention": call.cache, "parallel": call.caches[-1]}.get(case["what"])
    return {"what": "mixer", "layer": model.layers[0].mixer, "x": x, "ctx": ctx, "call": call, "runner": runner,
            "state": runner.storage[state] if state is not None else None}


@torch.no_grad()
def run(state: dict):
    if state["what"] == "serve":
        runner, out = state["runner"], []
        for row in range(state["rows"]):
            runner.add_request(row, state["reserve"])
        for entries in state["steps"]:
            logits = runner.step(entries)
            if len(logits):
                out.append(logits.clone())        # a decode step's logits belong to its graph
        for row in range(state["rows"]):
            runner.free_request(row)
        return out
    if state["what"] == "feed_forward":
        return state["layer"].forward(state["x"])
    out = state["layer"].forward(state["x"], state["ctx"], state["call"])
    return out if state["state"] is None else {"out": out, "state": state["state"]}


# ------------------------------------------------------------------------------------------------- work
def _matrix_work(rows: int, shapes, width_bytes: int) -> tuple[float, float]:
    """(weight bytes, FLOPs) of products of ``rows`` rows with [n, k] matrices."""
    elements = sum(n * k for n, k in shapes)
    return float(elements * width_bytes), 2.0 * rows * elements


def _seen(n: int, window: int = 0, keep: int = 0, chunk: int = 0) -> float:
    """Pairs of a query and a key that it sees, over n tokens from position 0."""
    i = torch.arange(n, dtype=F64)
    if chunk:
        return float((i % chunk + 1).sum())
    if window:
        return float((torch.clamp(i + 1, max=window) + torch.clamp(i + 1 - window, min=0, max=keep)).sum())
    return n * (n + 1) / 2.0


def _mixer_shapes(what: str, width: int):
    heads, kv = HEADS[width]
    if what in ("attention", "kept_window"):
        gate = heads if what == "kept_window" else 0
        return [((heads + 2 * kv) * 128 + gate, width), (width, heads * 128)]
    if what == "gla":
        return [(8 * 128 * 2 + 8 * 256 * 2 + 16, width), (8 * 128, 16), (width, 8 * 256)]
    if what == "mamba":
        return [(2 * 2048 + 2 * 256 + 32, width), (width, 2048)]
    if what == "delta":
        return [((2 * kv + 2 * heads) * 128 + 2 * heads, width), (width, heads * 128)]
    if what == "retention":
        n = {1024: 8, 2048: 16, 4096: 32}[width]
        return [(4 * n * 128, width), (width, n * 128)]
    m = _fekotar_latent(width)                                                    # latent
    return [(m["q_rank"] + 160 + 16 * 128, width), (16 * 160, m["q_rank"]), (2 * 16 * 128, 128), (width, 16 * 128)]


def _mixer_flops(what: str, width: int, lengths) -> tuple[float, float]:
    """(FLOPs between the projections, state bytes read and written)."""
    heads, _ = HEADS[width]
    tokens = sum(lengths)
    if what == "attention":
        return sum(4.0 * heads * 128 * _seen(n) for n in lengths), 0.0
    if what == "kept_window":
        return sum(4.0 * heads * 128 * _seen(n, 1024, 64) for n in lengths), 0.0
    if what == "latent":                # keys and values of all heads from one row of 160 (values: its first 128)
        return sum(2.0 * 16 * (160 + 128) * _seen(n) for n in lengths), 0.0
    if what == "gla":
        return 5.0 * tokens * 8 * 128 * 256, 8.0 * len(lengths) * 8 * 128 * 256
    if what == "mamba":
        return 5.0 * tokens * 32 * 128 * 64, 8.0 * len(lengths) * (32 * 128 * 64 + 3 * 2560)
    if what == "delta":
        return 8.0 * tokens * heads * 128 * 128, 8.0 * len(lengths) * (heads * 128 * 128 + 3 * (HEADS[width][1] * 2 + heads) * 128)
    n = {1024: 8, 2048: 16, 4096: 32}[width]                                       # retention
    return 5.0 * tokens * n * 128 * 128, 8.0 * len(lengths) * n * 128 * 128


def _layer_work(what: str, width: int, lengths, size: int) -> tuple[float, float]:
    """(bytes without inputs and outputs, FLOPs) of one mixer over a step's tokens."""
    if what == "parallel":
        left, right = _layer_work("attention", width, lengths, size), _layer_work("mamba", width, lengths, size)
        heads, _ = HEADS[width]
        chunked = sum(4.0 * heads * 128 * (_seen(n, chunk=1024) - _seen(n)) for n in lengths)
        return left[0] + right[0], left[1] + right[1] + chunked
    weights, products = _matrix_work(sum(lengths), _mixer_shapes(what, width), size)
    flops, state = _mixer_flops(what, width, lengths)
    return weights + state, products + flops


def work(case: dict) -> dict:
    width = case["width"]
    size = 4 if case.get("dtype") == "float32" else 2
    if case["what"] == "serve":
        return _serve_work(case)
    lengths = lengths_of(case)
    tokens = sum(lengths)
    rows = 2.0 * tokens * width * size                                  # the input and the output
    if case["what"] == "feed_forward":
        weights, flops = _matrix_work(tokens, [(2 * FF[width], width), (width, FF[width])], size)
    elif case["what"] == "routed":
        # Every expert's matrices are read once as soon as some token takes it; two outputs of 18 cost nothing.
        ff, hit = FF[width] // 4, 16 * (1.0 - (1.0 - 4 / 18) ** tokens)
        one, taken = _matrix_work(tokens, [(2 * ff, width), (width, ff)], size)
        weights, flops = hit * one, 4 * 16 / 18 * taken + 2.0 * tokens * 18 * width
    else:
        weights, flops = _layer_work(case["what"], width, lengths, size)
    return {"bytes": weights + rows, "flops": flops}


def _serve_work(case: dict) -> dict:
    """Every step reads every weight once, and a decode step the caches of its requests besides."""
    width, rows, layers, vocab = case["width"], case["rows"], case["layers"], case["vocab"]
    heads, kv = HEADS[width]
    total, flops = 0.0, 0.0
    head = 2.0 * vocab * width
    ff = [(2 * FF[width], width), (width, FF[width])]
    kinds = ["attention"] * layers if case["model"] == "qwen3" else [("gla", "parallel")[i % 2] for i in range(layers)]
    steps = [([b - a for _, a, b in step], [a for _, a, _ in step], sum(b == case["prompt"] for _, _, b in step))
             for step in _prompt_steps(case, [])]
    steps += [([1] * rows, [at] * rows, rows) for at in range(case["prompt"], case["prompt"] + case["new"])]
    for lengths, before, wanted in steps:
        tokens = sum(lengths)
        for kind in kinds:
            more, products = _matrix_work(tokens, ff, 2)
            own, inner = _layer_work(kind, width, lengths, 2)
            total, flops = total + more + own, flops + products + inner
            if kind != "gla":
                # keys and values of the positions before the step (a chunk's at most), and their scores
                old = [b if kind == "attention" else b % 1024 for b in before]
                total += sum(old) * 2.0 * kv * 128 * 2
                flops += sum(4.0 * heads * 128 * o * n for o, n in zip(old, lengths))
        total, flops = total + (head if wanted else 0.0) + 4.0 * wanted * vocab, flops + 2.0 * wanted * vocab * width
    return {"bytes": total, "flops": flops}


# ------------------------------------------------------------------------------------------------ tolerance
def tolerance(case: dict):
    if case.get("dtype") == "float32":
        return {"rel": 1e-5, "max": 1e-4}          # 2e-6 from float64
    # A layer is 0.002 to 0.004 from float64 with bfloat16 operands and outputs; whole passes over two to four layers 0.01
    # in every logit, a rounding in one layer travelling through those behind it.
    return {"rel": 2.5e-2 if case["what"] == "serve" else 1e-2, "max": 0.3}


# ------------------------------------------------------------------------------------------- plain float64
def _unit(x: torch.Tensor) -> torch.Tensor:
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS)


def _silu(x: torch.Tensor) -> torch.Tensor:
    return x * torch.sigmoid(x)


def _rotate_halves(x: torch.Tensor, freqs: torch.Tensor, mult: float = 1.0) -> torch.Tensor:
    """x [T, heads, d]: value i turns with value i + len(freqs) by position * freqs[i]; what lies beyond stays."""
    half = len(freqs)
    angle = (torch.arange(x.shape[0], dtype=F64, device=x.device)[:, None] * freqs)[:, None, :]
    c, s = torch.cos(angle) * mult, torch.sin(angle) * mult
    a, b = x[..., :half], x[..., half:2 * half]
    return torch.cat([a * c - b * s, b * c + a * s, x[..., 2 * half:]], dim=-1)


def _rotate_pairs(x: torch.Tensor, freqs: torch.Tensor) -> torch.Tensor:
    angle = (torch.arange(x.shape[0], dtype=F64, device=x.device)[:, None] * freqs)[:, None, :]
    c, s = torch.cos(angle), torch.sin(angle)
    a, b = x[..., 0::2], x[..., 1::2]
    return torch.stack([a * c - b * s, b * c + a * s], dim=-1).flatten(-2)


def _freqs(base: float, dims: int) -> torch.Tensor:
    return torch.tensor([base ** (-2.0 * i / dims) for i in range(dims // 2)], dtype=F64, device="cuda")


def _freqs_llama(base: float, dims: int, sc: dict) -> torch.Tensor:
    out = []
    for f in _freqs(base, dims).tolist():
        wave = 2.0 * math.pi / f
        if wave > sc["original"] / sc["low"]:
            f /= sc["factor"]
        elif wave >= sc["original"] / sc["high"]:
            s = (sc["original"] / wave - sc["low"]) / (sc["high"] - sc["low"])
            f = (1.0 - s) * f / sc["factor"] + s * f
        out.append(f)
    return torch.tensor(out, dtype=F64, device="cuda")


def _freqs_yarn(base: float, dims: int, sc: dict) -> tuple[torch.Tensor, float]:
    def at(turns):
        return dims * math.log(sc["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))
    low, high = max(math.floor(at(sc["fast"])), 0), min(math.ceil(at(sc["slow"])), dims - 1)
    ramp = torch.clamp((torch.arange(dims // 2, dtype=F64, device="cuda") - low) / max(high - low, 0.001), 0.0, 1.0)
    f = _freqs(base, dims)
    return f / sc["factor"] * ramp + f * (1.0 - ramp), 0.1 * math.log(sc["factor"]) + 1.0


def _attend(q, k, v, scale: float, window: int = 0, keep: int = 0, chunk: int = 0, sinks=None) -> torch.Tensor:
    """q [T, H, d] over k [T, G, d], v [T, G, dv], causal, within a window or a chunk; ``sinks`` [H] join the denominators."""
    T, H, _ = q.shape
    i, j = torch.arange(T, device=q.device)[:, None], torch.arange(T, device=q.device)[None, :]
    seen = j <= i
    if window:
        seen = seen & ((i - j < window) | (j < keep))
    if chunk:
        seen = seen & (i // chunk == j // chunk)
    out = []
    for h in range(H):
        g = h // (H // k.shape[1])
        score = (q[:, h] @ k[:, g].T * scale).masked_fill(~seen, -math.inf)
        if sinks is not None:
            score = torch.cat([score, sinks[h].expand(T, 1)], dim=1)
        p = torch.softmax(score, dim=-1)
        out.append(p[:, :T] @ v[:, g])
    return torch.stack(out, dim=1)


def _plain_attention(h, w, prefix, width):
    heads, kv = HEADS[width]
    T = h.shape[0]
    q, k, v = ((h @ w[f"{prefix}.{n}_proj.weight"].T).view(T, -1, 128) for n in "qkv")
    q, k = _unit(q) * w[f"{prefix}.q_norm.weight"], _unit(k) * w[f"{prefix}.k_norm.weight"]
    f = _freqs(1000000.0, 128)
    out = _attend(_rotate_halves(q, f), _rotate_halves(k, f), v, 128 ** -0.5)
    return out.reshape(T, -1) @ w[f"{prefix}.o_proj.weight"].T


def _plain_kept_window(h, w, prefix, width):
    m, T = _tedulorn_window(width), h.shape[0]
    q, k, v = ((h @ w[f"{prefix}.{n}"].T).view(T, -1, 128) for n in "qkv")
    f = _freqs(m["rot"]["base"], m["rot"]["dims"])
    q, k = (_rotate_halves(_unit(x) * w[f"{prefix}.{n}.norm"], f) for x, n in ((q, "q"), (k, "k")))
    out = _attend(q, k, v, m["scale"], m["mask"]["size"], m["mask"]["keep_first"], sinks=torch.zeros(m["heads"], dtype=F64, device=h.device))
    return (out * torch.sigmoid(h @ w[f"{prefix}.g"].T).unsqueeze(-1)).reshape(T, -1) @ w[f"{prefix}.o"].T


def _plain_latent(h, w, prefix, width):
    m, T = _fekotar_latent(width), h.shape[0]
    rank = m["kv_rank"]
    q = ((_unit(h @ w[f"{prefix}.dq"].T) * w[f"{prefix}.dq.norm"]) @ w[f"{prefix}.uq"].T).view(T, m["heads"], -1)
    down = h @ w[f"{prefix}.dkv"].T
    c = _unit(down[:, :rank]) * w[f"{prefix}.dkv.norm"]
    k, v = (c @ w[f"{prefix}.uk"].T).view(T, m["heads"], -1), (c @ w[f"{prefix}.uv"].T).view(T, m["heads"], -1)
    f, mult = _freqs_yarn(m["rot"]["base"], m["rot_dim"], m["rot"]["scaling"])
    turned = _rotate_halves(down[:, rank:].unsqueeze(1), f, mult).expand(T, m["heads"], m["rot_dim"])
    q = torch.cat([q[..., :m["dim"]], _rotate_halves(q[..., m["dim"]:], f, mult)], dim=-1)
    out = _attend(q, torch.cat([k, turned], dim=-1), v, m["scale"]).reshape(T, -1)
    return (out * torch.sigmoid(h @ w[f"{prefix}.g"].T)) @ w[f"{prefix}.o"].T


def _scan(q, k, v, decay):
    """S <- decay S + k v^T, o = S^T q per head; q, k [T, H, d], v [T, H, dv], decay [T, H, d or 1].  (o, the last S)"""
    S = torch.zeros(k.shape[1], k.shape[2], v.shape[2], dtype=F64, device=k.device)
    out = torch.empty_like(v)
    for t in range(len(v)):
        S = torch.addcmul(S * decay[t].unsqueeze(-1), k[t].unsqueeze(-1), v[t].unsqueeze(1))
        out[t] = torch.bmm(q[t].unsqueeze(1), S).squeeze(1)
    return out, S


def _plain_gla(h, w, prefix, width):
    T = h.shape[0]
    q, k = (h @ w[f"{prefix}.q"].T).view(T, 8, 128) * 128 ** -0.5, (h @ w[f"{prefix}.k"].T).view(T, 8, 128)
    v = (h @ w[f"{prefix}.v"].T).view(T, 8, 256)
    z = (h @ w[f"{prefix}.a1"].T) @ w[f"{prefix}.a2"].T + w[f"{prefix}.a2.b"]
    o, S = _scan(q, k, v, torch.exp(torch.nn.functional.logsigmoid(z) / 16.0).view(T, 8, 128))
    o = (_unit(o) * w[f"{prefix}.norm"]).reshape(T, -1)
    return (o * _silu(h @ w[f"{prefix}.g"].T)) @ w[f"{prefix}.o"].T, S.reshape(-1)


def _plain_retention(h, w, prefix, width):
    m, T = _tedulorn_retention(width), h.shape[0]
    q, k, v = ((h @ w[f"{prefix}.{n}"].T).view(T, -1, 128) for n in "qkv")
    f = _freqs(m["rot"]["base"], m["rot"]["dims"])
    q, k = _rotate_halves(q, f), _rotate_halves(k, f) * m["dim"] ** -0.5
    decay = torch.tensor(m["decay"], dtype=F64, device=h.device).view(1, -1, 1).expand(T, -1, 1)
    o, S = _scan(q, k, v, decay)
    return (_unit(o).reshape(T, -1) * _silu(h @ w[f"{prefix}.g"].T)) @ w[f"{prefix}.o"].T, S.reshape(-1)


def _convolve(x, taps):
    """Causal, zeros before the start: the last column of ``taps`` weighs the present token."""
    n = taps.shape[1]
    padded = torch.cat([x.new_zeros(n - 1, x.shape[1]), x])
    return sum(padded[j:j + len(x)] * taps[:, j] for j in range(n)), padded[len(padded) - n + 1:].reshape(-1)


def _plain_mamba(h, w, prefix, width):
    T, inner, H, N, groups = h.shape[0], 2048, 32, 128, 2
    projected = h @ w[f"{prefix}.in"].T
    z, xbc, dt = projected[:, :inner], projected[:, inner:2 * inner + 2 * groups * N], projected[:, 2 * inner + 2 * groups * N:]
    mixed, last = _convolve(xbc, w[f"{prefix}.conv"])
    mixed = _silu(mixed + w[f"{prefix}.conv.b"])
    x = mixed[:, :inner].view(T, H, -1)
    B, C = (part.reshape(T, groups, N).repeat_interleave(H // groups, dim=1) for part in mixed[:, inner:].split(groups * N, dim=1))
    dt = torch.nn.functional.softplus(dt + w[f"{prefix}.dt_bias"])
    decay = torch.exp(-torch.exp(w[f"{prefix}.A_log"]) * dt).unsqueeze(-1)
    o, S = _scan(C, B * dt.unsqueeze(-1), x, decay)
    y = (o + w[f"{prefix}.D"][:, None] * x).reshape(T, inner) * _silu(z)
    y = _unit(y.view(T, 2, -1)).reshape(T, inner) * w[f"{prefix}.norm"]
    return y @ w[f"{prefix}.o"].T, torch.cat([S.reshape(-1), last])


def _plain_parallel(h, w, prefix, width):
    left, T = f"{prefix}.left", h.shape[0]
    q, k, v = ((h @ w[f"{left}.{n}"].T + w[f"{left}.{n}.b"]).view(T, -1, 128) for n in "qkv")
    f = _freqs_llama(500000.0, 128, _rot_scaling_llama())
    q, k = (_rotate_pairs(_unit(x) * w[f"{left}.{n}.norm"], f) for x, n in ((q, "q"), (k, "k")))
    out = _attend(q, k, v, 128 ** -0.5, chunk=1024, sinks=w[f"{left}.sink"]).reshape(T, -1)
    mamba, state = _plain_mamba(h, w, f"{prefix}.right", width)
    return out @ w[f"{left}.o"].T + w[f"{left}.o.b"] + mamba, state


def _plain_delta(h, w, prefix, width):
    T, (H, G) = h.shape[0], HEADS[width]
    projected, lasts = [], []
    raw = [h @ w[f"{prefix}.{n}"].T for n in "qkv"]
    for x, n in zip(raw, "qkv"):
        mixed, last = _convolve(x, w[f"{prefix}.{n}.conv"])
        projected.append(_silu(mixed))
        lasts.append(last.view(3, -1))
    q, k = ((x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, dim=1)
            for x in (projected[0].view(T, G, 128), projected[1].view(T, G, 128)))
    q, v = q * 128 ** -0.5, projected[2].view(T, H, 128)
    beta = torch.sigmoid(h @ w[f"{prefix}.b"].T)
    decay = torch.exp(-torch.exp(w[f"{prefix}.A_log"]) * torch.nn.functional.softplus(h @ w[f"{prefix}.a"].T + w[f"{prefix}.dt_bias"]))
    S = torch.zeros(H, 128, 128, dtype=F64, device=h.device)
    out = torch.empty_like(v)
    for t in range(T):
        S = S * decay[t].view(H, 1, 1)
        u = beta[t].unsqueeze(-1) * (v[t] - torch.bmm(k[t].unsqueeze(1), S).squeeze(1))
        S = torch.addcmul(S, k[t].unsqueeze(-1), u.unsqueeze(1))
        out[t] = torch.bmm(q[t].unsqueeze(1), S).squeeze(1)
    o = (_unit(out) * w[f"{prefix}.norm"]).reshape(T, -1) * _silu(h @ w[f"{prefix}.g"].T)
    # The slot holds a head's state with a value column's channels together, and the convolution's last inputs.
    return o @ w[f"{prefix}.o"].T, torch.cat([S.transpose(1, 2).reshape(-1), torch.cat(lasts, dim=1).reshape(-1)])


def _plain_gated(h, w, prefix, gate, up, down):
    return (_silu(h @ w[f"{prefix}.{gate}"].T) * (h @ w[f"{prefix}.{up}"].T)) @ w[f"{prefix}.{down}"].T


def _plain_routed(h, w, prefix):
    scores = torch.softmax(h @ w[f"{prefix}.router"].T, dim=-1)
    taken = torch.topk(scores + w[f"{prefix}.correction"], 4, dim=-1).indices
    out = torch.zeros_like(h)
    for e in range(18):
        rows = (taken == e).any(-1).nonzero().view(-1)
        y = h[rows] if e >= 16 else _plain_gated(h[rows], w, f"{prefix}.e{e}", "gate", "up", "down")
        out.index_add_(0, rows, y * scores[rows, e].unsqueeze(-1))
    return out


PLAIN = {"attention": _plain_attention, "kept_window": _plain_kept_window, "latent": _plain_latent, "gla": _plain_gla,
         "retention": _plain_retention, "parallel": _plain_parallel, "delta": _plain_delta}


def _plain_qwen3(case, w, tokens, first):
    x = w["model.embed_tokens.weight"][tokens]
    for i in range(case["layers"]):
        at = f"model.layers.{i}"
        x = x + _plain_attention(_unit(x) * w[f"{at}.input_layernorm.weight"], w, f"{at}.self_attn", case["width"])
        x = x + _plain_gated(_unit(x) * w[f"{at}.post_attention_layernorm.weight"], w, f"{at}.mlp", "gate_proj.weight",
                             "up_proj.weight", "down_proj.weight")
    return (_unit(x[first:]) * w["model.norm.weight"]) @ w["model.embed_tokens.weight"].T


def _plain_legelix(case, w, tokens, first):
    def norm(x, name):
        x = x - x.mean(-1, keepdim=True)
        return _unit(x) * w[name] + w[f"{name}.b"]
    x = w["embed"][tokens]
    for i in range(case["layers"]):
        mixer = (_plain_gla, _plain_parallel)[i % 2]
        mixed, _ = mixer(norm(x, f"l{i}.norm1"), w, f"l{i}.mix", case["width"])
        x = x + 0.5 * norm(mixed, f"l{i}.norm1b")
        x = x + 0.5 * norm(_plain_gated(norm(x, f"l{i}.norm2"), w, f"l{i}.mlp", "gate", "up", "down"), f"l{i}.norm2b")
    return norm(x[first:], "final.norm") @ w["head"].T


@torch.no_grad()
def exact(case: dict, seed: int):
    from zephyr_b200.parts import expected_weights      # the tensors' names and shapes

    decls = expected_weights(_config(case).to_model_spec())
    w = {name: _tensor(seed, name, decl.shape, decl.role, _dtype(case)).to(F64) for name, decl in decls.items()}
    if case["what"] == "serve":
        plain = _plain_qwen3 if case["model"] == "qwen3" else _plain_legelix
        logits = [plain(case, w, torch.tensor(row, device="cuda"), case["prompt"] - 1) for row in _tokens(case, seed)]
        # What comes back: the prompt steps' logits in the order in which the prompts end, then every decode step's.
        out = []
        for step in _prompt_steps(case, []):
            ended = [row for row, _, b in step if b == case["prompt"]]
            if ended:
                out.append(torch.stack([logits[row][0] for row in ended]))
        return out + [torch.stack([one[1 + at] for one in logits]) for at in range(case["new"])]
    lengths, x, width = lengths_of(case), _hidden(case, seed).to(F64), case["width"]
    if case["what"] == "feed_forward":
        return _plain_gated(x, w, "model.layers.0.mlp", "gate_proj.weight", "up_proj.weight", "down_proj.weight")
    if case["what"] == "routed":
        return _plain_routed(x, w, "l0.mlp")
    prefix = "model.layers.0.self_attn" if case["what"] == "attention" else "l0.mix"
    got = [PLAIN[case["what"]](rows, w, prefix, width) for rows in x.split(lengths)]
    if not isinstance(got[0], tuple):
        return torch.cat(got)
    return {"out": torch.cat([out for out, _ in got]), "state": torch.stack([state for _, state in got])}
