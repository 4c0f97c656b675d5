"""The work that programs give this engine, as cases that can be timed and checked.

A case is one call, or a few that belong together, of the step function (`ModelRunner.step`): a batch of
decoded tokens, whole prompts, a prompt cut into portions, or decoded tokens beside new prompts, for a
model of the registry or of the design comparison, with seeded random weights.  `listed()` names the
representative ones, `draw()` makes more of the same ranges, `exact()` works the same logits out in
float64 from the models' definitions with plain torch operations.

The weights are random, but scaled as trained ones are where that matters to the values that a
kernel meets: matrices keep the size of what passes them, sublayers add less than the stream holds, decays
and step sizes lie where trained recurrences have them, and every token has experts it clearly prefers (so
that rounding does not choose other experts).
"""

from __future__ import annotations

import hashlib
import math
from typing import Any, Callable, Optional

import torch

from tokensprint_b200 import design_bench
from tokensprint_b200.config.registry import architecture_for, get_model_config
from tokensprint_b200.engine.runner import ModelRunner, StepEntry
from tokensprint_b200.models.api import build_model
from tokensprint_b200.weights.loader import WeightSource

PAGE = 16
BUDGET = 8192  # most tokens of one step, as the engine's scheduler has it by default
DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}
SIZES = {
    "fegetar": (design_bench.fegetar_config, design_bench.SIZES),
    "dazilix": (design_bench.dazilix_config, design_bench.DAZILIX_SIZES),
    "pekunex": (design_bench.pekunex_config, design_bench.PEKUNEX_SIZES),
    "vasosun": (design_bench.vasosun_config, design_bench.VASOSUN_SIZES),
    "mugulorn": (design_bench.mugulorn_config, design_bench.MUGULORN_SIZES),
    "vepevik": (design_bench.vepevik_config, design_bench.VEPEVIK_SIZES),
}


# ---------------------------------------------------------------------------
# the cases


def _case(name: Optional[str], model: str, size: str, *, dtype: str = "bfloat16", decodes: int = 0, context: int = 0, prompts: int = 0,
          prompt: int = 0, portion: int = 0, ragged: bool = False) -> dict[str, Any]:
    """`decodes` requests with about `context` cached tokens bring one token each; `prompts` requests bring
    about `prompt` tokens each, in steps of `portion` tokens if that is not 0; `ragged`: the lengths differ."""
    c = {"model": model, "size": size, "dtype": dtype, "decodes": decodes, "context": context, "prompts": prompts, "prompt": prompt,
         "portion": portion, "ragged": ragged}
    return c if name is None else {"name": name, **c}


def listed() -> list[dict[str, Any]]:
    return [
        # one user of the smallest preset: every launch and every gap shows
        _case("qwen3-0.6b decode 1", "qwen3", "0.6b", decodes=1, context=200),
        # the serving step the engine is quoted on: eight requests, contexts of a thousand tokens
        _case("qwen3-8b decode 8", "qwen3", "8b", decodes=8, context=1024),
        # a small batch of a routed design in the middle of a conversation
        _case("dazilix decode 5", "dazilix", "w2048", decodes=5, context=333, ragged=True),
        # a batch just above the few-row products, requests of all ages
        _case("vepevik decode 33", "vepevik", "w2048", decodes=33, context=1024, ragged=True),
        # a full server: latent attention over many contexts
        _case("fegetar decode 64", "fegetar", "w2048", decodes=64, context=1024),
        # the first token of one long question at the quoted size
        _case("qwen3-8b prompt 2048", "qwen3", "8b", prompts=1, prompt=2048),
        # a replay in float32, the yardstick of every comparison of logits
        _case("qwen3-0.6b float32 prompt 333", "qwen3", "0.6b", dtype="float32", prompts=1, prompt=333),
        # several questions of odd lengths arrive together
        _case("dazilix prompts 7 x 509", "dazilix", "w2048", prompts=7, prompt=509, ragged=True),
        # a prompt longer than a step's budget, state and cache carried from portion to portion
        _case("pekunex prompt 3000 by 1024", "pekunex", "w2048", prompts=1, prompt=3000, portion=1024),
        # continuous batching: running requests and new ones in one step
        _case("vasosun 24 beside 2 x 700", "vasosun", "w2048", decodes=24, context=900, prompts=2, prompt=700, ragged=True),
        # a document as one step, past the attention's window
        _case("mugulorn prompt 8191", "mugulorn", "w2048", prompts=1, prompt=8191),
        # the wider model: more experts, more heads
        _case("vepevik-w4096 prompt 2048", "vepevik", "w4096", prompts=1, prompt=2048),
    ]


def _log_uniform(rng, low: float, high: float) -> int:
    return max(int(low), min(int(high), int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng) -> dict[str, Any]:
    model = rng.choice(["qwen3"] + sorted(SIZES))
    wide = rng.random() < 0.25
    size = ("8b" if wide else "0.6b") if model == "qwen3" else ("w4096" if wide else "w2048")
    dtype = "float32" if not wide and rng.random() < 0.15 else "bfloat16"
    kind = rng.choice(["decode", "decode", "prompt", "prompt", "portions", "mixed"])
    most = 512 if dtype == "float32" else 2048 if model == "qwen3" else 4096  # new tokens of a step
    c = dict(decodes=0, context=0, prompts=0, prompt=0, portion=0)
    if kind in ("decode", "mixed"):
        c["decodes"] = _log_uniform(rng, 1, 8 if dtype == "float32" else 64)
        c["context"] = _log_uniform(rng, 16, 300 if dtype == "float32" else 2048 if c["decodes"] <= 24 else 1024)
    if kind == "prompt":
        c["prompts"] = _log_uniform(rng, 1, 8)
        c["prompt"] = _log_uniform(rng, 16, most / c["prompts"])
    if kind == "portions":
        c["prompts"] = 1
        c["prompt"] = _log_uniform(rng, 256, most)
        c["portion"] = _log_uniform(rng, 100, c["prompt"] / 1.5)
    if kind == "mixed":
        c["prompts"] = rng.randint(1, 4)
        c["prompt"] = _log_uniform(rng, 16, min(most, 2048) / c["prompts"])
    return _case(None, model, size, dtype=dtype, ragged=rng.random() < 0.6, **c)


def _config(case) -> dict[str, Any]:
    if case["model"] == "qwen3":
        return get_model_config("qwen3-" + case["size"]).to_dict()
    make, sizes = SIZES[case["model"]]
    return make(sizes[case["size"]])


def _lengths(count: int, longest: int, ragged: bool) -> list[int]:
    """Equal lengths, or ones spread between two fifths of the longest and the longest."""
    return [max(1, int(longest * (1.0 - 0.6 * ((i * 0.618034) % 1.0)))) if ragged else longest for i in range(count)]


def _spans(case) -> tuple[list[int], list[int]]:
    return _lengths(case["decodes"], case["context"], case["ragged"]), _lengths(case["prompts"], case["prompt"], case["ragged"])


# ---------------------------------------------------------------------------
# weights and tokens


def _generator(seed: int, name: str, device) -> torch.Generator:
    g = torch.Generator(device=device)
    g.manual_seed(int.from_bytes(hashlib.sha256(f"{seed}:{name}".encode()).digest()[:7], "little"))
    return g


class Weights(WeightSource):
    """Seeded random weights, made on the device tensor by tensor; the values depend on the seed and the name only."""

    where = "seeded random weights"

    def __init__(self, config: dict[str, Any], specs, seed: int, compute_dtype: torch.dtype, device="cuda") -> None:
        self.config, self.seed, self.dtype, self.device = config, seed, compute_dtype, torch.device(device)
        self.specs = {s.name: s for s in specs}
        self.qwen = "architecture" not in config
        self.width = config["hidden_size"] if self.qwen else config["width"]
        self.depth = config["num_hidden_layers"] if self.qwen else len(config["layers"])
        routers = [s.shape[0] for n, s in self.specs.items() if n.endswith("mlp.router")]
        self.leaning = None
        if routers:  # directions in the stream along which tokens lean towards experts
            d = torch.randn(max(routers), self.width, generator=_generator(seed, "leaning", self.device), device=self.device)
            self.leaning = d / d.norm(dim=1, keepdim=True)

    def shapes(self):
        return {n: tuple(s.shape) for n, s in self.specs.items()}

    def values(self, name: str) -> torch.Tensor:
        """Float32 (or int32) values of one tensor."""
        spec = self.specs[name]
        g = _generator(self.seed, name, self.device)
        rand = lambda: torch.rand(spec.shape, generator=g, device=self.device)  # noqa: E731
        randn = lambda: torch.randn(spec.shape, generator=g, device=self.device)  # noqa: E731
        last = name.split(".")[-1]
        if last == "router":
            gen = _generator(self.seed, name + ":order", self.device)
            order = torch.randperm(spec.shape[0], generator=gen, device=self.device)
            return 0.25 * self.leaning[order] + 0.002 / math.sqrt(self.width) * randn()
        if spec.role == "vector":
            if last == "A_log":
                return torch.log(1.0 + 15.0 * rand())
            if last == "dt_bias":  # softplus of it between 0.001 and 0.1
                step = torch.exp(math.log(1e-3) + math.log(100.0) * rand())
                return step + torch.log(-torch.expm1(-step))
            if last == "lam":  # a channel keeps between 0.9 and 0.999 of its state
                s = -torch.log(0.9 + 0.099 * rand()) / 8.0
                return torch.log(torch.expm1(s))
            if last.startswith("canon"):
                return 0.1 * randn()
            if last == "conv":
                return 0.5 * randn()
            if last in ("r1", "r2"):
                return 0.05 + 0.45 * rand()
            if last == "vmix":
                return 0.3 + 0.2 * rand()
            if last == "sink":
                return randn()
            if name.endswith("right.f.b"):
                return 3.0 + 3.0 * rand()
            if last == "b" or last == "correction" or name.endswith(("ra.b", "ri.b")):
                return 0.02 * randn()
            if self.config.get("architecture") == "Fegetar" and last in ("norm1", "norm2"):
                return -0.5 + 0.05 * randn()  # stored as the distance from one
            if self.config.get("architecture") == "Fegetar" and name == "final.norm":
                return 0.05 * randn()
            if last in ("norm1b", "norm2b", "ls1", "ls2") or name.endswith("side.norm"):
                return 0.6 * (1.0 + 0.05 * randn())
            return 1.0 + 0.05 * randn()
        if name in ("embed", "model.embed_tokens.weight"):
            x = randn()
            if self.leaning is not None:
                n = self.leaning.shape[0]
                first = torch.randint(0, n, spec.shape[:1], generator=g, device=self.device)
                second = (first + torch.randint(1, n, spec.shape[:1], generator=g, device=self.device)) % n
                x += 8.0 * self.leaning[first] + 6.0 * self.leaning[second]
            return x
        if name == "bigram":
            return 0.3 * randn()
        if name == "side.embed":
            return randn()
        fan_in = spec.shape[-1]
        scale = 1.0 / math.sqrt(fan_in)
        if last in ("o", "down", "proj") or name.endswith(("o_proj.weight", "down_proj.weight")):
            scale *= 1.0 / math.sqrt(self.depth)  # branches add up to about what the embedding brings
        return scale * randn()

    def stored(self, name: str) -> torch.Tensor:
        """The values as the device holds them: matrices in the compute dtype, vectors in float32."""
        x = self.values(name)
        return x.to(self.dtype) if self.specs[name].role == "matrix" else x

    def fetch(self, spec, device, compute_dtype):
        return self.stored(spec.name).contiguous()


def _weights(case, seed: int, specs) -> Weights:
    return Weights(_config(case), specs, seed, DTYPES[case["dtype"]])


def _token_ids(case, seed: int, vocab: int) -> tuple[list[list[int]], list[list[int]]]:
    """Per decoding request its context, one token more and the token to decode; per new request its prompt."""
    contexts, prompts = _spans(case)
    g = torch.Generator().manual_seed(1000003 * seed + 17)
    ids = lambda n: torch.randint(0, vocab, (n,), generator=g).tolist()  # noqa: E731
    return [ids(n + 2) for n in contexts], [ids(n) for n in prompts]


# ---------------------------------------------------------------------------
# what a program has in hand, and one pass


class State:
    runner: ModelRunner
    decodes: list
    prompts: list
    portion: int


def prepare(case, seed: int) -> State:
    config = _config(case)
    typed = get_model_config("qwen3-" + case["size"]) if case["model"] == "qwen3" else architecture_for(config).config_from_dict(config)
    model = build_model(typed, device="cuda", dtype=case["dtype"])
    model.load(_weights(case, seed, model.tensor_specs()))
    contexts, prompts = _token_ids(case, seed, model.spec.vocab_size)
    pages = sum(-(-len(x) // PAGE) + 1 for x in contexts + prompts)
    longest = max(len(x) for x in contexts + prompts)
    runner = ModelRunner(model, page_size=PAGE, num_pages=pages + 4, num_slots=max(1, len(contexts) + len(prompts)), max_num_batched_tokens=BUDGET,
                         enforce_eager=False, max_model_len=max(2048, longest + 8))
    s = State()
    s.runner, s.portion = runner, case["portion"]
    s.decodes, s.prompts = [], prompts
    batch: list[StepEntry] = []
    for i, ids in enumerate(contexts):  # the cached contexts
        rc = runner.cache_manager.admit(("running", i))
        runner.cache_manager.extend(rc, 0, len(ids) - 2)
        if sum(len(e.tokens) for e in batch) + len(ids) - 2 > BUDGET:
            runner.step(batch)
            batch = []
        batch.append(StepEntry(rc, ids[:-2], 0, ()))
        s.decodes.append((rc, ids))
    if batch:
        runner.step(batch)
    if s.decodes:  # a first decode step, which captures the batch's graph as an engine does when it starts
        runner.step([_decode_entry(runner, rc, ids, len(ids) - 2) for rc, ids in s.decodes])
    return s


def _decode_entry(runner: ModelRunner, rc, ids: list[int], at: int) -> StepEntry:
    if rc.num_tokens < at + 1:
        runner.cache_manager.extend(rc, at, at + 1)
    return StepEntry(rc, [ids[at]], at, (0,))


def run(s: State) -> list[torch.Tensor]:
    """One pass: the logits of every decoded token, then of every prompt's last token, as the steps give them."""
    runner = s.runner
    cm = runner.cache_manager
    decoded = [_decode_entry(runner, rc, ids, len(ids) - 1) for rc, ids in s.decodes]
    fresh = [cm.admit(("new", i)) for i in range(len(s.prompts))]
    out = []
    at = 0
    while at == 0 or any(at < len(ids) for ids in s.prompts):
        entries = decoded if at == 0 else []
        stop = at + s.portion if s.portion else BUDGET
        for rc, ids in zip(fresh, s.prompts):
            if at < len(ids):
                end = min(stop, len(ids))
                cm.extend(rc, at, end)
                entries = entries + [StepEntry(rc, ids[at:end], at, (end - at - 1,) if end == len(ids) else ())]
        logits = runner.step(entries)
        if logits.shape[0]:
            out.append(logits)
        at = stop
    for rc in fresh:
        runner.free(rc)
    return out


# ---------------------------------------------------------------------------
# what a pass cannot do without


def _layers(case) -> list[dict[str, Any]]:
    """Per layer run: attention as (heads, score width, value width, cached entries per token, reach), or a
    recurrence as (state entries, operations per entry)."""
    config, rows = _config(case), []
    if case["model"] == "qwen3":
        H, G, d = config["num_attention_heads"], config["num_key_value_heads"], config["head_dim"]
        return [{"attention": (H, d, d, 2 * G * d, None)}] * config["num_hidden_layers"]
    for layer in config["layers"]:
        m, kind = layer["mixer"], layer["type"]
        parts = [("sink", m["left"]), ("memory", m["right"])] if kind == "parallel" else [(kind, m)]
        for kind, m in parts:
            reach = (m.get("mask") or {}).get("size")
            if kind in ("attention", "sink"):
                rows.append({"attention": (m["heads"], m["dim"], m["vdim"], m["kv_heads"] * (m["dim"] + m["vdim"]), reach)})
            elif kind == "latent_attention":  # either form: per head d + r and e, or on the cached rows; the smaller one counts
                rows.append({"attention": (m["heads"], m["dim"] + m["rot_dim"], m["vdim"], m["kv_rank"] + m["rot_dim"], reach)})
            elif kind == "mamba2":
                rows.append({"state": (m["heads"] * m["vdim"] * m["state"], 6)})
            elif kind == "rglru":
                rows.append({"state": (m["width"], 6)})
            elif kind == "memory":
                rows.append({"state": (m["heads"] * m["dim"] * (m["vdim"] + 1), 6)})
            else:
                rows.append({"state": (m["heads"] * m["dim"] * m["vdim"], 8 if "delta" in kind else 6)})
    return rows


def work(case) -> dict[str, float]:
    config = _config(case)
    typed = get_model_config("qwen3-" + case["size"]) if case["model"] == "qwen3" else architecture_for(config).config_from_dict(config)
    spec = architecture_for(typed.to_dict()).build_spec(typed)
    size = torch.empty((), dtype=DTYPES[case["dtype"]]).element_size()
    contexts, prompts = _spans(case)
    spans = [(n + 1, n + 2) for n in contexts] + [(0, n) for n in prompts]  # first position and end of the new tokens
    T, R = sum(e - a for a, e in spans), len(spans)
    flops = bytes_ = 0.0
    vocab_rows = spec.vocab_size
    top, experts = {}, {}
    for i, layer in enumerate(config.get("layers", [])):
        r = (layer.get("mlp") or {}).get("router")
        if r:
            n = r["experts"] + (r.get("identity") or 0)
            top[f"l{i}."], experts[f"l{i}."] = r["top"] * r["experts"] / n, r["experts"]
    for t in spec.tensor_specs():
        n = math.prod(t.shape)
        held = n * (size if t.role == "matrix" else 4)
        if t.name in ("embed", "model.embed_tokens.weight", "bigram", "side.embed"):
            bytes_ += T * t.shape[-1] * size
            if t.name in ("embed", "model.embed_tokens.weight") and spec.lm_head is None:
                flops, bytes_ = flops + 2 * R * n, bytes_ + held
        elif len(t.shape) < 2 or t.shape[-1] <= 8:
            bytes_ += held
        elif t.shape[0] == vocab_rows:
            flops, bytes_ = flops + 2 * R * n, bytes_ + held
        elif ".mlp.e" in t.name:
            p = t.name.split(".")[0] + "."
            share = top[p] / experts[p]
            flops += 2 * T * share * n
            bytes_ += held * (1.0 - (1.0 - share) ** T)
        else:
            flops, bytes_ = flops + 2 * T * n, bytes_ + held
    for row in _layers(case):
        if "attention" in row:
            H, d, e, cached, reach = row["attention"]
            for a, end in spans:
                pairs = sum(min(p + 1, reach) if reach else p + 1 for p in range(a, end))
                flops += 2.0 * pairs * H * (d + e)
                bytes_ += cached * size * (end if reach is None else min(end, reach + end - a))
        else:
            entries, per = row["state"]
            flops += per * T * entries
            bytes_ += 4 * entries * R * 2
    return {"bytes": bytes_ + 4.0 * R * spec.vocab_size, "flops": flops}


def tolerance(case):
    """About four times the distance from `exact` that was measured: 1e-6 to 2e-6 in float32 and 0.002 to 0.005 in
    bfloat16, 0.013 where small branches pass a norm on their way out as well."""
    if case["dtype"] == "float32":
        return {"rel": 1e-5}
    return {"rel": 0.03 if case["model"] == "vasosun" else 0.02, "max": 0.3}


# ---------------------------------------------------------------------------
# the same logits in float64: the models' definitions on whole sequences, no cache


def _unit(x, eps):
    return x / torch.sqrt(x.pow(2).mean(-1, keepdim=True) + eps)


def _gelu(z):
    return torch.nn.functional.gelu(z, approximate="tanh")


_silu, _softplus, _sigmoid = torch.nn.functional.silu, lambda z: torch.logaddexp(z, torch.zeros_like(z)), torch.sigmoid


def _smooth_stretch(base, dims, s):
    i = torch.arange(dims // 2, dtype=torch.float64)
    f = float(base) ** (-2.0 * i / dims)
    if s is None:
        return f, 1.0
    if "low" in s:  # by wavelength: kept, divided, or blended
        turns = s["original"] * f / (2.0 * math.pi)
        blend = ((turns - s["low"]) / (s["high"] - s["low"])).clamp(0.0, 1.0)
        return (1.0 - blend) * f / s["factor"] + blend * f, 1.0
    where = lambda turns: dims * math.log(s["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))  # noqa: E731
    lo, hi = max(math.floor(where(s["fast"])), 0), min(math.ceil(where(s["slow"])), dims - 1)
    ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
    return f / s["factor"] * ramp + f * (1.0 - ramp), 0.1 * math.log(s["factor"]) + 1.0


def _rotate(x, rot, neighbours=False):
    """x [B, T, ..., n]: pairs of entries (halves, or neighbours) turn by position times frequency."""
    if not rot or not rot["dims"]:
        return x
    freq, mag = _smooth_stretch(rot["base"], rot["dims"], rot.get("scaling"))
    half = freq.numel()
    ang = torch.arange(x.shape[1], dtype=torch.float64, device=x.device)[:, None] * freq.to(x.device)[None, :]
    shape = [1, x.shape[1]] + [1] * (x.dim() - 3) + [half]
    c, s = (ang.cos() * mag).view(shape), (ang.sin() * mag).view(shape)
    if neighbours:
        u, v = x[..., 0:2 * half:2], x[..., 1:2 * half:2]
        turned = torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2)
    else:
        u, v = x[..., :half], x[..., half:2 * half]
        turned = torch.cat([u * c - v * s, v * c + u * s], -1)
    return torch.cat([turned, x[..., 2 * half:]], -1)


def _visible(T, device, window=None, chunk=None):
    p = torch.arange(T, device=device)
    dist = p[:, None] - p[None, :]
    see = dist >= 0
    if window:
        see &= dist < window
    if chunk:
        see &= p[:, None] // chunk == p[None, :] // chunk
    return see, dist.clamp(min=0)


def _attend(q, k, v, scale, see, *, cap=None, sink=None, bend: Optional[Callable] = None):
    """q [B, T, H, d], k and v [B, T, G, .]: softmax attention, one sequence and head at a time."""
    B, T, H, _ = q.shape
    share = H // k.shape[2]
    out = torch.empty(B, T, H, v.shape[-1], dtype=q.dtype, device=q.device)
    for b in range(B):
        for a in range(H):
            s = (q[b, :, a] @ k[b, :, a // share].T) * scale
            if cap is not None:
                s = cap * torch.tanh(s / cap)
            if bend is not None:
                s = bend(s, a)
            s.masked_fill_(~see, -math.inf)
            if sink is not None:
                top = s.amax(-1, keepdim=True).clamp(min=float(sink[a]))
                s = torch.exp(s - top)
                s = s / (s.sum(-1, keepdim=True) + torch.exp(sink[a] - top))
            else:
                s = torch.softmax(s, -1)
            out[b, :, a] = s @ v[b, :, a // share]
    return out


def _conv(h, w, bias=None):
    """h [B, T, C], w [C, taps]: causal, zeros before the start."""
    taps = w.shape[1]
    padded = torch.nn.functional.pad(h, (0, 0, taps - 1, 0))
    out = sum(padded[:, j:j + h.shape[1]] * w[:, j] for j in range(taps))
    return out if bias is None else out + bias


def _recurrence(q, k, v, decay, beta=None):
    """S <- decay S + k u^T, out = S^T q, per sequence and head; u = v, or beta (v - S^T k).  q, k [B, T, H, d],
    v [B, T, H, e], decay [B, T, H, d or 1]."""
    B, T, H, d = q.shape
    S = torch.zeros(B, H, d, v.shape[-1], dtype=q.dtype, device=q.device)
    out = torch.empty_like(v)
    for t in range(T):
        S = S * decay[:, t, :, :, None]
        u = v[:, t] if beta is None else beta[:, t, :, None] * (v[:, t] - (S * k[:, t, :, :, None]).sum(2))
        S = S + k[:, t, :, :, None] * u[:, :, None, :]
        out[:, t] = (S * q[:, t, :, :, None]).sum(2)
    return out


def _memory(q, k, v, log_i, log_f):
    """Matrix memory with exponential gates, kept in range by a running maximum that starts at 0."""
    B, T, H, d = q.shape
    S = torch.zeros(B, H, d, v.shape[-1], dtype=q.dtype, device=q.device)
    n = torch.zeros(B, H, d, dtype=q.dtype, device=q.device)
    m = torch.zeros(B, H, dtype=q.dtype, device=q.device)
    out = torch.empty_like(v)
    for t in range(T):
        new = torch.maximum(log_f[:, t] + m, log_i[:, t])
        keep, take = torch.exp(log_f[:, t] + m - new)[..., None], torch.exp(log_i[:, t] - new)[..., None]
        m = new
        S = keep[..., None] * S + (take * k[:, t])[..., None] * v[:, t, :, None, :]
        n = keep * n + take * k[:, t]
        below = torch.maximum((n * q[:, t]).sum(-1).abs(), torch.exp(-m)) + 1e-6
        out[:, t] = (S * q[:, t, :, :, None]).sum(2) / below[..., None]
    return out


class _Model64:
    """The seven models on padded batches of whole sequences [B, T], in float64."""

    def __init__(self, config, weights: Weights) -> None:
        self.config, self.weights = config, weights
        self.eps = float(config["rms_norm_eps"] if weights.qwen else config["norm"]["eps"])

    def w(self, name):
        return self.weights.stored(name).double()

    def lin(self, h, name):
        return h @ self.w(name).T

    def norm(self, x, name):
        return _unit(x, self.eps) * self.w(name)

    def heads(self, x, n):
        return x.view(*x.shape[:2], n, -1)

    # ---- mixers

    def attention(self, arch, h, m, p, carried):
        H, G, scale = m["heads"], m["kv_heads"], float(m["scale"])
        B, T = h.shape[:2]
        bias = arch == "Pekunex" and not p.endswith("left.")
        get = lambda n: self.lin(h, p + n) + (self.w(p + n + ".b") if bias else 0.0)  # noqa: E731
        q, k = get("q"), get("k")
        size = (m.get("mask") or {}).get("size")
        see, far = _visible(T, h.device, window=size if arch == "Vasosun" else None, chunk=size if arch in ("Dazilix", "Vepevik") else None)
        if arch == "Dazilix":
            v = self.heads(k, G)
            q, k = self.heads(self.norm(q, p + "q.norm"), H), self.heads(self.norm(k, p + "k.norm"), G)
            y = _attend(_rotate(q, m["rot"]), _rotate(k, m["rot"]), v, scale, see, sink=torch.zeros(H, dtype=h.dtype, device=h.device))
            return self.lin(y.flatten(2), p + "o")
        q, k, v = self.heads(q, H), self.heads(k, G), self.heads(get("v"), G)
        if arch == "Vasosun":
            if m.get("q_temp"):
                pos = torch.arange(T, dtype=torch.float64, device=h.device)
                q = q * (1.0 + m["q_temp"]["coef"] * torch.log(torch.floor((pos + 1.0) / m["q_temp"]["every"]) + 1.0))[None, :, None, None]
            r1, r2 = self.w(p + "r1"), self.w(p + "r2")
            y = _attend(q, k, v, scale, see, bend=lambda s, a: s - r1[a] * torch.log1p(r2[a] * far))
            return self.lin(y.flatten(2), p + "o")
        if arch == "Vepevik":
            q, k = self.norm(q, p + "q.norm"), self.norm(k, p + "k.norm")
            if m.get("v_mix"):
                if "values" in carried:
                    lam = self.w(p + "vmix")
                    v = (1.0 - lam) * v + lam * carried["values"]
                else:
                    carried["values"] = v
            y = _attend(_rotate(q, m.get("rot")), _rotate(k, m.get("rot")), v, scale, see)
            return self.lin((y * _sigmoid(self.lin(h, p + "g"))[..., None]).flatten(2), p + "o")
        q, k = _rotate(q, m.get("rot")), _rotate(k, m.get("rot"))
        if not bias:
            return self.lin(_attend(q, k, v, scale, see, sink=self.w(p + "sink")).flatten(2), p + "o")
        y = _attend(_unit(q, self.eps), _unit(k, self.eps), v, scale, see, cap=m.get("softcap"))
        return self.lin(y.flatten(2) * _sigmoid(self.lin(h, p + "g")), p + "o")

    def latent(self, arch, h, m, p, carried, i):
        H, d, R, T = m["heads"], m["dim"], m["kv_rank"], h.shape[1]
        near = arch != "Mugulorn"
        src = m.get("kv_from")
        if src is None:
            rows = self.lin(h, p + "dkv")
            carried[("latent", i)] = (self.norm(rows[..., :R], p + "dkv.norm"), _rotate(rows[..., R:], m["rot"], near))
            src = i
        c, r = carried[("latent", src)]
        q = self.lin(h, p + "q") if arch == "Fegetar" else self.lin(self.norm(self.lin(h, p + "dq"), p + "dq.norm"), p + "uq")
        q = self.heads(q, H)
        q = torch.cat([q[..., :d], _rotate(q[..., d:], m["rot"], near)], -1)
        k = torch.cat([self.heads(self.lin(c, p + "uk"), H), r[:, :, None, :].expand(-1, -1, H, -1)], -1)
        v = self.heads(self.lin(c, p + "uv"), H)
        see, _ = _visible(T, h.device, window=(m.get("mask") or {}).get("size"))
        y = _attend(q, k, v, float(m["scale"]), see, sink=self.w(p + "sink") if arch == "Mugulorn" else None)
        if arch == "Fegetar":
            y = y * _sigmoid(self.lin(h, p + "g"))[..., None]
        y = y.flatten(2)
        if arch == "Mugulorn":
            y = y * _sigmoid(self.lin(h, p + "g"))
        return self.lin(y, p + "o")

    def gla(self, h, m, p):
        H, d = m["heads"], m["dim"]
        z = self.lin(self.lin(h, p + "a1"), p + "a2") + self.w(p + "a2.b")
        decay = self.heads(torch.exp(torch.nn.functional.logsigmoid(z) / m["tau"]), H)
        o = _recurrence(self.heads(self.lin(h, p + "q"), H) * d ** -0.5, self.heads(self.lin(h, p + "k"), H), self.heads(self.lin(h, p + "v"), H), decay)
        return self.lin(self.norm(o, p + "norm").flatten(2) * _silu(self.lin(h, p + "g")), p + "o")

    def retention(self, h, m, p):
        H, d = m["heads"], m["dim"]
        q = _rotate(self.heads(self.lin(h, p + "q"), H), m.get("rot"))
        k = _rotate(self.heads(self.lin(h, p + "k"), H), m.get("rot")) * d ** -0.5
        decay = torch.tensor(m["decay"], dtype=h.dtype, device=h.device)[None, None, :, None].expand(*h.shape[:2], -1, -1)
        o = _unit(_recurrence(q, k, self.heads(self.lin(h, p + "v"), H), decay), self.eps)
        return self.lin(o.flatten(2) * _silu(self.lin(h, p + "g")), p + "o")

    def delta(self, h, m, p, per_channel):
        H, G, d = m["heads"], m["kv_heads"], m["dim"]
        short = lambda n, heads: self.heads(_silu(_conv(self.lin(h, p + n), self.w(p + n + ".conv"))), heads)  # noqa: E731
        long = lambda x: (x / torch.sqrt(x.pow(2).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 2)  # noqa: E731
        q, k, v = long(short("q", G)) * d ** -0.5, long(short("k", G)), short("v", H)
        rate = torch.exp(self.w(p + "A_log"))
        if per_channel:
            z = self.heads(self.lin(self.lin(h, p + "a1"), p + "a2") + self.w(p + "dt_bias"), H)
            decay = torch.exp(-rate[:, None] * _softplus(z))
            gate = _sigmoid(self.lin(self.lin(h, p + "g1"), p + "g2"))
        else:
            decay = torch.exp(-rate * _softplus(self.lin(h, p + "a") + self.w(p + "dt_bias")))[..., None]
            gate = _silu(self.lin(h, p + "g"))
        o = _recurrence(q, k, v, decay, _sigmoid(self.lin(h, p + "b")))
        return self.lin(self.norm(o, p + "norm").flatten(2) * gate, p + "o")

    def memory(self, h, m, p):
        H, d, cap = m["heads"], m["dim"], m["gate_cap"]
        bent = lambda n: cap * torch.tanh((self.lin(h, p + n) + self.w(p + n + ".b")) / cap)  # noqa: E731
        q, k, v = (self.heads(self.lin(h, p + n), H) for n in "qkv")
        o = _memory(q * d ** -0.5, k, v, bent("i"), torch.nn.functional.logsigmoid(bent("f")))
        return self.lin(_unit(o, self.eps).flatten(2) * self.w(p + "norm") * _sigmoid(self.lin(h, p + "g")), p + "o")

    def state_space(self, h, m, p):
        H, e, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
        inner = H * e
        z, rest, dt = self.lin(h, p + "in").split([inner, inner + 2 * G * N, H], -1)
        x, Bm, Cm = _silu(_conv(rest, self.w(p + "conv"), self.w(p + "conv.b"))).split([inner, G * N, G * N], -1)
        dt = _softplus(dt + self.w(p + "dt_bias"))
        x = self.heads(x, H)
        each = lambda t: self.heads(t, G).repeat_interleave(H // G, 2)  # noqa: E731
        decay = torch.exp(-torch.exp(self.w(p + "A_log")) * dt)[..., None]
        y = _recurrence(each(Cm), each(Bm), x * dt[..., None], decay) + self.w(p + "D")[:, None] * x
        y = _unit(self.heads(y.flatten(2) * _silu(z), m["norm_groups"]), self.eps).flatten(2) * self.w(p + "norm")
        return self.lin(y, p + "o")

    def rglru(self, h, m, p):
        y = _gelu(self.lin(h, p + "y") + self.w(p + "y.b"))
        u = _conv(self.lin(h, p + "x") + self.w(p + "x.b"), self.w(p + "conv"), self.w(p + "conv.b"))
        gate = lambda n: _sigmoid(torch.einsum("btni,noi->btno", self.heads(u, m["blocks"]), self.w(p + n)) + self.w(p + n + ".b")).flatten(2)  # noqa: E731
        log_a = -8.0 * gate("ra") * _softplus(self.w(p + "lam"))
        a, x = torch.exp(log_a), torch.sqrt(-torch.expm1(2.0 * log_a)) * gate("ri") * u
        S, out = torch.zeros_like(x[:, 0]), torch.empty_like(x)
        for t in range(x.shape[1]):
            S = a[:, t] * S + x[:, t]
            out[:, t] = S
        return self.lin(out * y, p + "o")

    # ---- feed-forwards

    def glu(self, h, p, act, limit=None):
        a, b = self.lin(h, p + "gate"), self.lin(h, p + "up")
        if limit is not None:
            a, b = a.clamp(max=limit), b.clamp(-limit, limit)
            return self.lin(a * _sigmoid(1.702 * a) * (b + 1.0), p + "down")
        return self.lin(act(a) * b, p + "down")

    def routed(self, arch, h, f, p):
        r = f["router"]
        E, top = r["experts"], r["top"]
        flat = h.flatten(0, 1)
        z = self.lin(flat, p + "router")
        if arch == "Fegetar":
            share, chosen = torch.topk(_sigmoid(z), top, -1)
        elif arch == "Dazilix":
            share, chosen = torch.topk(z + self.w(p + "router.b"), top, -1)
            share = torch.softmax(share, -1)
        elif arch == "Vasosun":
            s = torch.softmax(z, -1)
            chosen = torch.topk(s + self.w(p + "correction"), top, -1).indices
            share = s.gather(1, chosen)
        else:
            s = torch.softmax(z, -1)
            allowed = s
            if r.get("groups"):
                n, keep = r["groups"]["count"], r["groups"]["keep"]
                best = s.view(-1, n, E // n).amax(-1)
                kept = torch.zeros_like(best, dtype=torch.bool).scatter(1, torch.topk(best, keep, -1).indices, True)
                allowed = s.masked_fill(~kept.repeat_interleave(E // n, -1), -1.0)
            chosen = torch.topk(allowed, top, -1).indices
            share = s.gather(1, chosen)
            share = share / (share.sum(-1, keepdim=True) + 1e-20) * r["scale"]
        out = torch.zeros_like(flat)
        for e in range(E + (r.get("identity") or 0)):
            rows, slot = torch.nonzero(chosen == e, as_tuple=True)
            if not len(rows):
                continue
            x, a = flat[rows], share[rows, slot][:, None]
            pe = f"{p}e{e}."
            if e >= E:
                y = a * x
            elif arch == "Fegetar":
                y = self.glu(a * x, pe, None, f["expert"]["limit"])
            elif arch == "Vasosun":
                y = a * self.lin(torch.nn.functional.gelu(self.lin(x, pe + "up")), pe + "down")
            else:
                y = a * self.glu(x, pe, _silu)
            out.index_add_(0, rows, y)
        out = out.view_as(h)
        if f.get("shared"):
            out = out + self.glu(h, p + "shared.", None, f["shared"]["limit"])
        return out

    def feed_forward(self, arch, h, f, p):
        if f["kind"] == "moe":
            return self.routed(arch, h, f, p)
        if arch == "Fegetar":
            return self.lin(_gelu(self.lin(h, p + "up")), p + "down")
        return self.glu(h, p, _gelu if arch == "Mugulorn" else _silu, f.get("limit") if arch == "Vepevik" else None)

    # ---- whole models

    def embed(self, ids):
        x = self.w("embed")[ids]
        e = self.config.get("embedding") or {}
        if e.get("scale"):
            x = x * float(e["scale"])
        if e.get("bigram"):
            b = e["bigram"]
            rows = torch.full_like(ids, b["buckets"])
            rows[:, 1:] = (ids[:, :-1] * b["mul_prev"] + ids[:, 1:] * b["mul_cur"]) % b["buckets"]
            x = x + self.w("bigram")[rows]
        return self.norm(x, "embed.norm") if self.config["architecture"] == "Vepevik" else x

    def mixer(self, arch, kind, h, m, p, carried, i):
        if kind == "attention":
            return self.attention(arch, h, m, p, carried)
        if kind == "latent_attention":
            return self.latent(arch, h, m, p, carried, i)
        if kind == "parallel":
            left = self.attention(arch, h, m["left"], p + "left.", carried)
            return float(m["left_scale"]) * left + float(m["right_scale"]) * self.memory(h, m["right"], p + "right.")
        if kind in ("delta", "channel_delta"):
            return self.delta(h, m, p, kind == "channel_delta")
        return {"gla": self.gla, "retention": self.retention, "mamba2": self.state_space, "rglru": self.rglru}[kind](h, m, p)

    def design(self, ids):
        c = self.config
        arch, carried, x = c["architecture"], {}, self.embed(ids)
        side = self.w("side.embed")[ids] if c.get("token_side") else None
        shift = 1.0 if arch == "Fegetar" else 0.0
        for i, layer in enumerate(c["layers"]):
            p = f"l{i}."
            for half, f in ((1, None), (2, layer.get("mlp"))):
                if half == 2 and f is None:
                    continue
                h = x if arch == "Fegetar" else self.norm(x, f"{p}norm{half}")
                if arch == "Vasosun":
                    h = h + _conv(h, self.w(f"{p}canon{half}"))
                y = self.mixer(arch, layer["type"], h, layer["mixer"], p + "mix.", carried, i) if half == 1 else self.feed_forward(arch, h, f, p + "mlp.")
                if arch == "Fegetar":
                    y = _unit(y, self.eps) * (shift + self.w(f"{p}norm{half}"))
                elif arch in ("Dazilix", "Vasosun"):
                    y = self.norm(y, f"{p}norm{half}b") * (self.w(f"{p}ls{half}") if arch == "Dazilix" else 1.0)
                elif arch == "Mugulorn":
                    y = float(c["residual_mult"]) * y
                x = x + y
            if side is not None:
                n = c["token_side"]["dim"]
                y = self.lin(_gelu(self.lin(x, p + "side.gate")) * side[..., i * n:(i + 1) * n], p + "side.proj")
                x = x + self.norm(y, p + "side.norm")
        return x

    def head(self, x):
        c = self.config
        if self.weights.qwen:
            y = self.norm(x, "model.norm.weight")
            return self.lin(y, "model.embed_tokens.weight" if c["tie_word_embeddings"] else "lm_head.weight")
        y = _unit(x, self.eps) * ((1.0 if c["architecture"] == "Fegetar" else 0.0) + self.w("final.norm"))
        y = self.lin(y, "embed" if c["architecture"] in ("Mugulorn", "Vepevik") else "head") * float(c.get("logit_scale") or 1.0)
        cap = c.get("logit_softcap")
        return float(cap) * torch.tanh(y / float(cap)) if cap else y

    def dense(self, ids):
        c = self.config
        H, G, d = c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"]
        x = self.w("model.embed_tokens.weight")[ids]
        see, _ = _visible(ids.shape[1], ids.device)
        rot = {"base": float(c["rope_theta"]), "dims": d}
        for i in range(c["num_hidden_layers"]):
            p = f"model.layers.{i}."
            a, f = p + "self_attn.", p + "mlp."
            h = self.norm(x, p + "input_layernorm.weight")
            q = _rotate(self.norm(self.heads(self.lin(h, a + "q_proj.weight"), H), a + "q_norm.weight"), rot)
            k = _rotate(self.norm(self.heads(self.lin(h, a + "k_proj.weight"), G), a + "k_norm.weight"), rot)
            y = _attend(q, k, self.heads(self.lin(h, a + "v_proj.weight"), G), d ** -0.5, see)
            x = x + self.lin(y.flatten(2), a + "o_proj.weight")
            h = self.norm(x, p + "post_attention_layernorm.weight")
            y = _silu(self.lin(h, f + "gate_proj.weight")) * self.lin(h, f + "up_proj.weight")
            x = x + self.lin(y, f + "down_proj.weight")
        return x


@torch.no_grad()
def exact(case, seed: int) -> list[torch.Tensor]:
    config = _config(case)
    typed = get_model_config("qwen3-" + case["size"]) if case["model"] == "qwen3" else architecture_for(config).config_from_dict(config)
    spec = architecture_for(typed.to_dict()).build_spec(typed)
    weights = _weights(case, seed, spec.tensor_specs())
    contexts, prompts = _token_ids(case, seed, spec.vocab_size)
    seqs = contexts + prompts
    ids = torch.zeros(len(seqs), max(len(x) for x in seqs), dtype=torch.long, device="cuda")
    for i, x in enumerate(seqs):  # zeros behind a sequence change nothing before them
        ids[i, : len(x)] = torch.tensor(x, device="cuda")
    model = _Model64(config, weights)
    last = torch.tensor([len(x) - 1 for x in seqs], device="cuda")
    groups = [range(i, min(i + 8, len(seqs))) for i in range(0, len(seqs), 8)] if case["model"] == "qwen3" else [range(len(seqs))]
    rows = []
    for g in groups:
        x = model.dense(ids[g.start:g.stop]) if weights.qwen else model.design(ids[g.start:g.stop])
        rows.append(x[torch.arange(len(g), device="cuda"), last[g.start:g.stop]])
    logits = model.head(torch.cat(rows))
    if not case["portion"]:
        return [logits]
    order: dict[int, list[int]] = {}
    for i, x in enumerate(prompts):  # a prompt's logits come with the step of its last portion
        order.setdefault(-(-len(x) // case["portion"]), []).append(len(contexts) + i)
    if contexts:
        order.setdefault(1, [])[:0] = list(range(len(contexts)))
    return [logits[order[k]] for k in sorted(order)]
