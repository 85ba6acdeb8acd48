"""What the engine is timed on: requests carried from their prompts to their last token.

A case is a group of requests that one engine serves: their prompts arrive (together, or one a step while the
earlier ones are already answering), are prefilled in portions of at most ``PORTION`` tokens, and every request
then takes ``answer - 1`` single-token steps.  One pass is that whole life through ``Engine.step``, the step
function below ``LLM.generate``, the scheduler and trace replay, and ``Engine.end_request``.  The tokens are
given (as in trace replay) instead of sampled, so that a pass does the same work whatever its logits round to;
the pass returns the float32 logits at every place where a token would have been sampled.

Sizes are those of the repository's benchmarks: the MiniMax-M3 decoder at its real layer width (four layers of
it), and every served design at widths 2048 and 4096.  Weights are random with the benchmarks' scales.

``exact`` evaluates the same decoders in 64 bits in plain torch, a whole sequence at a time.
"""

from __future__ import annotations

import math
from typing import Any, Dict, List, Optional, Tuple

import numpy as np
import torch

from freetoken_b200 import Engine, EngineArgs, StepEntry
from freetoken_b200 import (besuzen_bench, design_bench, dizatar_bench, mezapel_bench, nirelix_bench,
                            tonapel_bench)
from freetoken_b200.benchmark import BENCH_CONFIG, bench_random_options
from freetoken_b200.models.model import Model
from freetoken_b200.registry import architecture_of
from freetoken_b200.weights import random_state
from freetoken_b200.weights.spec import take_apart

PORTION = 8192          # most prompt tokens of a step (the engine's and the scheduler's default)
PAGE = 64
MOST_TOKENS = 16384     # of a drawn case's prompts
POSITIONS = 1 << 17

Case = Dict[str, Any]
F64 = torch.float64


# ------------------------------------------------------------------------------------------- cases
def _case(name: str, model: str, size: str, requests: int, prompt: int, answer: int, ragged: bool = False,
          staggered: bool = False, dtype: str = "bfloat16") -> Case:
    return dict(name=name, model=model, size=size, requests=requests, prompt=prompt, answer=answer,
                ragged=ragged, staggered=staggered, dtype=dtype)


def listed() -> List[Case]:
    return [
        # a chat turn of one user on the flagship: a short odd prompt, then one token a step (latency)
        _case("chat_of_one", "minimax_m3", "real", 1, 37, 16),
        # the benchmark's serving point: eight requests on 2,048-token contexts
        _case("serve_eight", "minimax_m3", "real", 8, 2048, 24),
        # a busy server: 64 short ragged requests answered together
        _case("serve_sixty_four", "minimax_m3", "real", 64, 250, 8, ragged=True),
        # time to first token of one ordinary prompt
        _case("first_token", "minimax_m3", "real", 1, 2048, 1),
        # a book as the prompt: 65,536 tokens in portions, then a short answer (the largest work)
        _case("long_context", "minimax_m3", "real", 1, 65536, 9),
        # the 32-bit path, as it is used to check answers: two uneven requests
        _case("float32_check", "minimax_m3", "w2048", 2, 301, 5, ragged=True, dtype="float32"),
        # the smallest call: a few tokens in, a few out, on a small model; launches and host work count
        _case("short_reply", "fazinex", "w2048", 1, 9, 12),
        # one ordinary prompt and its answer on a model with recurrent states (state space, delta rule)
        _case("recurrent_turn", "tonapel", "w2048", 1, 2048, 16),
        # ragged requests on the wider model of retention and per-channel delta rule
        _case("recurrent_batch", "nirelix", "w4096", 4, 1500, 12, ragged=True),
        # requests that arrive while others are answering: prompts beside single tokens in one step
        _case("arrivals", "mezapel", "w2048", 8, 700, 12, ragged=True, staggered=True),
        # a document and its answer on latent attention, wide
        _case("document", "dizatar", "w4096", 1, 3001, 16),
        # eight requests on the model with time mixing beside attention
        _case("mixed_batch", "besuzen", "w2048", 8, 1000, 24, ragged=True),
    ]


def draw(rng) -> Case:
    def log_uniform(low: int, high: int) -> int:
        return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))

    model = rng.choice(["minimax_m3", "minimax_m3", "fazinex", "tonapel", "nirelix", "mezapel", "dizatar", "besuzen"])
    size = rng.choice(["real", "w2048"] if model == "minimax_m3" else ["w2048", "w4096"])
    # the 32-bit path serves small models and short prompts (checks); it is no serving path
    dtype = "float32" if model == "minimax_m3" and size == "w2048" and rng.random() < 0.5 else "bfloat16"
    requests = log_uniform(1, 4 if dtype == "float32" else 64)
    prompt = log_uniform(5, max(6, min(512 if dtype == "float32" else PORTION, MOST_TOKENS // requests)))
    answer = log_uniform(1, 8 if dtype == "float32" or requests > 16 else 24)
    ragged = rng.random() < 0.5
    staggered = 1 < requests <= 16 and rng.random() < 0.3
    c = _case("", model, size, requests, prompt, answer, ragged, staggered, dtype)
    del c["name"]
    return c


def model_config(case: Case) -> Dict[str, Any]:
    model, size = case["model"], case["size"]
    if model == "minimax_m3":
        if size == "real":
            return dict(BENCH_CONFIG, num_hidden_layers=4, max_position_embeddings=POSITIONS)
        return design_bench.minimax_config(design_bench.SIZES[size], POSITIONS)
    if model == "fazinex":
        return design_bench.fazinex_config(design_bench.SIZES[size])
    bench = {"tonapel": tonapel_bench, "nirelix": nirelix_bench, "mezapel": mezapel_bench, "dizatar": dizatar_bench,
             "besuzen": besuzen_bench}[model]
    return getattr(bench, f"{model}_config")(bench.SIZES[size])


def prompt_lengths(case: Case) -> List[int]:
    n, longest = case["requests"], case["prompt"]
    if not case["ragged"]:
        return [longest] * n
    shortest = max(1, longest // 4)
    return [shortest + int((longest - shortest) * ((1 + i) * 0.6180339887 % 1.0)) for i in range(n)]


def schedule(case: Case) -> List[List[Tuple[int, int, int, bool]]]:
    """The steps of a pass: ``(request, first token, end, wants logits of its last)`` per entry.  Prompts go in
    arrival order, cut where a step is full; requests whose prompt is in take one token a step."""
    lengths, answer = prompt_lengths(case), case["answer"]
    done = [0] * len(lengths)
    steps: List[List[Tuple[int, int, int, bool]]] = []
    while any(d < n + answer - 1 for d, n in zip(done, lengths)):
        arrived = len(steps) + 1 if case["staggered"] else len(lengths)
        entries, room = [], PORTION
        waiting = any(d < n for d, n in zip(done[:arrived], lengths))
        for i, n in enumerate(lengths[:arrived]):
            # requests that came together start to answer together
            if n <= done[i] < n + answer - 1 and (case["staggered"] or not waiting):
                entries.append((i, done[i], done[i] + 1, True))
            elif done[i] < n and room:
                end = min(n, done[i] + room)
                room -= end - done[i]
                entries.append((i, done[i], end, end == n))
        for i, _, end, _ in entries:
            done[i] = end
        steps.append(entries)
    return steps


def _token_ids(case: Case, seed: int, vocab: int) -> List[List[int]]:
    """Uniform random token ids: prompt and answer of every request."""
    rng = np.random.default_rng([seed, 77])
    return [rng.integers(0, vocab, n + case["answer"] - 1).tolist() for n in prompt_lengths(case)]


# --------------------------------------------------------------------------------------------- pass
def _with_kinds(tensors: Dict[str, torch.Tensor], specs, top: int, outputs: int, hidden: int, seed: int) -> None:
    """Routers that choose by a margin.  Every token id is of one of some kinds; its embedding carries the kind's
    direction, and a layer's router prefers ``top`` experts of its own for each kind.  (With plain random weights
    the last expert chosen and the first one left out lie within rounding of each other in a share of the rows,
    and two right implementations then differ by a whole expert.)"""
    routers = [s.name for s in specs if s.keep_float32_in_file and len(s.shape) == 2]
    if not routers:
        return
    device = tensors[routers[0]].device
    gen = torch.Generator(device=device).manual_seed(seed)
    kinds = max(64, outputs)
    basis = torch.linalg.qr(torch.randn(hidden, kinds, generator=gen, device=device))[0].T * hidden ** 0.5
    embed = next(tensors[s.name] for s in specs if s.tag == "embedding")
    plain = embed.float()
    kind = torch.arange(embed.shape[0], device=device) % kinds
    embed.copy_(plain - (plain @ basis.T) @ basis / hidden + 1.5 * basis[kind])
    for name in routers:
        chosen = torch.rand(kinds, outputs, generator=gen, device=device).topk(top, -1).indices
        level = torch.full((kinds, outputs), -0.8, device=device)
        level.scatter_(1, chosen, 0.8 + 0.8 * torch.rand(kinds, top, generator=gen, device=device))
        rows = tensors[name][:outputs]
        rows.mul_(0.1).add_(2.0 / hidden * (level.T @ basis))
    if "loop.in" in tensors:                     # the kind survives the map between passes
        half = tensors["loop.in"][:, :hidden]
        half.copy_(half + torch.eye(hidden, dtype=half.dtype, device=device))


def _engine(case: Case, seed: int) -> Engine:
    config = model_config(case)
    arch = architecture_of(config)
    typed = arch.read_config(config)
    plan = arch.build_plan(typed)
    specs = Model(plan).tensor_specs()
    dtype = getattr(torch, case["dtype"])
    tensors = random_state(specs, seed, "cuda", dtype, options=bench_random_options())
    top, outputs = max(_routing(config))
    _with_kinds(tensors, specs, top, outputs, plan.hidden_size, seed)
    lengths = [n + case["answer"] for n in prompt_lengths(case)]
    pages = sum(-(-n // PAGE) for n in lengths) + case["requests"]
    return Engine(arch, typed, tensors, EngineArgs(
        dtype=case["dtype"], page_size=PAGE, num_pages=pages, max_running_requests=case["requests"],
        max_seq_len=-(-max(lengths) // PAGE) * PAGE, max_step_tokens=PORTION))


def prepare(case: Case, seed: int) -> Dict[str, Any]:
    engine = _engine(case, seed)
    tokens = _token_ids(case, seed, engine.vocab_size)
    steps = [[StepEntry(i, tokens[i][a:b], [b - a - 1] if wants else []) for i, a, b, wants in entries]
             for entries in schedule(case)]
    return {"engine": engine, "steps": steps, "requests": list(range(case["requests"])),
            "rows": case["requests"] * case["answer"]}


def run(state: Dict[str, Any]) -> torch.Tensor:
    engine = state["engine"]
    out = torch.empty((state["rows"], engine.vocab_size), dtype=torch.float32, device=engine.device)
    at = 0
    for entries in state["steps"]:
        logits = engine.step(entries)
        n = logits.shape[0]
        if n:
            out[at:at + n].copy_(logits)         # the engine's logits are overwritten by its next step
            at += n
    for request in state["requests"]:
        engine.end_request(request)
    return out


# --------------------------------------------------------------------------------------------- work
def _parts(case: Case):
    """The model's tensors, its layers in the order they run and its typed size entries."""
    config = model_config(case)
    arch = architecture_of(config)
    plan = arch.build_plan(arch.read_config(config))
    return config, plan, Model(plan).tensor_specs()


def _routing(config: Dict[str, Any]) -> List[Tuple[int, int]]:
    """Per layer: experts chosen, experts there are (0, 0: a dense feed-forward)."""
    if "hidden_size" in config:
        return [(config["num_experts_per_tok"], config["num_local_experts"])] * config["num_hidden_layers"]
    routers = [(layer.get("mlp") or {}).get("router") for layer in config["layers"]]
    return [(r["top"], r["experts"] + (r.get("identity") or 0)) if r else (0, 0) for r in routers]


def _mixers(config: Dict[str, Any]) -> List[List[Dict[str, Any]]]:
    """Per layer: its mixers, as ``{kind, heads, kv values a token, query width, value width, state, reach}``."""
    def attention(m, kv_values=None):
        mask = (m.get("mask") or {}).get("size") or math.inf
        kv = kv_values or m["kv_heads"] * (m["dim"] + m["vdim"])
        return {"pair": 2 * m["heads"] * (m["dim"] + m.get("rot_dim", 0) + m["vdim"]), "kv": kv, "reach": mask}

    def recurrent(values, passes):
        return {"state": values, "flops": 2 * passes * values}

    if "hidden_size" in config:
        c = config
        m = {"heads": c["num_attention_heads"], "kv_heads": c["num_key_value_heads"], "dim": c["head_dim"],
             "vdim": c["head_dim"]}
        return [[attention(m)] for _ in range(c["num_hidden_layers"])]
    out = []
    for layer in config["layers"]:
        m, kind = layer["mixer"], layer["type"]
        if "left" in m:
            r = m["right"]
            state = r["heads"] * r["vdim"] * r["state"] if "state" in r else r["heads"] * r["dim"] ** 2
            out.append([attention(m["left"]), recurrent(state, 3)])
        elif kind in ("delta", "channel_delta"):
            out.append([recurrent(m["heads"] * m["dim"] * m["vdim"], 4)])
        elif kind == "retention":
            out.append([recurrent(m["heads"] * m["dim"] * m["vdim"], 3)])
        elif "kv_rank" in m:
            out.append([attention(m, m["kv_rank"] + m.get("rot_dim", 0))])
        elif config["architecture"] == "Fazinex":
            out.append([attention(m, m["kv_heads"] * m["dim"])])      # the values are the keys
        else:
            out.append([attention(m)])
    return out


def work(case: Case) -> Dict[str, float]:
    config, plan, specs = _parts(case)
    item = 2 if case["dtype"] == "bfloat16" else 4
    lengths = prompt_lengths(case)
    runs = [stop.layer for stop in plan.schedule]
    prefixes = [layer.prefix for layer in plan.layers]
    head = plan.vocab_size * plan.hidden_size
    # weights by layer: dense ones, and experts as (bytes of one, experts, chosen)
    dense = [0.0] * len(prefixes)
    small = [0.0] * len(prefixes)
    experts: List[List[Tuple[float, int]]] = [[] for _ in prefixes]
    for spec in specs:
        n = float(np.prod(spec.shape)) if spec.shape else 1.0
        layer = next((i for i, p in enumerate(prefixes) if p and spec.name.startswith(p + ".")), None)
        if layer is None:
            continue
        if len(spec.shape) == 3 and spec.shape[0] > 4:
            experts[layer].append((n / spec.shape[0], spec.shape[0]))
        elif spec.role == "matrix":
            dense[layer] += n
        else:
            small[layer] += n
    routing = _routing(config)
    mixers = _mixers(config)
    nbytes = flops = 0.0
    for entries in schedule(case):
        T = sum(b - a for _, a, b, _ in entries)
        N = sum(1 for e in entries if e[3])
        nbytes += (head * 2 if N else 0) + N * plan.vocab_size * 4.0 + T * plan.hidden_size * 2
        flops += 2.0 * head * N
        for layer in runs:
            nbytes += dense[layer] * 2 + small[layer] * 4
            flops += 2.0 * dense[layer] * T
            for size, count in experts[layer]:
                share = routing[layer][0] / routing[layer][1]
                nbytes += size * 2 * count * (1.0 - (1.0 - share) ** T)
                flops += 2.0 * size * T * share * count
            for m in mixers[layer]:
                for i, a, b, _ in entries:
                    if "state" in m:
                        nbytes += 8.0 * m["state"]                    # float32, read and written
                        flops += m["flops"] * (b - a)
                    else:
                        first = max(0, a - m["reach"]) if m["reach"] < math.inf else 0
                        nbytes += item * m["kv"] * (b - first)
                        p = np.arange(a + 1, b + 1, dtype=np.float64)
                        flops += m["pair"] * float(np.minimum(p, m["reach"]).sum())
    return {"bytes": nbytes, "flops": flops}


def tolerance(case: Case) -> Dict[str, float]:
    # About four times what a pass differs by from exact(): 8e-7 in 32 bits; in bfloat16, whose activations are
    # rounded a dozen times a layer, 1.6e-3 to 3e-3, and 5e-3 on Tonapel (every branch is normed before it joins
    # the residual, which amplifies its rounding) and Fazinex (keys that are values, capped logits).
    if case["dtype"] == "float32":
        return {"rel": 4e-6, "max": 1e-4}
    if case["model"] in ("tonapel", "fazinex"):
        return {"rel": 0.02, "max": 0.16}
    return {"rel": 0.01, "max": 0.06}


# ------------------------------------------------------------------------- the decoders in 64 bits
class _Weights:
    """Tensors by their checkpoint names, handed out in 64 bits."""

    def __init__(self, engine: Engine):
        self.parts: Dict[str, torch.Tensor] = {}
        for spec in engine.model.tensor_specs():
            if spec.name not in engine.tensors:
                continue
            if spec.sources:
                take_apart(spec.sources[0], engine.tensors[spec.name], self.parts)
            else:
                self.parts[spec.name] = engine.tensors[spec.name]

    def __getitem__(self, name: str) -> torch.Tensor:
        return self.parts[name].to(F64)

    def rows(self, name: str, ids: torch.Tensor) -> torch.Tensor:
        return self.parts[name][ids].to(F64)


def _rms(v, eps):
    return v / torch.sqrt((v * v).mean(-1, keepdim=True) + eps)


def _layer_norm(v, w, b, eps):
    d = v - v.mean(-1, keepdim=True)
    return d / torch.sqrt((d * d).mean(-1, keepdim=True) + eps) * w + b


def _silu(v):
    return v * torch.sigmoid(v)


def _gelu(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


def _swiglu_clamped(g, u, limit):
    g, u = g.clamp(max=limit), u.clamp(-limit, limit)
    return g * torch.sigmoid(1.702 * g) * (u + 1.0)


def _softplus(v):
    return torch.nn.functional.softplus(v, threshold=40.0)


def _rotate(v, freqs, magnitude=1.0, pairs=False):
    """``v`` ``[T, heads, dim]`` at positions 0..T-1; dimension i turns with i + len(freqs), or 2i with 2i + 1."""
    half = len(freqs)
    if half == 0:
        return v
    f = torch.tensor(freqs, dtype=F64, device=v.device)
    a = torch.arange(v.shape[0], dtype=F64, device=v.device)[:, None] * f
    cos, sin = (a.cos() * magnitude)[:, None], (a.sin() * magnitude)[:, None]
    x, y = (v[..., 0:2 * half:2], v[..., 1:2 * half:2]) if pairs else (v[..., :half], v[..., half:2 * half])
    turned = (x * cos - y * sin, y * cos + x * sin)
    turned = torch.stack(turned, -1).flatten(-2) if pairs else torch.cat(turned, -1)
    return torch.cat([turned, v[..., 2 * half:]], -1)


def _plain_frequencies(base, dims):
    return [float(base) ** (-2.0 * i / dims) for i in range(dims // 2)]


def _yarn(base, dims, s):
    def dim_of(turns):
        return dims * math.log(s["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))
    lo, hi = max(math.floor(dim_of(s["fast"])), 0), min(math.ceil(dim_of(s["slow"])), dims - 1)
    ramp = [min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0) for i in range(dims // 2)]
    return ([f / s["factor"] * r + f * (1.0 - r) for f, r in zip(_plain_frequencies(base, dims), ramp)],
            0.1 * math.log(s["factor"]) + 1.0)


def _llama3(base, dims, s):
    out = []
    for f in _plain_frequencies(base, dims):
        wave = 2.0 * math.pi / f
        t = min(max((s["original"] / wave - s["low"]) / (s["high"] - s["low"]), 0.0), 1.0)
        out.append((1.0 - t) * f / s["factor"] + t * f)
    return out, 1.0


def _attend(q, k, v, scale, first=None, cap=0.0, sink=None):
    """Causal softmax attention of one sequence, query rows in slices; ``first`` ``[T]``: the first key a row sees."""
    T, H, D = q.shape
    G = k.shape[1]
    kt, vt = k.permute(1, 2, 0), v.permute(1, 0, 2)
    out = torch.empty(T, H, v.shape[2], dtype=F64, device=q.device)
    rows = max(1, min(T, (1 << 27) // (H * T)))
    at = torch.arange(T, device=q.device)
    for a in range(0, T, rows):
        b = min(T, a + rows)
        lo = int(first[a]) if first is not None else 0
        s = q[a:b].view(b - a, G, H // G, D).permute(1, 2, 0, 3).reshape(G, -1, D) @ kt[:, :, lo:b]
        s = s.view(H, b - a, b - lo) * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        seen = at[None, lo:b] <= at[a:b, None]
        if first is not None:
            seen &= at[None, lo:b] >= first[a:b, None]
        s = s.masked_fill_(~seen, float("-inf"))
        if sink is None:
            p = torch.softmax(s, -1)
        else:
            top = torch.maximum(s.amax(-1, keepdim=True), sink[:, None, None])
            p = torch.exp(s - top)
            p = p / (p.sum(-1, keepdim=True) + torch.exp(sink[:, None, None] - top))
        o = p.view(G, -1, b - lo) @ vt[:, lo:b]
        out[a:b] = o.view(G, H // G, b - a, -1).permute(2, 0, 1, 3).reshape(b - a, H, -1)
    return out


def _conv(u, w):
    taps = w.shape[1]
    padded = torch.cat([u.new_zeros(taps - 1, u.shape[1]), u])
    return sum(padded[j:j + u.shape[0]] * w[:, j] for j in range(taps))


def _state_loop(keys, values, reads, decay, write=None, bonus=None):
    """``S <- decay S`` by rows, ``S <- S + k u^T``, ``o = S^T r`` a token at a time, all heads at once.  ``write``:
    ``u = write (v - S^T k)``.  ``bonus``: the state is read before the token's own write, which then counts
    times the bonus, and decays afterwards."""
    T, H, D = keys.shape
    S = torch.zeros(H, D, values.shape[2], dtype=F64, device=keys.device)
    out = torch.empty(T, H, values.shape[2], dtype=F64, device=keys.device)
    decay = decay.expand(T, H, D) if decay.dim() == 3 else decay[:, :, None].expand(T, H, D)
    for t in range(T):
        k, v = keys[t][:, :, None], values[t][:, None]
        if bonus is not None:
            kv = k * v
            out[t] = ((S + bonus[:, :, None] * kv) * reads[t][:, :, None]).sum(1)
            S = S * decay[t][:, :, None] + kv
            continue
        S = S * decay[t][:, :, None]
        if write is not None:
            v = write[t][:, None, None] * (v - k.transpose(1, 2) @ S)
        S = torch.baddbmm(S, k, v)
        out[t] = (reads[t][:, None] @ S)[:, 0]
    return out


def _experts(h, ids, weights, expert):
    out = torch.zeros_like(h)
    for e in ids.unique().tolist():
        rows, slot = (ids == e).nonzero(as_tuple=True)
        out.index_add_(0, rows, weights[rows, slot][:, None] * expert(e, h[rows]))
    return out


def _grouped_choice(choice, top, groups, group_value):
    E, count = choice.shape[1], groups["count"]
    best = group_value(choice.view(-1, count, E // count)).topk(groups["keep"], -1).indices
    kept = torch.zeros(choice.shape[0], count, dtype=torch.bool, device=choice.device).scatter_(1, best, True)
    return choice.masked_fill(~kept.repeat_interleave(E // count, 1), float("-inf")).topk(top, -1).indices


class _Decoder:
    """``x`` and every sublayer's input hold the rows of all sequences one after the other; mixers take one
    sequence at a time."""

    def __init__(self, config, weights: _Weights, tokens: List[List[int]]):
        self.c, self.w = config, weights
        self.cuts = np.cumsum([0] + [len(t) for t in tokens]).tolist()
        self.tokens = tokens
        self.ids = torch.tensor(sum(tokens, []), device="cuda")
        self.eps = config["rms_norm_eps"] if "hidden_size" in config else config["norm"]["eps"]

    def each(self, fn, *rows):
        return torch.cat([fn(*(r[a:b] for r in rows)) for a, b in zip(self.cuts, self.cuts[1:])])

    def order(self):
        n, loop = len(self.c["layers"]), self.c.get("loop")
        if not loop:
            return [(i, False) for i in range(n)]
        a, b = loop["start"], loop["stop"]
        return ([(i, False) for i in range(a)] + [(i, i == a) for _ in range(loop["times"]) for i in range(a, b)]
                + [(i, False) for i in range(b, n)])

    def lin(self, h, name, bias=False):
        y = h @ self.w[name].T
        return y + self.w[name + ".b"] if bias else y

    def first_of(self, size, kind, T):
        i = torch.arange(T, device="cuda")
        return (i - size + 1).clamp(min=0) if kind == "window" else i // size * size

    def streams(self, fn, x, p, q):
        """A hyper-connected sublayer on ``x`` ``[T, streams, W]``."""
        w, n = self.w, f"{p}hc{q}."
        h = _layer_norm(torch.einsum("s,tsw->tw", w[n + "in"], x), w[f"{p}norm{q}"], w[f"{p}norm{q}.b"], self.eps)
        return torch.einsum("sr,tsw->trw", w[n + "mix"], x) + w[n + "out"][:, None] * fn(h)[:, None]

    def glu(self, h, p, act=_silu):
        return self.lin(act(self.lin(h, p + "gate")) * self.lin(h, p + "up"), p + "down")

    # ---- MiniMax-M3
    def minimax_m3(self):
        c, w, eps = self.c, self.w, self.eps
        one = 1.0 if c["use_gemma_norm"] else 0.0
        H, G, D = c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"]
        freqs = _plain_frequencies(c["rope_theta"], c["rotary_dim"])
        x = w.rows("model.embed_tokens.weight", self.ids)
        for i in range(c["num_hidden_layers"]):
            p = f"model.layers.{i}."
            h = _rms(x, eps) * (w[p + "input_layernorm.weight"] + one)
            a = p + "self_attn."
            qn, kn = w[a + "q_norm.weight"] + one, w[a + "k_norm.weight"] + one
            q, k, v = (self.lin(h, a + n + "_proj.weight") for n in "qkv")
            if c["qk_norm_type"] == "per_layer":
                q, k = _rms(q, eps) * qn, _rms(k, eps) * kn
            q, k, v = q.view(-1, H, D), k.view(-1, G, D), v.view(-1, G, D)
            if c["qk_norm_type"] == "per_head":
                q, k = _rms(q, eps) * qn, _rms(k, eps) * kn
            o = self.each(lambda q, k, v: _attend(_rotate(q, freqs), _rotate(k, freqs), v, D ** -0.5), q, k, v)
            x = x + self.lin(o.flatten(1), a + "o_proj.weight")
            h = _rms(x, eps) * (w[p + "post_attention_layernorm.weight"] + one)
            m = p + "block_sparse_moe."
            s = torch.sigmoid(self.lin(h, m + "gate.weight"))
            ids = (s + w[m + "e_score_correction_bias"]).topk(c["num_experts_per_tok"], -1).indices
            picked = s.gather(1, ids)
            x = x + _experts(h, ids, picked / (picked.sum(-1, keepdim=True) + 1e-20), lambda e, r: self.lin(
                _silu(self.lin(r, f"{m}experts.{e}.w1.weight")) * self.lin(r, f"{m}experts.{e}.w3.weight"),
                f"{m}experts.{e}.w2.weight"))
        return _rms(x, eps) * (w["model.norm.weight"] + one), "lm_head.weight"

    # ---- Fazinex
    def fazinex(self):
        c, w, eps = self.c, self.w, self.eps
        x = _rms(w.rows("embed", self.ids), eps) * w["embed.norm"]
        for i, _ in self.order():
            layer, p = c["layers"][i], f"l{i}."
            m, n = layer["mixer"], p + "mix."
            h = _rms(x, eps) * w[p + "norm1"]
            H, D = m["heads"], m["dim"]
            q = self.lin(h, n + "q").view(-1, H, D)
            if layer["type"] == "attention":
                k = self.lin(h, n + "k").view(-1, m["kv_heads"], D)

                def attend(q, k):
                    at = torch.arange(q.shape[0], device="cuda")
                    warmth = 1.0 + m["q_temp"]["coef"] * torch.log(((at + 1) // m["q_temp"]["every"]).to(F64) + 1.0)
                    return _attend(q * warmth[:, None, None], k, k, m["scale"])
                o = self.each(attend, q, k)
            else:
                latent = _rms(self.lin(h, n + "dkv"), eps) * w[n + "dkv.norm"]
                k, v = self.lin(latent, n + "uk").view(-1, H, D), self.lin(latent, n + "uv").view(-1, H, m["vdim"])
                o = self.each(lambda q, k, v: _attend(q, k, v, m["scale"]), q, k, v)
                o = o * torch.sigmoid(self.lin(h, n + "g"))[:, :, None]
            y = self.lin(o.flatten(1), n + "o")
            if layer.get("mlp"):
                y = y + self.lin(torch.relu(self.lin(h, p + "mlp.up")) ** 2, p + "mlp.down")
            x = x + y
        return _rms(x, eps) * w["final.norm"], "embed"

    # ---- Tonapel
    def tonapel(self):
        c, w, eps = self.c, self.w, self.eps
        norm = lambda v, name: _rms(v, eps) * (1.0 + w[name])
        x = w.rows("embed", self.ids)
        for i, layer in enumerate(c["layers"]):
            p, m, mlp = f"l{i}.", layer["mixer"], layer["mlp"]
            mixer = self.tonapel_parallel if layer["type"] == "parallel" else self.tonapel_delta
            y = mixer(norm(x, p + "norm1"), p + "mix.", m)
            x = x + c["residual_mult"] * norm(y, p + "norm1b")
            h, f = norm(x, p + "norm2"), p + "mlp."
            if mlp["kind"] == "dense":
                y = self.glu(h, f, _gelu)
            else:
                best = self.lin(h, f + "router").topk(mlp["router"]["top"], -1)
                y = _experts(h, best.indices, torch.softmax(best.values, -1), lambda e, r: self.lin(_swiglu_clamped(
                    self.lin(r, f"{f}e{e}.gate"), self.lin(r, f"{f}e{e}.up"), mlp["expert"]["limit"]), f"{f}e{e}.down"))
            x = x + c["residual_mult"] * norm(y, p + "norm2b")
        return norm(x, "final.norm"), "head"

    def tonapel_parallel(self, h, p, m):
        w, a, r, n = self.w, m["left"], m["right"], p + "left."
        H, G = a["heads"], a["kv_heads"]
        freqs = _plain_frequencies(a["rot"]["base"], a["rot"]["dims"])
        q, k, v = (self.lin(h, n + s, True) for s in "qkv")
        o = self.each(lambda q, k, v: _attend(_rotate(q, freqs), _rotate(k, freqs), v, a["scale"],
                                              self.first_of(a["mask"]["size"], "window", q.shape[0])),
                      q.view(-1, H, a["dim"]), k.view(-1, G, a["dim"]), v.view(-1, G, a["vdim"]))
        left = self.lin(o.flatten(1), n + "o", True)
        n = p + "right."
        H, P, N, G = r["heads"], r["vdim"], r["state"], r["groups"]
        inner = H * P
        z, xbc, dt = self.lin(h, n + "in").split([inner, inner + 2 * G * N, H], -1)

        def scan(xbc, dt):
            u, b, read = _silu(_conv(xbc, w[n + "conv"]) + w[n + "conv.b"]).split([inner, G * N, G * N], -1)
            step = _softplus(dt + w[n + "dt_bias"])
            u = u.view(-1, H, P)
            per_head = lambda v: v.view(-1, G, N).repeat_interleave(H // G, 1)
            y = _state_loop(per_head(b), step[:, :, None] * u, per_head(read), torch.exp(-torch.exp(w[n + "A_log"]) * step))
            return (y + w[n + "D"][:, None] * u).flatten(1)
        y = self.each(scan, xbc, dt) * _silu(z)
        parts = r["norm_groups"]
        y = _rms(y.view(-1, parts, inner // parts), self.eps).flatten(1) * w[n + "norm"]
        return m["left_scale"] * left + m["right_scale"] * self.lin(y, n + "o")

    def _unit(self, v):
        return v / torch.sqrt((v * v).sum(-1, keepdim=True) + 1e-6)

    def _delta_qkv(self, q, k, v, n, m):
        """Convolutions and unit norms of one sequence; key heads repeated for the heads they serve."""
        H, G, D = m["heads"], m["kv_heads"], m["dim"]
        q, k = (self._unit(_silu(_conv(u, self.w[f"{n}{s}.conv"])).view(-1, G, D)).repeat_interleave(H // G, 1)
                for u, s in ((q, "q"), (k, "k")))
        return q * D ** -0.5, k, _silu(_conv(v, self.w[n + "v.conv"])).view(-1, H, m["vdim"])

    def tonapel_delta(self, h, p, m):
        w = self.w
        q, k, v, a, b = (self.lin(h, p + s) for s in "qkvab")

        def scan(q, k, v, a, b):
            q, k, v = self._delta_qkv(q, k, v, p, m)
            decay = torch.exp(-torch.exp(w[p + "A_log"]) * _softplus(a + w[p + "dt_bias"]))
            return _state_loop(k, v, q, decay, torch.sigmoid(b))
        o = _rms(self.each(scan, q, k, v, a, b), self.eps) * w[p + "norm"]
        return self.lin(o.flatten(1) * _silu(self.lin(h, p + "g")), p + "o")

    # ---- Nirelix
    def nirelix(self):
        c, w, eps = self.c, self.w, self.eps
        x = w.rows("embed", self.ids)[:, None].repeat(1, c["streams"], 1)
        for i, layer in enumerate(c["layers"]):
            p, m, mlp = f"l{i}.", layer["mixer"], layer["mlp"]
            mixer = getattr(self, "nirelix_" + layer["type"])
            x = self.streams(lambda h: mixer(h, p + "mix.", m), x, p, 1)
            f = p + "mlp."
            if mlp["kind"] == "dense":
                x = self.streams(lambda h: self.lin(_swiglu_clamped(self.lin(h, f + "gate"), self.lin(h, f + "up"),
                                                                    mlp["limit"]), f + "down"), x, p, 2)
            else:
                x = self.streams(lambda h: self.nirelix_experts(h, f, mlp["router"]), x, p, 2)
        return _layer_norm(x.sum(1), w["final.norm"], w["final.norm.b"], eps), "head"

    def nirelix_experts(self, h, f, r):
        s = torch.sigmoid(self.lin(h, f + "router"))
        ids = _grouped_choice(s + self.w[f + "correction"], r["top"], r["groups"],
                              lambda v: v.topk(min(2, v.shape[-1]), -1).values.sum(-1))
        picked = s.gather(1, ids)
        return _experts(h, ids, picked / (picked.sum(-1, keepdim=True) + 1e-20) * r["scale"],
                        lambda e, rows: self.glu(rows, f"{f}e{e}."))

    def nirelix_retention(self, h, p, m):
        H, D, P = m["heads"], m["dim"], m["vdim"]
        freqs = _plain_frequencies(m["rot"]["base"], m["rot"]["dims"])
        decay = torch.tensor(m["decay"], dtype=F64, device="cuda")
        q, k, v = (self.lin(h, p + s) for s in "qkv")
        o = self.each(lambda q, k, v: _state_loop(_rotate(k, freqs) * D ** -0.5, v, _rotate(q, freqs),
                                                  decay.expand(q.shape[0], H)),
                      q.view(-1, H, D), k.view(-1, H, D), v.view(-1, H, P))
        return self.lin(_rms(o, self.eps).flatten(1) * _silu(self.lin(h, p + "g")), p + "o")

    def nirelix_channel_delta(self, h, p, m):
        w, H, D = self.w, m["heads"], m["dim"]
        q, k, v, b = (self.lin(h, p + s) for s in "qkvb")
        a = self.lin(self.lin(h, p + "a1"), p + "a2")

        def scan(q, k, v, a, b):
            q, k, v = self._delta_qkv(q, k, v, p, m)
            decay = torch.exp(-torch.exp(w[p + "A_log"])[:, None] * _softplus(a + w[p + "dt_bias"]).view(-1, H, D))
            return _state_loop(k, v, q, decay, torch.sigmoid(b))
        o = _rms(self.each(scan, q, k, v, a, b), self.eps) * w[p + "norm"]
        return self.lin(o.flatten(1) * torch.sigmoid(self.lin(self.lin(h, p + "g1"), p + "g2")), p + "o")

    def _latent(self, h, q, p, m, freqs, pairs, first):
        """Attention of keys and values made from a normed latent row, beside one rotated key part."""
        H, D, R, rank = m["heads"], m["dim"], m["rot_dim"], m["kv_rank"]
        down = self.lin(h, p + "dkv")
        latent = _rms(down[:, :rank], self.eps) * self.w[p + "dkv.norm"]
        k, v = self.lin(latent, p + "uk").view(-1, H, D), self.lin(latent, p + "uv").view(-1, H, m["vdim"])

        def attend(q, k, shared, v):
            q = torch.cat([q[..., :D], _rotate(q[..., D:], freqs, pairs=pairs)], -1)
            k = torch.cat([k, _rotate(shared[:, None], freqs, pairs=pairs).expand(-1, H, -1)], -1)
            return _attend(q, k, v, m["scale"], first(q.shape[0]))
        return self.each(attend, q.view(-1, H, D + R), k, down[:, rank:], v).flatten(1)

    def nirelix_latent_attention(self, h, p, m):
        q = self.lin(_rms(self.lin(h, p + "dq"), self.eps) * self.w[p + "dq.norm"], p + "uq")
        o = self._latent(h, q, p, m, _plain_frequencies(m["rot"]["base"], m["rot"]["dims"]), True,
                         lambda T: self.first_of(m["mask"]["size"], "window", T))
        return self.lin(o * torch.sigmoid(self.lin(h, p + "g")), p + "o")

    # ---- Mezapel
    def mezapel(self):
        c, w, eps = self.c, self.w, self.eps
        big = c["embedding"]["bigram"]
        rows = []
        for seq in self.tokens:
            rows += [big["buckets"]] + [(a * big["mul_prev"] + b * big["mul_cur"]) % big["buckets"]
                                        for a, b in zip(seq, seq[1:])]
        x = w.rows("embed", self.ids) * c["embedding"]["scale"] + w.rows("bigram", torch.tensor(rows, device="cuda"))
        x = x[:, None].repeat(1, c["streams"], 1)
        for i, _ in self.order():
            layer, p = c["layers"][i], f"l{i}."
            mixer = self.mezapel_chunked if layer["type"] == "attention" else self.mezapel_windowed
            x = self.streams(lambda h: mixer(h, p + "mix.", layer["mixer"]), x, p, 1)
            x = self.streams(lambda h: self.glu(h, p + "mlp."), x, p, 2)
        return _layer_norm(x.sum(1), w["final.norm"], w["final.norm.b"], eps), "head"

    def mezapel_chunked(self, h, p, m):
        w, H, G = self.w, m["heads"], m["kv_heads"]
        freqs, size = _yarn(m["rot"]["base"], m["rot"]["dims"], m["rot"]["scaling"])
        q = _rms(self.lin(h, p + "q"), self.eps) * w[p + "q.norm"]
        k = _rms(self.lin(h, p + "k"), self.eps) * w[p + "k.norm"]
        none = torch.zeros(H, dtype=F64, device="cuda")            # the 1 in 1 + sum exp(s)
        o = self.each(lambda q, k, v: _attend(_rotate(q, freqs, size), _rotate(k, freqs, size), v, m["scale"],
                                              self.first_of(m["mask"]["size"], "chunk", q.shape[0]), sink=none),
                      q.view(-1, H, m["dim"]), k.view(-1, G, m["dim"]), self.lin(h, p + "v").view(-1, G, m["vdim"]))
        return self.lin((o * torch.sigmoid(self.lin(h, p + "g"))[:, :, None]).flatten(1), p + "o")

    def mezapel_windowed(self, h, p, m):
        w, H, G = self.w, m["heads"], m["kv_heads"]
        freqs, size = _llama3(m["rot"]["base"], m["rot"]["dims"], m["rot"]["scaling"])

        def attend(q, k, v):
            q, k, v = (_conv(u, w[f"{p}{s}.conv"]) for u, s in ((q, "q"), (k, "k"), (v, "v")))
            q = _rms(q.view(-1, H, m["dim"]), self.eps) * w[p + "q.norm"]
            k = _rms(k.view(-1, G, m["dim"]), self.eps) * w[p + "k.norm"]
            return _attend(_rotate(q, freqs, size), _rotate(k, freqs, size), v.view(-1, G, m["vdim"]), m["scale"],
                           self.first_of(m["mask"]["size"], "window", q.shape[0]), m["softcap"], w[p + "sink"])
        o = self.each(attend, *(self.lin(h, p + s) for s in "qkv"))
        return self.lin(o.flatten(1) * torch.sigmoid(self.lin(h, p + "g")), p + "o")

    # ---- Dizatar
    def dizatar(self):
        c, w, eps, mult = self.c, self.w, self.eps, self.c["residual_mult"]
        embedded = x = w.rows("embed", self.ids)
        for i, starts_pass in self.order():
            layer, p = c["layers"][i], f"l{i}."
            m, mlp, n = layer["mixer"], layer["mlp"], p + "mix."
            if starts_pass:
                x = self.lin(torch.cat([x, embedded], -1), "loop.in")
            h = _rms(x, eps) * w[p + "norm1"]
            y = self._latent(h, self.lin(h, n + "q"), n, m, _plain_frequencies(m["rot"]["base"], m["rot_dim"]), False,
                             lambda T: None)
            x = x + mult * w[p + "ls1"] * (_rms(self.lin(y, n + "o"), eps) * w[p + "norm1b"])
            h, f, r = _rms(x, eps) * w[p + "norm2"], p + "mlp.", mlp["router"]
            s = torch.softmax(self.lin(h, f + "router"), -1)
            ids = (s + w[f + "correction"]).topk(r["top"], -1).indices
            picked = s.gather(1, ids)
            y = _experts(h, ids, picked / (picked.sum(-1, keepdim=True) + 1e-20),
                         lambda e, rows: rows if e >= r["experts"] else self.glu(rows, f"{f}e{e}."))
            y = y + self.glu(h, f + "shared.")
            x = x + mult * w[p + "ls2"] * (_rms(y, eps) * w[p + "norm2b"])
        return _rms(x, eps) * w["final.norm"], "head"

    # ---- Besuzen
    def besuzen(self):
        c, w, eps = self.c, self.w, self.eps
        x = w.rows("embed", self.ids) * c["embedding"]["scale"]
        first = None
        for i, layer in enumerate(c["layers"]):
            p, m, mlp = f"l{i}.", layer["mixer"], layer["mlp"]
            h, g = (_layer_norm(x, w[p + n], 0.0, eps) for n in ("norm1", "norm2"))
            if layer["type"] == "attention":
                n = p + "mix."
                freqs = _plain_frequencies(m["rot"]["base"], m["rot"]["dims"])
                q, k, v = self.besuzen_qkv(h, n, m)
                if first is None:
                    first = v
                else:
                    v = (1.0 - w[n + "vmix"]) * v + w[n + "vmix"] * first
                o = self.each(lambda q, k, v: _attend(_rotate(q, freqs, pairs=True), _rotate(k, freqs, pairs=True), v,
                                                      m["scale"]), q, k, v)
                y = self.lin(o.flatten(1) * torch.sigmoid(self.lin(h, n + "g")), n + "o")
            else:
                n, a = p + "mix.left.", m["left"]
                o = self.each(lambda q, k, v: _attend(q, k, v, a["scale"]), *self.besuzen_qkv(h, n, a))
                left = self.lin((o * torch.sigmoid(self.lin(h, n + "g"))[:, :, None]).flatten(1), n + "o")
                y = m["left_scale"] * left + m["right_scale"] * self.besuzen_time_mixing(h, p + "mix.right.", m["right"])
            f = p + "mlp."
            if mlp["kind"] == "dense":
                x = x + y + self.glu(g, f, _gelu)
                continue
            s, r = torch.softmax(self.lin(g, f + "router"), -1), mlp["router"]
            ids = _grouped_choice(s, r["top"], r["groups"], lambda v: v.amax(-1))
            picked = s.gather(1, ids)
            z = _experts(g, ids, picked / (picked.sum(-1, keepdim=True) + 1e-20), lambda e, rows: self.glu(rows, f"{f}e{e}."))
            x = x + y + z + torch.sigmoid(self.lin(g, f + "shared.sg")) * self.glu(g, f + "shared.")
        return _layer_norm(x, w["final.norm"], 0.0, eps) * c["logit_scale"], "head"

    def besuzen_qkv(self, h, n, m):
        q, k, v = (self.lin(h, n + s, True) for s in "qkv")
        return q.view(-1, m["heads"], m["dim"]), k.view(-1, m["kv_heads"], m["dim"]), v.view(-1, m["kv_heads"], m["vdim"])

    def besuzen_time_mixing(self, h, p, m):
        w, H, D = self.w, m["heads"], m["dim"]
        before = self.each(lambda h: torch.cat([torch.zeros_like(h[:1]), h[:-1]]), h)
        r, k, v, g = (self.lin(h + (before - h) * w[f"{p}mu.{s}"], p + s) for s in "rkvg")
        low = torch.tanh(self.lin(h + (before - h) * w[p + "mu.w"], p + "w1"))
        decay = torch.exp(-torch.exp(self.lin(low, p + "w2") + w[p + "w0"]))
        o = self.each(lambda r, k, v, d: _state_loop(k, v, r, d, bonus=w[p + "u"]),
                      *(u.view(-1, H, D) for u in (r, k, v, decay)))
        return self.lin(_rms(o, self.eps).flatten(1) * w[p + "norm"] * _silu(g), p + "o")


def exact(case: Case, seed: int) -> Optional[torch.Tensor]:
    config = model_config(case)
    tokens = sum(prompt_lengths(case)) + case["requests"] * (case["answer"] - 1)
    loops = 0 if "hidden_size" in config else sum("state" in m for layer in _mixers(config) for m in layer)
    # about 20 us an operation of a token-by-token loop, 20 TFLOP/s of 64-bit products
    if loops * tokens * 1.5e-4 + work(case)["flops"] / 2e13 > 18.0:
        return None
    engine = _engine(case, seed)
    ids = _token_ids(case, seed, engine.vocab_size)
    weights = _Weights(engine)
    decoder = _Decoder(config, weights, ids)
    x, head = getattr(decoder, case["model"])()
    rows = [decoder.cuts[i] + b - 1 for entries in schedule(case) for i, _, b, wants in entries if wants]
    logits = x[torch.tensor(rows, device="cuda")] @ weights[head].T
    cap = config.get("logit_softcap")
    return cap * torch.tanh(logits / cap) if cap else logits
