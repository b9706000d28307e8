"""What this framework is measured by: conversations served through the step function.

A case is a model (a preset, or a preset's sizes at the 32-bit path), some requests that are live at once, the length of the
longest prompt, and how many tokens every request decodes after it.  One pass takes every request in, feeds its prompt (whole, or
in portions), decodes token by token and lets the request go, as a serving program does; the tokens are given, so that a pass does
not depend on how near two logits lie.  What comes back are the 32-bit logits of every prompt's last token and of every decoded
token and, on the 32-bit path, the tokens that the sampler chooses from them.

The weights are drawn from the seed with the distributions of the package's random mode (no checkpoints are at hand); the sizes
are those of the presets.
"""

from __future__ import annotations

import math
import random
import re
import zlib

import torch

from llmserve_triton_kernels_b200.cache import CacheManager
from llmserve_triton_kernels_b200.config.presets import PRESETS
from llmserve_triton_kernels_b200.config.registry import architecture_of
from llmserve_triton_kernels_b200.engine.batch import StepEntry
from llmserve_triton_kernels_b200.engine.step import StepFunction
from llmserve_triton_kernels_b200.models.load import resolve_dtype
from llmserve_triton_kernels_b200.models.model import Model
from llmserve_triton_kernels_b200.sampling import Sampler, SamplingParams

DEVICE = "cuda:0"
PAGE = 16
SLOTS = 8  # live requests an engine has room for, unless told otherwise
BUDGET = 4096  # tokens of a step, unless told otherwise
F64 = torch.float64


def listed():
    """``requests`` live at once; ``prompt``: the longest prompt (the others are ragged fractions of it); ``portion``: a prompt is
    fed in portions of so many tokens (0: whole); ``late``: the last request arrives while the others decode already, so that its
    portions ride beside their tokens; ``decode``: tokens every request decodes."""

    def case(name, model, requests, prompt, decode, portion=0, late=False, dtype="bfloat16"):
        return {"name": name, "model": model, "dtype": dtype, "requests": requests, "prompt": prompt, "portion": portion, "late": late, "decode": decode}

    return [
        # the smallest call: one user's short question to a small model, where launches and latency count
        case("nurolorn_small_short_chat", "nurolorn-small", 1, 9, 8),
        # one user's short question to the model that the repository is measured by
        case("llama_short_chat", "tinyllama-1.1b", 1, 13, 16),
        # a full batch of users at ragged lengths, decoding for a while
        case("llama_batch_of_8", "tinyllama-1.1b", 8, 509, 24),
        # one long document, whole, and the first words of an answer
        case("llama_long_prompt", "tinyllama-1.1b", 1, 2041, 2),
        # the 32-bit path, as replays of traces use it, with the sampler
        case("llama_float32", "tinyllama-1.1b", 2, 150, 6, dtype="float32"),
        # the largest model: four users, one of whom arrives while the others decode
        case("llama3_8b_late_arrival", "llama3-8b", 4, 701, 6, portion=512, late=True),
        # the other designs at their 1b sizes: a long prompt, ordinary ones, portions, one user, full batches
        case("nurolorn_long_prompt", "nurolorn-1b", 1, 1500, 8),
        case("kafepel_batch_of_4", "kafepel-1b", 4, 600, 12),
        case("nudodra_long_prompt", "nudodra-1b", 1, 1801, 6),
        case("tenotar_one_user", "tenotar-1b", 1, 120, 24),
        case("pefedra_batch_of_8", "pefedra-1b", 8, 400, 12),
        case("zifuzen_portions", "zifuzen-1b", 3, 1030, 12, portion=512, late=True),
    ]


MODELS = ("tinyllama-1.1b", "nurolorn-small", "nurolorn-1b", "kafepel-small", "kafepel-1b", "nudodra-small", "nudodra-1b", "tenotar-small",
          "tenotar-1b", "pefedra-small", "pefedra-1b", "zifuzen-small", "zifuzen-1b")


def draw(rng):
    """A conversation of the same ranges: any of the designs, 1 to 8 requests, prompts of 5 to 2,041 tokens, 1 to 24 decoded."""
    largest = max(_cost(c) for c in listed())
    while True:
        dtype = "float32" if rng.random() < 0.12 else "bfloat16"
        case = {
            "model": rng.choice(MODELS), "dtype": dtype, "requests": rng.choice((1, 1, 2, 3, 4, 5, 6, 7, 8)),
            "prompt": int(round(math.exp(rng.uniform(math.log(5), math.log(160 if dtype == "float32" else 2041))))),
            "portion": rng.choice((0, 0, 256, 384, 512)), "late": False, "decode": int(round(math.exp(rng.uniform(0, math.log(24))))),
        }
        case["late"] = case["requests"] > 1 and rng.random() < 0.3
        tokens = sum(_prompt_lengths(case))
        # the 32-bit path runs on the CUDA cores: what it is given stays as small as the listed case
        if _cost(case) <= largest and tokens <= (300 if dtype == "float32" else BUDGET):
            return case


def _cost(case):
    w = work(case)
    return max(w["bytes"], w["flops"] / 50)


# ---------------------------------------------------------------------------------------------- the conversation
def _prompt_lengths(case):
    """Ragged, from the sizes alone: the first request's prompt is the longest."""
    part = (1.0, 0.61, 0.87, 0.33, 0.72, 0.49, 0.94, 0.21)
    return [max(1, int(round(case["prompt"] * part[r % 8]))) for r in range(case["requests"])]


def _steps(case):
    """The steps of a pass: lists of (request, first token, tokens, places wanted), under the step's token budget.  The last
    token of a prompt and every decoded token want their logits."""
    lengths, portion = _prompt_lengths(case), case["portion"] or BUDGET
    ends = [n + case["decode"] for n in lengths]
    at = [0] * len(lengths)
    steps, arrived = [], len(lengths) - (1 if case["late"] else 0)
    while any(a < e for a, e in zip(at, ends)):
        budget, step = BUDGET, []
        for decoding in (True, False):
            for r in range(arrived):
                if at[r] >= ends[r] or (at[r] >= lengths[r]) != decoding or not budget:
                    continue
                n = 1 if decoding else min(lengths[r] - at[r], portion, budget)
                step.append((r, at[r], n, [n - 1] if at[r] + n >= lengths[r] else []))
                budget -= n
        step.sort()
        for r, _, n, _ in step:
            at[r] += n
        steps.append(step)
        if arrived < len(lengths) and (all(a >= n for a, n in zip(at[:arrived], lengths))):
            arrived = len(lengths)
    return steps


def _rows(case):
    return sum(len(want) for step in _steps(case) for *_, want in step)


def _tokens(case, seed, vocab):
    rng = random.Random(int(seed) * 7919 + 17)
    return [[rng.randrange(vocab) for _ in range(n + case["decode"])] for n in _prompt_lengths(case)]


# ---------------------------------------------------------------------------------------------- weights
def _generator(name, seed):
    return torch.Generator(device=DEVICE).manual_seed((int(seed) * 1_000_003 + zlib.crc32(name.encode())) % 2**63)


def _tensor(name, spec, seed, layers, scaled):
    """One tensor with the distribution of the package's random mode (stored in bfloat16), drawn on the GPU.  Matrices that write
    to the residual stream are smaller by sqrt(2 layers), as models are initialised and as trained ones are: a model of 32 layers
    otherwise doubles a rounding error every few layers, which says nothing about the kernels."""
    shape = tuple(spec.free_size if d == -1 else d for d in spec.shape)
    g = _generator(name, seed)
    if spec.init == "zeros":
        return torch.zeros(shape, dtype=torch.bfloat16, device=DEVICE)
    if spec.init.startswith("distinct:"):
        count = int(spec.init.split(":")[1])
        return torch.rand((shape[0], count), generator=g, device=DEVICE).argsort(dim=1)[:, : shape[1]].to(torch.int32).contiguous()
    x = torch.randn(shape, generator=g, device=DEVICE).mul_(0.02)
    if re.search(r"(\.o|\.down|o_proj\.weight|down_proj\.weight)$", name):
        x *= (2 * layers) ** -0.5
    elif name in ("embed", "model.embed_tokens.weight") and not scaled:
        x *= 25.0  # tokens' rows of the size that the other designs' factor on the embedding gives them
    base = {"normal": 0.0, "ones_plus_normal": 1.0, "half_plus_normal": 0.5, "mean_plus_normal": 1.0 / (shape or (1,))[-1]}
    if spec.init == "eye_plus_normal":
        x += torch.eye(*shape, device=DEVICE)
    else:
        x += base[spec.init]
    return x.to(torch.bfloat16)


def _plan(case):
    arch = architecture_of(PRESETS[case["model"]])
    return arch, arch.plan(arch.config_class.from_dict(PRESETS[case["model"]]))


def _weights(case, seed):
    arch, plan = _plan(case)
    specs = (arch.model_class or Model)(plan, torch.bfloat16, "cpu").tensor_specs()
    scaled = plan.embedding_scale != 1.0
    tensors = {name: _tensor(name, spec, seed, len(plan.schedule), scaled) for name, spec in specs.items()}
    _train_routers(PRESETS[case["model"]], tensors, seed)
    return tensors


def _train_routers(cfg, tensors, seed):
    """Routers that tell tokens apart as trained ones do, mostly by the token itself: every token id has ``top`` features of as many
    as there are experts in its embedding, and every layer gives every feature to an expert of its own.  Which experts a token uses
    is then as random as with random rows, and evenly spread; but random rows leave the border of the chosen within bfloat16's
    rounding for every tenth token, and no two orders of the same sums would choose the same experts."""
    routed = [i for i, layer in enumerate(cfg.get("layers", ())) if f"l{i}.mlp.router" in tensors]
    if not routed:
        return
    router, embed = cfg["layers"][routed[0]]["mlp"]["router"], tensors["embed"]
    experts, groups = router["experts"], router.get("groups") or {"count": 1, "keep": 1}
    (vocab, width), run, keep = embed.shape, experts // groups["count"], groups["keep"]
    g = _generator("features", seed)
    directions = torch.nn.functional.normalize(torch.randn((experts, width), generator=g, device=DEVICE), dim=1)
    # a token's features: from ``keep`` of the runs of neighbours, as many of each
    runs = torch.rand((vocab, groups["count"]), generator=g, device=DEVICE).argsort(1)[:, :keep]
    within = torch.rand((vocab, keep, run), generator=g, device=DEVICE).argsort(2)[:, :, : router["top"] // keep]
    features = (runs[:, :, None] * run + within).flatten(1)
    strength = 60.0 / (cfg.get("embedding") or {"scale": 1.0})["scale"]
    tensors["embed"] = (embed.float() + strength * directions[features].sum(1)).to(torch.bfloat16)
    for i in routed:
        g = _generator(f"l{i}.features", seed)
        order = torch.rand((groups["count"], run), generator=g, device=DEVICE).argsort(1)
        mine = (torch.rand(groups["count"], generator=g, device=DEVICE).argsort()[:, None] * run + order).flatten()
        name = f"l{i}.mlp.router"
        tensors[name] = (0.1 * tensors[name].float() + (0.1 if groups["count"] > 1 else 0.25) * directions[mine]).to(torch.bfloat16)


def prepare(case, seed):
    """A loaded model with its cache and step function, and the tokens of a conversation."""
    arch, plan = _plan(case)
    dtype = resolve_dtype(case["dtype"])
    model = (arch.model_class or Model)(plan, dtype, DEVICE)
    model.bind(_weights(case, seed))
    pages = SLOTS * -(-(plan.max_positions or BUDGET) // PAGE)
    cache = CacheManager(model.cache_specs(), plan.schedule, page_size=PAGE, num_pages=pages, max_requests=SLOTS, dtype=dtype, device=DEVICE)
    tokens = _tokens(case, seed, plan.vocab_size)
    steps = [[(r, tokens[r][a : a + n], want) for r, a, n, want in step] for step in _steps(case)]
    state = {
        "step": StepFunction(model, cache), "cache": cache, "steps": steps, "requests": case["requests"],
        "logits": torch.empty((_rows(case), plan.vocab_size), dtype=torch.float32, device=DEVICE), "sampler": None,
    }
    if case["dtype"] == "float32":
        state["sampler"], state["params"] = Sampler(torch.device(DEVICE)), SamplingParams()
    return state


def run(state):
    """One conversation: logits ``[wanted places, vocab]`` in the order of the steps (and the sampled tokens)."""
    out, at, chosen = state["logits"], 0, []
    for step in state["steps"]:
        logits = state["step"]([StepEntry(r, tokens, want) for r, tokens, want in step])
        n = logits.shape[0]
        if n:
            out[at : at + n].copy_(logits)
            at += n
            if state["sampler"] is not None:
                chosen += state["sampler"](logits, [state["params"]] * n, [0] * n, [0] * n)
    for r in range(state["requests"]):
        state["cache"].free_request(r)
    return (out, torch.tensor(chosen, dtype=torch.int32)) if state["sampler"] is not None else (out,)


# ---------------------------------------------------------------------------------------------- what a pass cannot do without
def _layer_runs(cfg):
    """How often every layer runs in a step."""
    if "layers" not in cfg:
        return [1] * cfg["num_hidden_layers"]
    runs, loop = [1] * len(cfg["layers"]), cfg.get("loop")
    for i in range(loop["start"], loop["stop"]) if loop else ():
        runs[i] = loop["times"]
    return runs


def _keys_per_query(cfg):
    """For every layer, once a run: (span of keys or None, flops a query and key pair, elements kept a key, elements of state)."""
    out = []
    if "layers" not in cfg:
        heads, d = cfg["num_attention_heads"], cfg["hidden_size"] // cfg["num_attention_heads"]
        return [(None, 4 * heads * d, 2 * cfg["num_key_value_heads"] * d, 0)] * cfg["num_hidden_layers"]
    for layer, times in zip(cfg["layers"], _layer_runs(cfg)):
        m, one = layer["mixer"], []
        for part in ([m["left"], m["right"]] if "left" in m else [m]):
            span = (part.get("mask") or {}).get("size")
            if "kv_rank" in part:
                one.append((span, 2 * part["heads"] * (part["dim"] + part["rot_dim"] + part["vdim"]), part["kv_rank"] + part["rot_dim"], 0))
            elif "scale" in part:
                maps = 2 if part.get("diff") is not None else 1
                one.append((span, 2 * maps * part["heads"] * (part["dim"] + part["vdim"]), part["kv_heads"] * (maps * part["dim"] + part["vdim"]), 0))
            elif "width" in part:
                one.append((0, 0, 0, part["width"]))
            else:
                one.append((0, 0, 0, part["heads"] * part["dim"] * part["vdim"]))
        out += one * times
    return out


def work(case):
    """Bytes: every weight that a step's tokens use, once a step; keys and state that are read and written; logits.
    Flops: two a weight and token, and those of every visible (query, key) pair."""
    cfg = PRESETS[case["model"]]
    arch, plan = _plan(case)
    specs = (arch.model_class or Model)(plan, torch.bfloat16, "cpu").tensor_specs()
    size = 4 if case["dtype"] == "float32" else 2
    runs, mixers = _layer_runs(cfg), _keys_per_query(cfg)
    plain, routed, experts, top = 0.0, 0.0, 1, 1
    for name, spec in specs.items():
        layer = re.match(r"(?:model\.layers\.|l)(\d+)\.", name)
        if layer is None or len(spec.shape) != 2 or name.endswith("table"):
            continue
        n = math.prod(spec.free_size if d == -1 else d for d in spec.shape) * runs[int(layer.group(1))]
        if re.search(r"\.e\d+\.", name):
            routed += n
        else:
            plain += n
    for layer in cfg.get("layers", ()):
        if (layer.get("mlp") or {}).get("kind") == "moe":
            experts, top = layer["mlp"]["router"]["experts"], layer["mlp"]["router"]["top"]
    head = plan.vocab_size * plan.hidden_size
    total_bytes = total_flops = 0.0
    for step in _steps(case):
        tokens, rows = sum(n for _, _, n, _ in step), sum(len(w) for *_, w in step)
        used = 1.0 - (1.0 - top / experts) ** tokens
        total_bytes += size * (plain + used * routed + (head if rows else 0) + tokens * plan.hidden_size) + 4.0 * rows * plan.vocab_size
        total_flops += 2.0 * tokens * (plain + routed * top / experts) + 2.0 * rows * head
        for span, flops, kept, state in mixers:
            for _, start, n, _ in step:
                end = start + n
                seen = sum(min(p + 1, span) for p in range(start, end)) if span else (end * (end + 1) - start * (start + 1)) / 2
                total_flops += flops * seen + 4.0 * state * n
                total_bytes += size * kept * (min(end, span + n) if span else end) + 8.0 * state
    return {"bytes": total_bytes, "flops": total_flops}


def tolerance(case):
    """About four times what two orders of the same sums leave: 6e-7 of the result's norm on the 32-bit path, up to 0.005 with
    bfloat16 operands between the layers of a whole model, and 0.011 over the 32 layers of the largest one."""
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-4, "differ": 0.01}
    return {"rel": 0.03, "max": 0.25} if case["model"] == "llama3-8b" else {"rel": 0.015, "max": 0.12}


# ---------------------------------------------------------------------------------------------- the same in 64 bits
class _Weights:
    """The checkpoint's tensors in 64 bits, each when it is asked for."""

    def __init__(self, tensors, prefix=""):
        self.tensors, self.prefix = tensors, prefix

    def under(self, prefix):
        return _Weights(self.tensors, self.prefix + prefix)

    def has(self, name):
        return self.prefix + name in self.tensors

    def __call__(self, name):
        return self.tensors[self.prefix + name].to(F64)

    def linear(self, x, name):
        y = x @ self(name).T
        return y + self(name + ".b") if self.has(name + ".b") else y


def _rms(x, eps, weight=None):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if weight is None else y * weight


def _layer_norm(x, eps, weight):
    d = x - x.mean(-1, keepdim=True)
    return d / torch.sqrt((d * d).mean(-1, keepdim=True) + eps) * weight


def _silu(x):
    return x * torch.sigmoid(x)


def _frequencies(dims, base, scaling=None):
    f = float(base) ** (-2 * torch.arange(dims // 2, dtype=F64, device=DEVICE) / dims)
    if scaling and "low" in scaling:
        factor, low, high, original = (float(scaling[k]) for k in ("factor", "low", "high", "original"))
        wavelength = 2 * math.pi / f
        t = (original / wavelength - low) / (high - low)
        f = torch.where(wavelength < original / high, f, torch.where(wavelength > original / low, f / factor, (1 - t) * f / factor + t * f))
    elif scaling:
        f = f / float(scaling["factor"])
    return f


def _turn(x, f, neighbours=False, sign=1.0):
    """x [T, heads, D]: pairs of lanes (i, i + n), or (2i, 2i + 1), of the first 2n lanes turn by position * f_i."""
    n = f.numel()
    a = sign * torch.arange(x.shape[0], dtype=F64, device=x.device)[:, None] * f
    c, s = a.cos()[:, None], a.sin()[:, None]
    if neighbours:
        u, v = x[..., 0 : 2 * n : 2], x[..., 1 : 2 * n : 2]
        return torch.cat((torch.stack((u * c - v * s, v * c + u * s), -1).flatten(-2), x[..., 2 * n :]), -1)
    u, v = x[..., :n], x[..., n : 2 * n]
    return torch.cat((u * c - v * s, v * c + u * s, x[..., 2 * n :]), -1)


def _rotated(x, rot, neighbours=False):
    return _turn(x, _frequencies(rot["dims"], rot["base"], rot.get("scaling")), neighbours) if rot and rot.get("dims") else x


def _visible(T, window=None, keep=0, block=None):
    i, j = torch.arange(T, device=DEVICE)[:, None], torch.arange(T, device=DEVICE)[None]
    see = j <= i
    if window:
        see = see & ((i - j < window) | (j < keep))
    if block:
        see = see & (i // block == j // block)
    return see


def _attend(q, k, v, scale, see, cap=None, slopes=None, sink=None):
    """Softmax attention, a key/value head for every run of query heads."""
    H, T = q.shape[1], q.shape[0]
    k, v = (x.repeat_interleave(H // x.shape[1], dim=1) for x in (k, v))
    s = torch.einsum("ihd,jhd->hij", q, k) * float(scale)
    if cap:
        s = cap * torch.tanh(s / cap)
    if slopes is not None:
        i = torch.arange(T, device=q.device)
        s -= slopes[:, None, None] * (i[:, None] - i[None])
    s = s.masked_fill(~see, -math.inf)
    if sink is not None:
        s = torch.cat((s, sink[:, None, None].expand(H, T, 1)), -1)
    w = torch.softmax(s, -1)[..., :T]
    return torch.einsum("hij,jhd->ihd", w, v)


def _slopes(H):
    return 2.0 ** (-8.0 * torch.arange(1, H + 1, dtype=F64, device=DEVICE) / H)


def _heads(x, heads):
    return x.view(x.shape[0], heads, -1)


def _short_conv(u, w):
    taps = w.shape[1]
    padded = torch.cat((u.new_zeros(taps - 1, u.shape[1]), u))
    return sum(w[:, j] * padded[j : j + u.shape[0]] for j in range(taps))


def _recurrence(q, k, v, decay):
    """S <- decay_t S + k v^T, o = S^T q; decay [T, H, D] or [T, H, 1]."""
    S, out = v.new_zeros(q.shape[1], q.shape[2], v.shape[2]), []
    for t in range(q.shape[0]):
        S = torch.baddbmm(decay[t][:, :, None] * S, k[t][:, :, None], v[t][:, None])
        out.append(torch.bmm(q[t][:, None], S)[:, 0])
    return torch.stack(out)


def _pick(weights, x, expert):
    """Sum over experts of their weight times their output, each expert on the tokens that use it."""
    out = torch.zeros_like(x)
    for e in range(weights.shape[1]):
        mine = weights[:, e].nonzero()[:, 0]
        if mine.numel():
            out[mine] += weights[mine, e][:, None] * expert(x[mine], e)
    return out


def _chosen(scores, top):
    return torch.zeros_like(scores).scatter(1, scores.topk(top, dim=-1).indices, 1.0)


def _bounded(x, W, limit):
    g, u = torch.clamp(x @ W("gate").T, max=float(limit)), torch.clamp(x @ W("up").T, -float(limit), float(limit))
    return (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ W("down").T


def _gated(x, W):
    return W.linear(_silu(W.linear(x, "gate")) * W.linear(x, "up"), "down")


def _llama(cfg, W, ids, want):
    eps, H, G = cfg["rms_norm_eps"], cfg["num_attention_heads"], cfg["num_key_value_heads"]
    D, see = cfg["hidden_size"] // H, _visible(len(ids))
    f, x = _frequencies(D, cfg["rope_theta"]), W("model.embed_tokens.weight")[ids]
    for i in range(cfg["num_hidden_layers"]):
        L = W.under(f"model.layers.{i}.")
        h = _rms(x, eps, L("input_layernorm.weight"))
        q, k, v = (_heads(h @ L(f"self_attn.{n}_proj.weight").T, g) for n, g in (("q", H), ("k", G), ("v", G)))
        x = x + _attend(_turn(q, f), _turn(k, f), v, D**-0.5, see).flatten(1) @ L("self_attn.o_proj.weight").T
        h = _rms(x, eps, L("post_attention_layernorm.weight"))
        x = x + (_silu(h @ L("mlp.gate_proj.weight").T) * (h @ L("mlp.up_proj.weight").T)) @ L("mlp.down_proj.weight").T
    return _rms(x[want], eps, W("model.norm.weight")) @ W("lm_head.weight").T


def _nurolorn(cfg, W, ids, want):
    eps, groups, factor, T = cfg["norm"]["eps"], cfg["norm"]["groups"], cfg["residual_mult"], len(ids)

    def norm(x, w):
        return _rms(x.view(x.shape[0], groups, -1), eps).flatten(1) * w

    def latent(h, L, m):
        H, D, R = m["heads"], m["dim"], m["kv_rank"]
        q, down = _heads(h @ L("q").T, H), h @ L("dkv").T
        c = _rms(down[:, :R], eps, L("dkv.norm"))
        turned = _rotated(down[:, None, R:], m["rot"], True).expand(T, H, -1)
        q = torch.cat((q[..., :D], _rotated(q[..., D:], m["rot"], True)), -1)
        o = _attend(q, torch.cat((_heads(c @ L("uk").T, H), turned), -1), _heads(c @ L("uv").T, H), m["scale"], _visible(T))
        return (o.flatten(1) * torch.sigmoid(h @ L("g").T)) @ L("o").T

    def mingru(h, L, m):
        z, u = torch.sigmoid(L.linear(h, "z")), L.linear(h, "x")
        c, s, states = torch.where(u >= 0, u + 0.5, torch.sigmoid(u)), 0.0, []
        keep, new = 1 - z, z * c
        for t in range(T):
            s = keep[t] * s + new[t]
            states.append(s)
        return (torch.stack(states) * _silu(h @ L("g").T)) @ L("o").T

    def window(h, L, m):
        q, k, v = (_heads(h @ L(n).T, m[g]) for n, g in (("q", "heads"), ("k", "kv_heads"), ("v", "kv_heads")))
        return _attend(_rms(q, eps), _rms(k, eps), v, m["scale"], _visible(T, m["mask"]["size"]), slopes=_slopes(m["heads"])).flatten(1) @ L("o").T

    mixers = {"latent_attention": latent, "mingru": mingru, "attention": window}
    loop, n = cfg["loop"], len(cfg["layers"])
    order = [(i, None) for i in range(loop["start"])]
    order += [(i, t) for t in range(loop["times"]) for i in range(loop["start"], loop["stop"])]
    order += [(i, None) for i in range(loop["stop"], n)]
    embedded = x = W("embed")[ids]
    for i, t in order:
        if t is not None and i == loop["start"]:
            x = x + (embedded if t > 0 else 0.0) + W("loop.step")[t]
        L, layer = W.under(f"l{i}."), cfg["layers"][i]
        x = x + factor * mixers[layer["type"]](norm(x, L("norm1")), L.under("mix."), layer["mixer"])
        x = x + factor * (torch.relu(norm(x, L("norm2")) @ L("mlp.up").T) ** 2 @ L("mlp.down").T)
    return norm(x[want], W("final.norm")) @ W("head").T * cfg["logit_scale"]


def _kafepel(cfg, W, ids, want):
    eps, T = cfg["norm"]["eps"], len(ids)
    see = _visible(T).to(F64)

    def left(h, L, m):
        H, G = m["heads"], m["kv_heads"]
        q = _rotated(_heads(_rms(h @ L("q").T, eps, L("q.norm")), H), m["rot"])
        k = _rotated(_heads(_rms(h @ L("k").T, eps, L("k.norm")), G), m["rot"]).repeat_interleave(H // G, 1)
        v = _heads(h @ L("v").T, G).repeat_interleave(H // G, 1)
        s = m["softcap"] * torch.tanh(torch.einsum("ihd,jhd->hij", q, k) * m["scale"] / m["softcap"])
        w = torch.sigmoid(s + L("pb")[:, None, None]) * see
        w = (L("talk") @ w.flatten(1)).view_as(w)
        return torch.einsum("hij,jhd->ihd", w, v).flatten(1) @ L("o").T

    def right(h, L, m):
        H, D = m["heads"], m["dim"]
        q, k, v = (_heads(h @ L(n).T, H) for n in ("q", "k", "v"))
        decay = torch.tensor(m["decay"], dtype=F64, device=DEVICE)[None, :, None].expand(T, H, 1)
        o = _recurrence(_rotated(q, m["rot"]), _rotated(k, m["rot"]) * D**-0.5, v, decay)
        return (_rms(o, eps).flatten(1) * _silu(h @ L("g").T)) @ L("o").T

    def unit(h, L):
        return torch.relu(h @ L("up").T) ** 2 @ L("down").T

    def routed(h, L, c):
        s = torch.softmax(h @ L("router").T, -1)
        w = _chosen(s + L("correction"), c["router"]["top"]) * s * c["router"]["scale"]
        return _pick(w, h, lambda x, e: unit(x, L.under(f"e{e}."))) + torch.sigmoid(h @ L("shared.sg").T) * unit(h, L.under("shared."))

    x = W("embed")[ids] * cfg["embedding"]["scale"]
    for i, layer in enumerate(cfg["layers"]):
        L, m, c = W.under(f"l{i}."), layer["mixer"], layer["mlp"]
        h, M = _rms(x, eps, L("norm1")), L.under("mix.")
        x = x + 0.5 * (_rms(left(h, M.under("left."), m["left"]), eps, M("left.out")) + _rms(right(h, M.under("right."), m["right"]), eps, M("right.out")))
        h, M = _rms(x, eps, L("norm2")), L.under("mlp.")
        x = x + (_gated(h, M) if c["kind"] == "dense" else routed(h, M, c))
    return _rms(x[want], eps, W("final.norm")) @ W("head").T


def _nudodra(cfg, W, ids, want):
    eps, T = cfg["norm"]["eps"], len(ids)
    see, held = _visible(T), {}

    def attention(h, L, m, i):
        H, G = m["heads"], m["kv_heads"]
        q = _heads(L.linear(h, "q"), H)
        if m.get("kv_from") is None:
            held[i] = _heads(L.linear(h, "k"), G), _heads(L.linear(h, "v"), G)
        k, v = held[i if m.get("kv_from") is None else m["kv_from"]]
        p = torch.arange(T, dtype=F64, device=DEVICE)
        q = q * (1.0 + m["q_temp"]["coef"] * torch.log(torch.floor((p + 1) / m["q_temp"]["every"]) + 1.0))[:, None, None]
        return (_attend(q, k, v, m["scale"], see).flatten(1) * torch.sigmoid(h @ L("g").T)) @ L("o").T

    def left(h, L, m):
        q, v = _heads(L.linear(h, "q"), m["heads"]), _heads(L.linear(h, "k"), m["kv_heads"])
        q, k = _rotated(_rms(q, eps, L("q.norm")), m["rot"]), _rotated(_rms(v, eps, L("k.norm")), m["rot"])
        return _attend(q, k, v, m["scale"], see, sink=L("sink")).flatten(1) @ L("o").T

    def right(h, L, m):
        H, D = m["heads"], m["dim"]
        q, k, v = (_heads(h @ L(n).T, H) for n in ("q", "k", "v"))
        z = (h @ L("a1").T) @ L("a2").T + L("a2.b")
        o = _recurrence(q * D**-0.5, k, v, _heads(torch.sigmoid(z) ** (1.0 / m["tau"]), H))
        return (_rms(o, eps, L("norm")).flatten(1) * _silu(h @ L("g").T)) @ L("o").T

    def routed(h, L, c):
        w = torch.zeros(T, c["router"]["experts"], dtype=F64, device=DEVICE).scatter(1, L.tensors[L.prefix + "table"][ids].long(), 1.0 / c["router"]["top"])
        return _pick(w, h, lambda x, e: _bounded(x, L.under(f"e{e}."), c["expert"]["limit"])) + _bounded(h, L.under("shared."), c["shared"]["limit"])

    X = W("embed")[ids][None].repeat(cfg["streams"], 1, 1)

    def sublayer(X, L, weight, part):
        y = part(_rms(torch.einsum("s,stw->tw", L("in"), X), eps, weight))
        return torch.einsum("st,snw->tnw", L("mix"), X) + L("out")[:, None, None] * y

    for i, layer in enumerate(cfg["layers"]):
        L, m = W.under(f"l{i}."), layer["mixer"]
        if layer["type"] == "attention":
            X = sublayer(X, L.under("hc1."), L("norm1"), lambda h: attention(h, L.under("mix."), m, i))
        else:
            X = sublayer(X, L.under("hc1."), L("norm1"), lambda h: m["left_scale"] * left(h, L.under("mix.left."), m["left"])
                         + m["right_scale"] * right(h, L.under("mix.right."), m["right"]))
        X = sublayer(X, L.under("hc2."), L("norm2"), lambda h: routed(h, L.under("mlp."), layer["mlp"]))
    return _rms(X.sum(0)[want], eps, W("final.norm")) @ W("head").T


def _tenotar(cfg, W, ids, want):
    eps, T, first = cfg["norm"]["eps"], len(ids), []

    def mixed(v, L):
        if not first:
            first.append(v)
            return v
        lam = L("vmix").reshape(())
        return (1 - lam) * v + lam * first[0]

    def window(h, L, m):
        H, G = m["heads"], m["kv_heads"]
        q, k = _heads(L.linear(h, "q"), H), _heads(L.linear(h, "k"), G)
        q, k = _rotated(_rms(q, eps, L("q.norm")), m["rot"], True), _rotated(_rms(k, eps, L("k.norm")), m["rot"], True)
        v = _heads(mixed(L.linear(h, "v"), L), G)
        return L.linear(_attend(q, k, v, m["scale"], _visible(T, m["mask"]["size"], m["mask"]["keep_first"])).flatten(1), "o")

    def block(h, L, m):
        H, G = m["heads"], m["kv_heads"]
        q, k, v = (_short_conv(h @ L(n).T, L(n + ".conv")) for n in ("q", "k", "v"))
        return _attend(_heads(q, H), _heads(k, G), _heads(mixed(v, L), G), m["scale"], _visible(T, block=m["mask"]["size"]),
                       cap=float(m["softcap"]), slopes=_slopes(H)).flatten(1) @ L("o").T

    def latent(h, L, m):
        H, D, R = m["heads"], m["dim"], m["kv_rank"]
        q = _heads(_rms(h @ L("dq").T, eps, L("dq.norm")) @ L("uq").T, H)
        down = h @ L("dkv").T
        c = _rms(down[:, :R], eps, L("dkv.norm"))
        k = torch.cat((_heads(c @ L("uk").T, H), _rotated(down[:, None, R:], m["rot"]).expand(T, H, -1)), -1)
        q = torch.cat((q[..., :D], _rotated(q[..., D:], m["rot"])), -1)
        o = _attend(q, k, _heads(c @ L("uv").T, H), m["scale"], _visible(T, m["mask"]["size"]))
        return (o * torch.sigmoid(h @ L("g").T)[:, :, None]).flatten(1) @ L("o").T

    def routed(h, L, c):
        z = L.linear(h, "router")
        w = torch.softmax(z.masked_fill(_chosen(z, c["router"]["top"]) == 0, -math.inf), -1)
        return _pick(w, h, lambda x, e: _gated(x, L.under(f"e{e}."))) + _gated(h, L.under("shared."))

    mixers = {"attention": window, "attention_2": block, "latent_attention": latent}
    x = W("embed")[ids]
    for i, layer in enumerate(cfg["layers"]):
        L, c = W.under(f"l{i}."), layer["mlp"]
        x = x + mixers[layer["type"]](_rms(x, eps, L("norm1")), L.under("mix."), layer["mixer"])
        h, M = _rms(x, eps, L("norm2")), L.under("mlp.")
        x = x + (_gated(h, M) if c["kind"] == "dense" else routed(h, M, c))
    return _rms(x[want], eps, W("final.norm")) @ W("head").T * cfg["logit_scale"]


def _pefedra(cfg, W, ids, want):
    eps, T = cfg["norm"]["eps"], len(ids)

    def two_maps(h, L, m):
        H, G = m["heads"], m["kv_heads"]
        q, k = (_rotated(_heads(L.linear(h, n), 2 * g), m["rot"]).view(T, g, 2, -1) for n, g in (("q", H), ("k", G)))
        v, see = _heads(L.linear(h, "v"), G), _visible(T, m["mask"]["size"])
        a, b = (_attend(q[:, :, i], k[:, :, i], v, m["scale"], see) for i in (0, 1))
        share = torch.exp((L("lq1") * L("lk1")).sum()) - torch.exp((L("lq2") * L("lk2")).sum()) + m["diff"]
        return (_rms(a - share * b, eps) * (1.0 - m["diff"])).flatten(1) @ L("o").T

    def turned(h, L, m):
        H, G = m["heads"], m["kv_heads"]
        q, k = (_rotated(_heads(_rms(L.linear(h, n), eps, L(n + ".norm")), g), m["rot"]) for n, g in (("q", H), ("k", G)))
        f = _frequencies(m["vdim"], m["rot"]["base"])
        o = _attend(q, k, _turn(_heads(L.linear(h, "v"), G), f), m["scale"], _visible(T, m["mask"]["size"]))
        return (_turn(o, f, sign=-1.0) * torch.sigmoid(h @ L("g").T)[:, :, None]).flatten(1) @ L("o").T

    mixers = {"attention": two_maps, "attention_2": turned}
    x = W("embed")[ids] * cfg["embedding"]["scale"]
    for i, layer in enumerate(cfg["layers"]):
        L = W.under(f"l{i}.")
        h = _rms(x, eps, L("norm1"))
        h = h + (torch.cat((torch.zeros_like(h[:1]), h[:-1])) - h) * L("shift")
        y = mixers[layer["type"]](h, L.under("mix."), layer["mixer"])
        x = x + y + torch.nn.functional.gelu(_rms(x, eps, L("norm2")) @ L("mlp.up").T) @ L("mlp.down").T
    return _rms(x[want], eps, W("final.norm")) @ W("head").T


def _zifuzen(cfg, W, ids, want):
    eps, T = cfg["norm"]["eps"], len(ids)
    see, kept = _visible(T), {}

    def attention(h, L, m, i):
        if m.get("kv_from") is None:
            kept[i] = _rms(_heads(h @ L("k").T, m["kv_heads"]), eps, L("k.norm")), _heads(h @ L("v").T, m["kv_heads"])
        k, v = kept[i if m.get("kv_from") is None else m["kv_from"]]
        q = _rms(_heads(h @ L("q").T, m["heads"]), eps, L("q.norm"))
        return _attend(q, k, v, m["scale"], see).flatten(1) @ L("o").T

    def delta(h, L, m):
        H, G, D = m["heads"], m["kv_heads"], m["dim"]
        q, k, v = (_silu(_short_conv(h @ L(n).T, L(n + ".conv"))) for n in ("q", "k", "v"))

        def unit(x):
            x = _heads(x, G)
            return (x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 1)

        q, k, v, beta = unit(q) * D**-0.5, unit(k), _heads(v, H), torch.sigmoid(h @ L("b").T)
        decay = torch.exp(-torch.exp(L("A_log")) * torch.nn.functional.softplus(h @ L("a").T + L("dt_bias"), threshold=1e9))
        S, out = v.new_zeros(H, D, v.shape[2]), []
        for t in range(T):
            S = S * decay[t][:, None, None]
            u = beta[t][:, None, None] * (v[t][:, None] - torch.bmm(k[t][:, None], S))
            S = torch.baddbmm(S, k[t][:, :, None], u)
            out.append(torch.bmm(q[t][:, None], S)[:, 0])
        return (_rms(torch.stack(out), eps, L("norm")).flatten(1) * _silu(h @ L("g").T)) @ L("o").T

    def routed(h, L, c):
        r = c["router"]
        s = torch.sigmoid(h @ L("router").T)
        z, count = s + L("correction"), r["groups"]["count"]
        best = _chosen(z.view(T, count, -1).topk(2, dim=-1).values.sum(-1), r["groups"]["keep"])
        z = z.masked_fill(best.repeat_interleave(z.shape[1] // count, 1) == 0, -math.inf)
        w = s * _chosen(z, r["top"])
        w = w / (w.sum(-1, keepdim=True) + 1e-20) * r["scale"]
        return _pick(w, h, lambda x, e: _bounded(x, L.under(f"e{e}."), c["expert"]["limit"])) + _bounded(h, L.under("shared."), c["shared"]["limit"])

    def dense(h, L):
        return L.linear(torch.nn.functional.gelu(L.linear(h, "gate"), approximate="tanh") * L.linear(h, "up"), "down")

    x = W("embed")[ids] * cfg["embedding"]["scale"] + W("pos")[:T]
    for i, layer in enumerate(cfg["layers"]):
        L, c = W.under(f"l{i}."), layer["mlp"]
        M, m = L.under("mix."), layer["mixer"]
        y = attention(x, M, m, i) if layer["type"] == "attention" else delta(x, M, m)
        x = x + _layer_norm(y, eps, L("norm1"))
        M = L.under("mlp.")
        x = x + _layer_norm(dense(x, M) if c["kind"] == "dense" else routed(x, M, c), eps, L("norm2"))
    cap = cfg["logit_softcap"]
    return cap * torch.tanh(_layer_norm(x[want], eps, W("final.norm")) @ W("head").T / cap)


def exact(case, seed):
    """Whole sequences in 64 bits, request by request; the rows in the order that :func:`run` returns them in."""
    cfg = PRESETS[case["model"]]
    design = {"llama": _llama, "nurolorn": _nurolorn, "kafepel": _kafepel, "nudodra": _nudodra, "tenotar": _tenotar, "pefedra": _pefedra, "zifuzen": _zifuzen}
    kind = next(f for n, f in design.items() if n in case["model"])
    W = _Weights(_weights(case, seed))
    vocab = cfg.get("vocab_size") or cfg["vocab"]
    lengths, rows = _prompt_lengths(case), []
    for n, tokens in zip(lengths, _tokens(case, seed, vocab)):
        want = torch.arange(n - 1, n + case["decode"], device=DEVICE)
        rows.append(kind(cfg, W, torch.tensor(tokens, device=DEVICE), want))
    logits = torch.stack([rows[r][a + w - (lengths[r] - 1)] for step in _steps(case) for r, a, _, want in step for w in want])
    return (logits, logits.argmax(-1).to(torch.int32)) if case["dtype"] == "float32" else (logits,)
