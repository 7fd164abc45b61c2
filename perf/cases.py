"""Performance cases: the calls a program makes through this package, over the sizes it is used at.

A case names what is called (``call``), a layer size (``size``), the batch (``requests``: ``history+new`` per request,
a request that brings one token behind a history is a decoded token, one that brings more is a portion of a prompt)
and the engine's data type.  The calls:

    step         ModelRunner.step: a whole Qwen3 decode step, host side included, logits out
    attention    the grouped-query attention mixer (Qwen3) over the paged cache
    mlp          the gated feed-forward (Qwen3)
    moe          the routed feed-forward (router, groups of experts, clamped gated experts)
    latent       the latent attention mixer in its absorbed form
    delta        the gated delta rule mixer, one decay per head
    state_space  the state-space mixer
    sample       logits rows to token ids through the Sampler

Parts are built from the registries as a model builds them, and get the batch as the step function's plan describes it.
``exact`` writes the same results out in 64 bits with plain torch.
"""
from __future__ import annotations

import dataclasses
import math

import torch

from dinfer_b200.cache.manager import CacheManager, GroupSpec
from dinfer_b200.config.engine_config import EngineConfig
from dinfer_b200.engine.batch import PlanBuilder, StepEntry
from dinfer_b200.engine.runner import ModelRunner
from dinfer_b200.kernels import lib as kernel_lib
from dinfer_b200.models import decoder  # noqa: F401  (registers the parts)
from dinfer_b200.parts.base import FEED_FORWARDS, MIXERS, BuildEnv, CacheBinding, split_needs
from dinfer_b200.parts.spec import PartSpec
from dinfer_b200.sampling.params import SamplingParams
from dinfer_b200.sampling.sampler import Sampler
from dinfer_b200.weights.random_init import RandomSource

VOCAB = 151936
PAGE = 16
EPS = 1e-6
F64 = torch.float64
DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}

# layer sizes of the package's benchmark: the Qwen3 0.6B and 8B shapes around a middle one, and the other designs'
# small, medium and large layers
QWEN3 = {"small": dict(width=1024, heads=16, kv_heads=8, dim=128, ff=3072, theta=1e6),
         "medium": dict(width=2048, heads=16, kv_heads=4, dim=128, ff=7680, theta=1e6),
         "large": dict(width=4096, heads=32, kv_heads=8, dim=128, ff=12288, theta=1e6)}
MOE = {"small": dict(width=1024, experts=16, top=4, ff=512, groups=4, keep=2),
       "medium": dict(width=2048, experts=64, top=8, ff=1408, groups=8, keep=4),
       "large": dict(width=4096, experts=64, top=8, ff=2048, groups=8, keep=4)}
LATENT = {"small": dict(width=1024, heads=8, nope=64, rope=32, vdim=64, rank=256, q_rank=512, theta=1e4),
          "medium": dict(width=2048, heads=16, nope=128, rope=64, vdim=128, rank=512, q_rank=1536, theta=1e4),
          "large": dict(width=4096, heads=32, nope=128, rope=64, vdim=128, rank=512, q_rank=1536, theta=1e4)}
DELTA = {"small": dict(width=1024, heads=16, kv_heads=8, dim=64, taps=4),
         "medium": dict(width=2048, heads=16, kv_heads=8, dim=128, taps=4),
         "large": dict(width=4096, heads=32, kv_heads=16, dim=128, taps=4)}
STATE = {"small": dict(width=1024, heads=16, vdim=64, state=64, groups=2, taps=4),
         "medium": dict(width=2048, heads=32, vdim=64, state=128, groups=4, taps=4),
         "large": dict(width=4096, heads=64, vdim=64, state=128, groups=8, taps=4)}
SIZES = {"attention": QWEN3, "mlp": QWEN3, "moe": MOE, "latent": LATENT, "delta": DELTA, "state_space": STATE}
LIMIT, ALPHA = 7.0, 1.702           # the clamped gate's constants


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # one user's chat on a small model: the smallest step there is, launches and hand-overs count
        {"name": "step_small_b1", "call": "step", "size": "small", "layers": 28, "requests": "1000+1", "dtype": "bfloat16"},
        # a few users on a middle-sized model at long contexts (four of its layers, and the head)
        {"name": "step_large_b8", "call": "step", "size": "large", "layers": 4,
         "requests": ",".join("%d+1" % (4090 - 61 * i) for i in range(8)), "dtype": "bfloat16"},
        # a loaded server's decode step: 64 requests at contexts all over the range
        {"name": "attention_decode_b64", "call": "attention", "size": "large",
         "requests": ",".join("%d+1" % (300 + 59 * i) for i in range(64)), "dtype": "bfloat16"},
        # a long prompt taken in whole
        {"name": "attention_prompt", "call": "attention", "size": "large", "requests": "0+2048", "dtype": "bfloat16"},
        # a step's portions of three prompts, one far into its context
        {"name": "mlp_portions", "call": "mlp", "size": "large", "requests": "3584+512,0+250,0+15", "dtype": "bfloat16"},
        # the 32-bit engine on a short prompt
        {"name": "mlp_float32", "call": "mlp", "size": "small", "requests": "0+333", "dtype": "float32"},
        # eight users of a model with routed experts: the experts' weights are what is read
        {"name": "moe_decode_b8", "call": "moe", "size": "large", "requests": ",".join(["500+1"] * 8), "dtype": "bfloat16"},
        # and a long prompt through the same design
        {"name": "moe_prompt", "call": "moe", "size": "medium", "requests": "0+2048", "dtype": "bfloat16"},
        # prompts through the other mixers: attention over a latent, and the two recurrences
        {"name": "latent_prompt", "call": "latent", "size": "medium", "requests": "0+2048", "dtype": "bfloat16"},
        {"name": "delta_prompt", "call": "delta", "size": "medium", "requests": "0+2000", "dtype": "bfloat16"},
        {"name": "state_space_prompt", "call": "state_space", "size": "large", "requests": "0+1500,0+547", "dtype": "bfloat16"},
        # a loaded server's sampling: 64 rows of a large vocabulary, every user with options of their own
        {"name": "sample_b64", "call": "sample", "rows": 64, "options": "mixed"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _requests(rng, tokens, context, together):
    """A decode batch, a whole prompt, a portion behind a history, or several at once."""
    kind = rng.choice(["decode", "prompt", "portion", "several"])
    if kind == "decode":
        return ",".join("%d+1" % _log_int(rng, 16, context) for _ in range(_log_int(rng, 1, together)))
    if kind == "prompt":
        return "0+%d" % _log_int(rng, 7, tokens)
    if kind == "portion":
        return "%d+%d" % (_log_int(rng, 16, context), _log_int(rng, 7, min(tokens, 1024)))
    n = rng.randint(2, 6)
    return ",".join("%d+%d" % (rng.choice([0, _log_int(rng, 16, context)]), _log_int(rng, 1, tokens // n)) for _ in range(n))


def draw(rng):
    call = rng.choice(["step", "attention", "attention", "mlp", "moe", "moe", "latent", "delta", "state_space", "sample"])
    if call == "sample":
        return {"call": call, "rows": _log_int(rng, 1, 64), "options": rng.choice(["greedy", "temperature", "top_k_top_p", "top_p", "mixed"])}
    if call == "step":
        size = rng.choice(["small", "medium", "large"])
        batch = _log_int(rng, 1, 12)
        return {"call": call, "size": size, "layers": rng.randint(2, 6), "dtype": "bfloat16",
                "requests": ",".join("%d+1" % _log_int(rng, 16, 3000) for _ in range(batch))}
    dtype = "float32" if call == "mlp" and rng.random() < 0.3 else "bfloat16"
    size = "small" if dtype == "float32" else rng.choice(["small", "medium", "large"])
    return {"call": call, "size": size, "requests": _requests(rng, 300 if dtype == "float32" else 2000, 4000, 64), "dtype": dtype}


def _batch(case):
    """[(history, new)] of the case."""
    return [tuple(int(v) for v in r.split("+")) for r in case["requests"].split(",")]


# ---------------------------------------------------------------- what a program holds before the call
def _spec(case):
    c, s = case["call"], SIZES[case["call"]][case["size"]]
    if c == "attention":
        return MIXERS, PartSpec("gqa_attention", {
            "num_heads": s["heads"], "num_kv_heads": s["kv_heads"], "head_dim": s["dim"], "qk_norm": True, "eps": EPS,
            "position": PartSpec("rope_neox", {"head_dim": s["dim"], "theta": s["theta"], "max_positions": 40960})})
    if c == "mlp":
        return FEED_FORWARDS, PartSpec("swiglu", {"intermediate_size": s["ff"]})
    if c == "moe":
        return FEED_FORWARDS, PartSpec("moe", {
            "num_experts": s["experts"], "top_k": s["top"], "expert_size": s["ff"], "groups": (s["groups"], s["keep"]),
            "group_rank": 2, "activation": ("clamped_swish", LIMIT, ALPHA), "gated": True, "scoring": "sigmoid",
            "renormalize": True})
    if c == "latent":
        return MIXERS, PartSpec("latent_attention", {
            "num_heads": s["heads"], "nope_dim": s["nope"], "rope_dim": s["rope"], "v_dim": s["vdim"], "kv_rank": s["rank"],
            "q_rank": s["q_rank"], "eps": EPS,
            "position": PartSpec("rope", {"head_dim": s["rope"], "rotary_dim": s["rope"], "theta": s["theta"],
                                          "max_positions": 40960, "style": "interleaved"})})
    if c == "delta":
        return MIXERS, PartSpec("gated_delta", {
            "num_heads": s["heads"], "num_kv_heads": s["kv_heads"], "key_dim": s["dim"], "value_dim": s["dim"],
            "conv": s["taps"], "eps": EPS, "decay": "head", "gate": "silu", "out_float32": True})
    return MIXERS, PartSpec("state_space", {
        "num_heads": s["heads"], "value_dim": s["vdim"], "state_dim": s["state"], "groups": s["groups"], "conv": s["taps"],
        "norm_parts": s["groups"], "eps": EPS})


def _weights(part, gen, dt):
    """Every tensor the part declares: matrices that keep their input's size, norms around one, decays and step sizes
    over the range such mixers are trained to."""
    W = {}
    for d in part.declare():
        r = lambda: torch.rand(d.shape, generator=gen, device="cuda")
        if d.name.endswith("A_log"):
            t = torch.log(1.0 + 15.0 * r())
        elif d.name.endswith("dt_bias"):
            step = torch.exp(math.log(1e-3) + (math.log(1e-1) - math.log(1e-3)) * r())
            t = step + torch.log(-torch.expm1(-step))
        elif d.init == "ones":
            t = 1.0 + 0.2 * (r() - 0.5)
        else:
            t = torch.randn(d.shape, generator=gen, device="cuda") * d.shape[-1] ** -0.5
        W[d.name] = t.to(dt)
    return W


def _context(batch, width_pages, needs):
    """The step's context as the step function builds it: pages of the histories and the new tokens allocated, the plan
    on the device."""
    total = sum((h + n + PAGE - 1) // PAGE for h, n in batch)
    manager = CacheManager([GroupSpec()], PAGE, total, len(batch))
    entries = []
    for i, (h, n) in enumerate(batch):
        if not manager.allocate(i, h + n):
            raise RuntimeError("no pages")
        manager.advance(i, h)
        entries.append(StepEntry(i, [0] * n, []))
    plan = PlanBuilder(manager, "cuda", sum(n for _, n in batch), len(batch), width_pages)
    _, _, ctx = plan.build(entries, [h for h, _ in batch])
    for i, (h, _) in enumerate(batch):
        if h:
            ctx.state_fresh[i] = 0
    return ctx, total, plan


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    if case["call"] == "sample":
        return _prepare_sample(case, seed, gen)
    if case["call"] == "step":
        return _prepare_step(case, seed, gen)
    dt, s = DTYPES[case["dtype"]], SIZES[case["call"]][case["size"]]
    torch.backends.cuda.matmul.allow_tf32 = False           # as the engine sets them
    torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction = False
    batch = _batch(case)
    longest = max(h + n for h, n in batch)
    registry, spec = _spec(case)
    part = registry.get(spec.kind)(spec.params, BuildEnv(torch.device("cuda"), dt, s["width"], longest), "")
    W = _weights(part, gen, dt)
    part.bind(W)
    kernel_lib.preload(part.kernel_libraries())
    T = sum(n for _, n in batch)
    x = torch.randn((T, s["width"]), generator=gen, device="cuda").to(dt)
    state = {"call": case["call"], "part": part, "W": W, "x": x, "batch": batch}
    if registry is FEED_FORWARDS:
        return state
    kv, rec = split_needs(part.cache_need())
    state["ctx"], pages, state["plan"] = _context(batch, (longest + PAGE - 1) // PAGE, part.cache_need())
    binding = CacheBinding()
    if kv is not None:
        binding.kv = torch.randn((pages, kv.planes, kv.num_kv_heads, PAGE, kv.head_dim), generator=gen, device="cuda",
                                 dtype=dt)
        binding.group = 0
    if rec is not None:
        binding.state = torch.randn((len(batch) + 1,) + tuple(rec.shape), generator=gen, device="cuda") * 0.1
    state["cache"] = binding
    return state


def _config(case):
    s = QWEN3[case["size"]]
    return dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", vocab_size=VOCAB, hidden_size=s["width"],
                intermediate_size=s["ff"], num_hidden_layers=case["layers"], num_attention_heads=s["heads"],
                num_key_value_heads=s["kv_heads"], head_dim=s["dim"], rms_norm_eps=EPS, rope_theta=s["theta"],
                max_position_embeddings=40960, tie_word_embeddings=case["size"] == "small", attention_bias=False,
                hidden_act="silu")


def _prepare_step(case, seed, gen):
    cfg, batch = _config(case), _batch(case)
    longest = max(h + 1 for h, _ in batch)
    source = RandomSource(cfg, seed, std=0.02, norm_jitter=0.1)
    runner = ModelRunner(cfg, source, EngineConfig(
        max_model_len=longest + PAGE, max_num_seqs=len(batch), max_num_batched_tokens=max(2048, longest), block_size=PAGE,
        num_blocks=sum(h // PAGE + 2 for h, _ in batch), dtype=case["dtype"], mixed_cuda_graph=False))
    prompts = [torch.randint(VOCAB, (h,), generator=gen, device="cuda").tolist() for h, _ in batch]
    for i, p in enumerate(prompts):
        runner.step([StepEntry(i, p, [])])
    last = torch.randint(VOCAB, (len(batch),), generator=gen, device="cuda").tolist()
    return {"call": "step", "runner": runner, "source": source, "cfg": cfg, "batch": batch, "prompts": prompts, "last": last,
            "entries": [StepEntry(i, [t], [0]) for i, t in enumerate(last)]}


def _prepare_sample(case, seed, gen):
    R = case["rows"]
    # a few dozen likely tokens above a wide floor, as a trained model's logits have
    logits = torch.randn((R, VOCAB), generator=gen, device="cuda") * 1.5
    likely = torch.rand((R, VOCAB), generator=gen, device="cuda").topk(40, dim=1).indices
    logits.scatter_add_(1, likely, (14.0 - 0.25 * torch.arange(40, device="cuda")).expand(R, 40))
    kinds = {"greedy": SamplingParams(temperature=0.0), "temperature": SamplingParams(temperature=0.7),
             "top_k_top_p": SamplingParams(temperature=0.6, top_k=20, top_p=0.95),
             "top_p": SamplingParams(temperature=0.8, top_p=0.9)}
    cycle = list(kinds) if case["options"] == "mixed" else [case["options"]]
    return {"call": "sample", "sampler": Sampler("cuda"), "logits": logits,
            "params": [kinds[cycle[i % len(cycle)]] for i in range(R)], "seeds": [seed * 1000 + i for i in range(R)],
            "generated": [3 * i + 1 for i in range(R)]}


# ---------------------------------------------------------------- one pass
def run(state):
    call = state["call"]
    if call == "sample":
        return state["sampler"](state["logits"], state["params"], state["seeds"], state["generated"])
    if call == "step":
        runner = state["runner"]
        logits = runner.step(state["entries"])
        for i, (h, _) in enumerate(state["batch"]):          # the token is taken back: the next pass decodes the same place
            runner.manager.advance(i, h)
        return logits
    if call in ("mlp", "moe"):
        return state["part"].forward(state["x"])
    # a step's context is made for one step: what parts derive from it is not kept for the next
    y = state["part"].forward(state["x"], dataclasses.replace(state["ctx"], derived={}), state["cache"])
    cache = state["cache"]
    return {"y": y, "cache": cache.kv} if cache.kv is not None else {"y": y, "state": cache.state}


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    if case["call"] == "sample":
        n = case["rows"] * VOCAB
        return {"bytes": 4 * n, "flops": 2 * n}
    batch = _batch(case)
    T = sum(n for _, n in batch)
    elt = 4 if case["dtype"] == "float32" else 2
    pairs = sum(n * h + n * (n + 1) // 2 for h, n in batch)
    held = sum(h + n for h, n in batch)
    c = case["call"]
    if c == "step":
        s, L = QWEN3[case["size"]], case["layers"]
        row = (s["heads"] + 2 * s["kv_heads"]) * s["dim"]
        weights = L * (s["width"] * row + s["width"] * s["heads"] * s["dim"] + 3 * s["width"] * s["ff"]) + VOCAB * s["width"]
        return {"bytes": elt * (weights + L * held * 2 * s["kv_heads"] * s["dim"]) + 4 * T * VOCAB,
                "flops": 2 * T * weights + L * 4 * pairs * s["heads"] * s["dim"]}
    s = SIZES[c][case["size"]]
    w = s["width"]
    ends = 2 * elt * T * w                                   # the rows in and out
    if c == "attention":
        weights = w * (2 * s["heads"] + 2 * s["kv_heads"]) * s["dim"]
        return {"bytes": elt * (weights + held * 2 * s["kv_heads"] * s["dim"]) + ends,
                "flops": 2 * T * weights + 4 * pairs * s["heads"] * s["dim"]}
    if c == "mlp":
        weights = 3 * w * s["ff"]
        return {"bytes": elt * weights + ends, "flops": 2 * T * weights}
    if c == "moe":
        one = 3 * w * s["ff"]
        # experts that T tokens meet, if every choice is as likely
        met = s["experts"] * (1 - (1 - s["top"] / s["experts"]) ** T)
        return {"bytes": int(elt * (met * one + w * s["experts"]) + ends), "flops": 2 * T * (s["top"] * one + w * s["experts"])}
    if c == "latent":
        H = s["heads"]
        weights = (w * (s["q_rank"] + s["rank"] + s["rope"]) + s["q_rank"] * H * (s["nope"] + s["rope"])
                   + H * s["rank"] * (s["nope"] + s["vdim"]) + H * s["vdim"] * w)
        return {"bytes": elt * (weights + held * (s["rank"] + s["rope"])) + ends,
                "flops": 2 * T * weights + 2 * pairs * H * (s["nope"] + s["rope"] + s["vdim"])}
    if c == "delta":
        H, G, D = s["heads"], s["kv_heads"], s["dim"]
        weights = w * (2 * G * D + 2 * H * D + 2 * H) + H * D * w
        return {"bytes": elt * weights + ends + 4 * len(batch) * H * D * D, "flops": 2 * T * weights + 6 * T * H * D * D}
    inner = s["heads"] * s["vdim"]
    weights = w * (2 * inner + 2 * s["groups"] * s["state"] + s["heads"]) + inner * w
    return {"bytes": elt * weights + ends + 4 * len(batch) * inner * s["state"],
            "flops": 2 * T * weights + 4 * T * inner * s["state"]}


def tolerance(case):
    if case["call"] == "sample":
        return "exact"
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-4}
    return {"rel": TOLERANCE[case["call"]], "max": 0.5}


# bfloat16 layers are 2e-3 to 5e-3 off the same results in 64 bits (rounded products and activations), two correct ones up
# to 1.4 times that apart; whole models carry every layer's rounding on (7e-3 to 1.3e-2)
TOLERANCE = {"step": 0.03, "attention": 0.01, "mlp": 0.01, "moe": 0.01, "latent": 0.02, "delta": 0.01, "state_space": 0.01}


# ---------------------------------------------------------------- the same results in 64 bits
def _rms(x, w):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS) * w.double()


def _lin(x, w):
    return x @ w.double().T


def _silu(z):
    return z * torch.sigmoid(z)


def _softplus(z):
    return torch.clamp(z, min=0.0) + torch.log1p(torch.exp(-z.abs()))


def _turn(x, pos, theta, pairs):
    """x [T, heads, n]: every pair turned by position times theta^(-2i/n); pairs (2i, 2i + 1), or (i, i + n/2)."""
    n = x.shape[-1]
    f = theta ** (-2.0 * torch.arange(n // 2, dtype=F64, device=x.device) / n)
    a = pos.double()[:, None] * f[None, :]
    c, s = a.cos()[:, None, :], a.sin()[:, None, :]
    u, v = (x[..., 0::2], x[..., 1::2]) if pairs else (x[..., :n // 2], x[..., n // 2:])
    a, b = u * c - v * s, v * c + u * s
    return torch.stack([a, b], -1).flatten(-2) if pairs else torch.cat([a, b], -1)


def _attend(q, k, v, hist, scale):
    """q [n, H, D] behind ``hist`` tokens, k [hist + n, G, D], v [hist + n, G, Dv] -> [n, H, Dv]."""
    n, H, G = q.shape[0], q.shape[1], k.shape[1]
    out = []
    hidden = torch.arange(k.shape[0], device=q.device)[None, :] > hist + torch.arange(n, device=q.device)[:, None]
    for h in range(H):
        s = (q[:, h] @ k[:, h * G // H].T * scale).masked_fill(hidden, -math.inf)
        out.append(torch.softmax(s, -1) @ v[:, h * G // H])
    return torch.stack(out, 1)


def _gqa(x, W, s, pos, hist, k_old, v_old, names=("q_proj.weight", "k_proj.weight", "v_proj.weight", "o_proj.weight",
                                                  "q_norm.weight", "k_norm.weight")):
    """One request's rows through the attention layer: (result, its keys, its values)."""
    n, H, G, D = x.shape[0], s["heads"], s["kv_heads"], s["dim"]
    wq, wk, wv, wo, qn, kn = (W[m] for m in names)
    q = _turn(_rms(_lin(x, wq).reshape(n, H, D), qn), pos, s["theta"], False)
    k = _turn(_rms(_lin(x, wk).reshape(n, G, D), kn), pos, s["theta"], False)
    v = _lin(x, wv).reshape(n, G, D)
    k, v = torch.cat([k_old, k]), torch.cat([v_old, v])
    return _lin(_attend(q, k, v, hist, D ** -0.5).reshape(n, H * D), wo), k, v


def _mlp(x, g, u, d):
    return _lin(_silu(_lin(x, g)) * _lin(x, u), d)


def _old_rows(state, i, hist):
    """Rows of request i's history in the cache: [hist, planes, heads, dim]."""
    pages = state["ctx"].groups[0].block_table[i].long()[:(hist + PAGE - 1) // PAGE]
    rows = state["cache"].kv[pages].double()                 # [pages, planes, heads, PAGE, dim]
    return rows.permute(0, 3, 1, 2, 4).flatten(0, 1)[:hist]


def exact(case, seed):
    if case["call"] == "sample":
        return None
    state = prepare(case, seed)
    if case["call"] == "step":
        return _exact_step(state, case)
    W, x, c = state["W"], state["x"].double(), case["call"]
    s = SIZES[c][case["size"]]
    if c == "mlp":
        return _mlp(x, W["gate_proj.weight"], W["up_proj.weight"], W["down_proj.weight"])
    if c == "moe":
        return _exact_moe(x, W, s)
    ys, at = [], 0
    carried = state["cache"].state.double() if state["cache"].state is not None else None
    for i, (h, n) in enumerate(state["batch"]):
        rows = x[at:at + n]
        at += n
        pos = torch.arange(h, h + n, device=x.device)
        if c == "attention":
            old = _old_rows(state, i, h)
            ys.append(_gqa(rows, W, s, pos, h, old[:, 0], old[:, 1])[0])
        elif c == "latent":
            ys.append(_exact_latent(rows, W, s, pos, h, _old_rows(state, i, h)[:, 0, 0]))
        else:
            slot = int(state["ctx"].state_slots[i])
            if not h:
                carried[slot] = 0.0
            ys.append((_exact_delta if c == "delta" else _exact_state_space)(rows, W, s, carried[slot]))
    y = torch.cat(ys)
    return {"y": y, "cache": None} if carried is None else {"y": y, "state": carried}


def _exact_step(state, case):
    s, src = QWEN3[case["size"]], state["source"]
    get = lambda name: src.get(name)
    table = get("model.embed_tokens.weight")
    out = []
    xs = [table[torch.tensor(p + [t], device="cuda")].double() for p, t in zip(state["prompts"], state["last"])]
    none = torch.zeros((0, s["kv_heads"], s["dim"]), dtype=F64, device="cuda")
    for l in range(case["layers"]):
        at = "model.layers.%d." % l
        W = {n: get(at + n) for n in ("input_layernorm.weight", "post_attention_layernorm.weight", "self_attn.q_proj.weight",
                                      "self_attn.k_proj.weight", "self_attn.v_proj.weight", "self_attn.o_proj.weight",
                                      "self_attn.q_norm.weight", "self_attn.k_norm.weight", "mlp.gate_proj.weight",
                                      "mlp.up_proj.weight", "mlp.down_proj.weight")}
        names = tuple("self_attn." + n for n in ("q_proj.weight", "k_proj.weight", "v_proj.weight", "o_proj.weight",
                                                 "q_norm.weight", "k_norm.weight"))
        for i, x in enumerate(xs):
            pos = torch.arange(x.shape[0], device="cuda")
            x = x + _gqa(_rms(x, W["input_layernorm.weight"]), W, s, pos, 0, none, none, names)[0]
            xs[i] = x + _mlp(_rms(x, W["post_attention_layernorm.weight"]), W["mlp.gate_proj.weight"], W["mlp.up_proj.weight"],
                             W["mlp.down_proj.weight"])
    head = table if state["cfg"]["tie_word_embeddings"] else get("lm_head.weight")
    norm = get("model.norm.weight")
    for x in xs:
        out.append(_lin(_rms(x[-1:], norm), head))
    return torch.cat(out)


def _exact_moe(x, W, s):
    score = torch.sigmoid(_lin(x, W["router.weight"]))
    T, E, size = x.shape[0], s["experts"], s["experts"] // s["groups"]
    best = score.reshape(T, s["groups"], size).topk(2, dim=-1).values.sum(-1)
    kept = torch.zeros_like(best, dtype=torch.bool).scatter_(1, best.topk(s["keep"], dim=1).indices, True)
    w, ids = score.masked_fill(~kept.repeat_interleave(size, 1), -1.0).topk(s["top"], dim=1)
    w = w / (w.sum(1, keepdim=True) + 1e-20)
    out = torch.zeros_like(x)
    for e in range(E):
        t, k = (ids == e).nonzero(as_tuple=True)
        if t.numel():
            at = "experts.%d." % e
            g = torch.clamp(_lin(x[t], W[at + "gate.weight"]), max=LIMIT)
            u = torch.clamp(_lin(x[t], W[at + "up.weight"]), min=-LIMIT, max=LIMIT)
            out[t] += w[t, k, None] * _lin(g * torch.sigmoid(ALPHA * g) * (u + 1.0), W[at + "down.weight"])
    return out


def _exact_latent(x, W, s, pos, hist, old):
    n, H, D, P, V, R = x.shape[0], s["heads"], s["nope"], s["rope"], s["vdim"], s["rank"]
    q = _lin(_rms(_lin(x, W["q_down.weight"]), W["q_norm.weight"]), W["q_up.weight"]).reshape(n, H, D + P)
    down = _lin(x, W["kv_down.weight"])
    c = torch.cat([old[:, :R], _rms(down[:, :R], W["kv_norm.weight"])])
    kr = torch.cat([old[:, R:], _turn(down[:, None, R:], pos, s["theta"], True)[:, 0]])
    k = _lin(c, W["k_up.weight"]).reshape(-1, H, D)
    k = torch.cat([k, kr[:, None].expand(-1, H, -1)], -1)
    v = _lin(c, W["v_up.weight"]).reshape(-1, H, V)
    q = torch.cat([q[..., :D], _turn(q[..., D:], pos, s["theta"], True)], -1)
    return _lin(_attend(q, k, v, hist, (D + P) ** -0.5).reshape(n, H * V), W["o_proj.weight"])


def _conv(x, w, bias, old):
    """Causal convolution per channel and silu; ``old`` [taps - 1, C] holds the inputs before and takes the last ones."""
    full, n = torch.cat([old, x]), x.shape[0]
    y = sum(full[j:j + n] * w[:, j].double() for j in range(w.shape[1]))
    old.copy_(full[n:])
    return _silu(y if bias is None else y + bias.double())


def _exact_delta(x, W, s, row):
    n, H, G, D = x.shape[0], s["heads"], s["kv_heads"], s["dim"]
    S = row[:H * D * D].view(H, D, D)
    old = row[H * D * D:].view(s["taps"] - 1, -1)
    xs = torch.cat([_lin(x, W[m]) for m in "qkv"], 1)
    xs = _conv(xs, torch.cat([W[m + ".conv"] for m in "qkv"]), None, old)
    q, k, v = torch.split(xs, [G * D, G * D, H * D], 1)
    unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)
    q = unit(q.reshape(n, G, D)).repeat_interleave(H // G, 1) * D ** -0.5
    k = unit(k.reshape(n, G, D)).repeat_interleave(H // G, 1)
    v = v.reshape(n, H, D)
    beta = torch.sigmoid(_lin(x, W["b"]))
    g = torch.exp(-torch.exp(W["A_log"].double()) * _softplus(_lin(x, W["a"]) + W["dt_bias"].double()))
    o = torch.empty_like(v)
    for t in range(n):
        S.mul_(g[t, :, None, None])
        u = beta[t, :, None] * (v[t] - torch.bmm(k[t, :, None], S)[:, 0])
        S.baddbmm_(k[t, :, :, None], u[:, None])
        o[t] = torch.bmm(q[t, :, None], S)[:, 0]
    o = _rms(o, W["norm"]).reshape(n, H * D) * _silu(_lin(x, W["g"]))
    return _lin(o, W["o"])


def _exact_state_space(x, W, s, row):
    n, H, P, N, G = x.shape[0], s["heads"], s["vdim"], s["state"], s["groups"]
    inner = H * P
    channels = inner + 2 * G * N
    S = row[:H * N * P].view(H, N, P)
    old = row[H * N * P:H * N * P + (s["taps"] - 1) * channels].view(s["taps"] - 1, channels)
    z, xbc, dt = torch.split(_lin(x, W["in"]), [inner, channels, H], 1)
    xs, B, C = torch.split(_conv(xbc, W["conv"], W["conv.b"], old), [inner, G * N, G * N], 1)
    xs = xs.reshape(n, H, P)
    B, C = (t.reshape(n, G, N).repeat_interleave(H // G, 1) for t in (B, C))
    dt = _softplus(dt + W["dt_bias"].double())
    g = torch.exp(-torch.exp(W["A_log"].double()) * dt)
    y = torch.empty_like(xs)
    for t in range(n):
        S.mul_(g[t, :, None, None])
        S.baddbmm_((dt[t, :, None] * B[t])[:, :, None], xs[t, :, None])
        y[t] = torch.bmm(C[t, :, None], S)[:, 0]
    y = (y + W["D"].double()[:, None] * xs).reshape(n, inner) * _silu(z)
    parts = s["groups"]
    p = y.reshape(n, parts, inner // parts)
    y = (p / torch.sqrt((p * p).mean(-1, keepdim=True) + EPS)).reshape(n, inner) * W["norm"].double()
    return _lin(y, W["o"])
