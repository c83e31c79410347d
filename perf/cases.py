"""What users of this package have it do, as cases that can be timed and checked.

Most cases are one layer part of a decoder (an attention, a recurrent mixer, a feed-forward, the
head with the sampler), built from its spec as the model builder does and called as a block calls
it; two kinds of whole calls go through the step function, from prompts to decoded tokens.  Sizes
are those of the decoders this repository measures (Orpheus 3B and the Llama 3.2 1B shape; the
"small" and "medium" shapes of the further architectures), tokens run from one decoded token to
prompts of 2,048.
"""
import math

import torch

from mstar_b200.config import layout as L
from mstar_b200.config.registry import config_from_dict
from mstar_b200.engine.model import load_model
from mstar_b200.engine.step import StepEntry, make_stepper
from mstar_b200.parts.base import LayerCache, Runtime, StepContext
from mstar_b200.parts.registry import build_part, part_class
from mstar_b200.sampling.params import SamplingParams
from mstar_b200.sampling.sampler import Sampler
from mstar_b200.weights.random_init import random_checkpoint

DEVICE = "cuda:0"
PAGE = 16
DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}
LLAMA3 = {"rope_type": "llama3", "factor": 32.0, "low_freq_factor": 1.0, "high_freq_factor": 4.0,
          "original_max_position_embeddings": 8192}


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # one user's short request, start to end: a prompt of 37 tokens, then token by token;
        # every launch counts (Llama 3.2 1B layers, four of them)
        dict(name="serve_one", kind="serve", arch="llama", width=2048, heads=32, kv_heads=8, dim=64,
             ff=8192, vocab=128256, depth=4, requests=1, prompt=37, new=8),
        # a small batch of ragged prompts in one step, then decoded together: the serving loop at
        # the sizes of Orpheus 3B (four layers of it, its whole vocabulary)
        dict(name="serve_batch", kind="serve", arch="llama", width=3072, heads=24, kv_heads=8,
             dim=128, ff=8192, vocab=156940, depth=4, requests=8, prompt=509, new=8),
        # decoding for many users at once: 64 requests of up to 2,048 cached tokens each
        dict(name="attention_decode", kind="attention", width=3072, heads=24, kv_heads=8, dim=128,
             requests=64, cached=2047, new=1, dtype="bfloat16"),
        # a prompt portion on top of what an earlier one cached (odd sizes on purpose)
        dict(name="attention_prefill", kind="attention", width=3072, heads=24, kv_heads=8, dim=128,
             requests=1, cached=1001, new=2011, dtype="bfloat16"),
        # the 32-bit mode, in which runs are compared between implementations
        dict(name="attention_float32", kind="attention", width=2048, heads=32, kv_heads=8, dim=64,
             requests=2, cached=0, new=256, dtype="float32"),
        # the dense gated feed-forward on a prompt
        dict(name="mlp_prefill", kind="mlp", width=3072, ff=8192, rows=2048, dtype="bfloat16"),
        # a prompt through the soft-capped attention with sink, temperature and feature gate
        dict(name="softcap_attention_prefill", kind="optioned", style="sink", width=2048, heads=16,
             kv_heads=4, requests=1, cached=0, new=2048),
        # a prompt through the latent attention with normed query latents
        dict(name="latent_attention_prefill", kind="latent", style="q_latent", width=2048, heads=16,
             dim=128, rot=64, rank=512, q_rank=1024, requests=1, cached=0, new=2048),
        # a prompt through routed experts beside a shared one
        dict(name="experts_prefill", kind="experts", style="grouped", width=2048, experts=32, top=4,
             ff=512, shared=2048, rows=2048),
        # a prompt through the gated delta rule with a decay a key channel
        dict(name="delta_prefill", kind="delta", style="channel", width=2048, heads=16, kv_heads=16,
             rank=128, requests=1, cached=0, new=2048),
        # prompts of several users through the selective scan
        dict(name="scan_prefill", kind="scan", width=2048, inner=4096, state=16, rank=128,
             requests=2, cached=0, new=1024),
        # the end of a decode step for 64 users: logits over the whole vocabulary, a token each
        dict(name="head_and_sample", kind="head", width=3072, vocab=156940, rows=64,
             temperature=0.6, top_p=0.8, penalty=1.1),
    ]


def _between(rng, lo, hi):
    """A whole number, its logarithm spread evenly; odd ones as often as even ones."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))
    return max(lo, min(hi, n))


def _tokens(rng, most):
    """(requests, cached, new): one request's prompt portion, several at once, or decoding."""
    shape = rng.choice(("prompt", "prompts", "decode"))
    if shape == "prompt":
        return 1, rng.choice((0, _between(rng, 1, most))), _between(rng, 2, most)
    if shape == "prompts":
        n = rng.randint(2, 5)
        return n, rng.choice((0, _between(rng, 1, most // 2))), _between(rng, 2, most // n)
    return _between(rng, 1, 64), _between(rng, 1, most), 1


def draw(rng):
    kind = rng.choice(("serve", "attention", "attention", "mlp", "optioned", "latent", "experts",
                       "delta", "scan", "head"))
    shape = rng.choice(((1024, 8, 2), (2048, 16, 4)))
    width = shape[0]
    if kind == "serve":
        width, heads, dim, ff, vocab = rng.choice(((2048, 32, 64, 8192, 128256),
                                                   (3072, 24, 128, 8192, 156940)))
        return dict(kind=kind, arch="llama", width=width, heads=heads, kv_heads=8, dim=dim, ff=ff,
                    vocab=vocab, depth=rng.randint(2, 3), requests=rng.randint(1, 8),
                    prompt=_between(rng, 2, 300), new=rng.randint(2, 7))
    if kind == "attention":
        width, heads, dim = rng.choice(((2048, 32, 64), (3072, 24, 128)))
        small = rng.random() < 0.3
        requests, cached, new = _tokens(rng, 250 if small else 2000)
        return dict(kind=kind, width=width, heads=heads, kv_heads=8, dim=dim, requests=requests,
                    cached=cached, new=new, dtype="float32" if small else "bfloat16")
    if kind == "mlp":
        small = rng.random() < 0.3
        return dict(kind=kind, width=rng.choice((2048, 3072)), ff=rng.choice((5632, 8192)),
                    rows=_between(rng, 1, 256 if small else 2048),
                    dtype="float32" if small else "bfloat16")
    if kind == "optioned":
        requests, cached, new = _tokens(rng, 2000)
        return dict(kind=kind, style=rng.choice(("sink", "window", "keep_first", "chunk")),
                    width=width, heads=shape[1], kv_heads=shape[2], requests=requests, cached=cached,
                    new=new)
    if kind == "latent":
        requests, cached, new = _tokens(rng, 2000)
        big = width == 2048
        return dict(kind=kind, style=rng.choice(("q_latent", "window")), width=width, heads=shape[1],
                    dim=128 if big else 64, rot=64 if big else 32, rank=512 if big else 256,
                    q_rank=1024 if big else 384, requests=requests, cached=cached, new=new)
    if kind == "experts":
        big = width == 2048
        return dict(kind=kind, style=rng.choice(("grouped", "scaled_input", "clamped")), width=width,
                    experts=32 if big else 16, top=4 if big else 2, ff=512,
                    shared=2048 if big else 1024, rows=_between(rng, 1, 2048))
    if kind == "delta":
        requests, cached, new = _tokens(rng, 2000)
        style = rng.choice(("channel", "head"))
        return dict(kind=kind, style=style, width=width, heads=shape[1],
                    kv_heads=shape[1] if style == "channel" else shape[1] // 2, rank=width // 16,
                    requests=requests, cached=cached, new=new)
    if kind == "scan":
        requests, cached, new = _tokens(rng, 2000)
        return dict(kind=kind, width=width, inner=2 * width, state=16, rank=width // 16,
                    requests=requests, cached=cached, new=new)
    return dict(kind="head", width=3072, vocab=rng.choice((128256, 156940)),
                rows=_between(rng, 1, 64), temperature=rng.choice((0.0, 0.6, 0.8)),
                top_p=rng.choice((0.8, 0.95)), penalty=rng.choice((1.0, 1.1)))


# ------------------------------------------------------------------ batches
def _lengths(case):
    """(tokens already cached, new tokens) of each request: ragged, the first the longest."""
    n, cached, new = case["requests"], case["cached"], case["new"]
    return [(cached - i * cached // (2 * n), new - i * new // (2 * n) if new > 1 else 1)
            for i in range(n)]


def _context(lengths, gen):
    """The step context of these requests and their shared block table."""
    n = len(lengths)
    q_lens = [new for _, new in lengths]
    kv_lens = [cached + new for cached, new in lengths]
    singles = sum(1 for q in q_lens if q == 1)
    width = max(-(-k // PAGE) for k in kv_lens)

    def i32(values):
        return torch.tensor(values, dtype=torch.int32, device=DEVICE)

    pages = torch.randperm(n * width, generator=gen, device=DEVICE).to(torch.int32)
    starts = [0]
    for q in q_lens:
        starts.append(starts[-1] + q)
    positions = i32([c + k for c, q in lengths for k in range(q)])
    ctx = StepContext(
        num_tokens=starts[-1], num_entries=n,
        token_req=i32([r for r, q in enumerate(q_lens) for _ in range(q)]), positions=positions,
        cache_pos=positions, qo_indptr=i32(starts), kv_len=i32(kv_lens), slots=i32(list(range(n))),
        q_lens=q_lens, kv_lens=kv_lens, host_slots=list(range(n)), max_q_len=max(q_lens),
        max_kv_len=max(kv_lens), num_decode=singles if singles == n else 0)
    return ctx, pages.view(n, width)


# ------------------------------------------------------------------ specs
def _rope(dim, rotary, theta=500000.0, scaling=None):
    return L.PositionSpec(kind="rope", head_dim=dim, rotary_dim=rotary, theta=theta, scaling=scaling)


def _spec(case):
    kind, width = case["kind"], case["width"]
    if kind == "attention":
        return "mixer", L.AttentionSpec(
            hidden_size=width, num_heads=case["heads"], num_kv_heads=case["kv_heads"],
            head_dim=case["dim"],
            position=_rope(case["dim"], case["dim"], scaling=L.RopeScalingSpec(**LLAMA3)))
    if kind == "mlp":
        return "ffn", L.GatedMLPSpec(hidden_size=width, intermediate_size=case["ff"])
    if kind == "optioned":
        base = dict(hidden_size=width, num_heads=case["heads"], num_kv_heads=case["kv_heads"],
                    head_dim=128, v_head_dim=128, scale=128 ** -0.5)
        style = case["style"]
        if style == "sink":         # Mokotar's
            return "mixer", L.AttentionSpec(**base, position=L.PositionSpec(kind="none", head_dim=128),
                                            qk_norm_eps=1e-6, feature_gate=True, q_temp=(0.3, 512),
                                            softcap=30.0, sink="learned")
        if style == "window":       # Famarax's
            return "mixer", L.AttentionSpec(**base, position=_rope(128, 128), window=1024,
                                            qk_norm_eps=1e-6, qk_norm_weight=False, softcap=30.0)
        if style == "keep_first":   # Vudivik's
            return "mixer", L.AttentionSpec(**base, position=_rope(128, 128), window=1024,
                                            keep_first=4, bias=True, qk_norm_eps=1e-6)
        return "mixer", L.AttentionSpec(**base, position=_rope(128, 64), feature_gate=True,
                                        softcap=30.0, chunk=1024, weights="sigmoid",
                                        score_bias=True)        # Sokalorn's
    if kind == "latent":
        base = dict(hidden_size=width, num_heads=case["heads"], qk_dim=case["dim"],
                    rot_dim=case["rot"], v_dim=case["dim"], kv_rank=case["rank"],
                    scale=(case["dim"] + case["rot"]) ** -0.5,
                    position=_rope(case["rot"], case["rot"]))
        if case["style"] == "q_latent":     # Relurax's
            return "mixer", L.LatentAttentionSpec(**base, gate_per_head=True, q_rank=case["q_rank"])
        return "mixer", L.LatentAttentionSpec(**base, window=1024)      # Tifosun's
    if kind == "experts":
        base = dict(hidden_size=width, num_experts=case["experts"], top=case["top"],
                    expert_size=case["ff"], shared_size=case["shared"])
        if case["style"] == "grouped":      # Famarax's
            return "ffn", L.RoutedExpertsSpec(**base, score="softmax", renormalize=True,
                                              renorm_eps=1e-20, weight_scale=2.0, scale_input=False,
                                              choice_bias=True, groups=(case["experts"] // 4,
                                                                        case["experts"] // 8))
        if case["style"] == "scaled_input":     # Tifosun's
            return "ffn", L.RoutedExpertsSpec(**base)
        return "ffn", L.RoutedExpertsSpec(**base, score="softmax", renormalize=True,
                                          scale_input=False, activation="clamped_swish", limit=7.0,
                                          shared_limit=7.0, shared_gate=True)   # Sokalorn's
    if kind == "delta":
        head = case["style"] == "head"
        return "mixer", L.GatedDeltaSpec(
            hidden_size=width, num_heads=case["heads"], num_kv_heads=case["kv_heads"], qk_dim=128,
            v_dim=128, conv=4, decay_rank=0 if head else case["rank"],
            gate_rank=0 if head else case["rank"], head_decay=head, full_gate=head,
            gate_activation="silu" if head else "sigmoid")
    if kind == "scan":
        return "mixer", L.SelectiveScanSpec(hidden_size=width, inner=case["inner"],
                                            state=case["state"], dt_rank=case["rank"], conv=4)
    return "head", L.HeadSpec(vocab_size=case["vocab"], hidden_size=width)


def _parameters(case, category, spec, gen, dtype):
    """Random parameters with the spread that trained ones have."""
    def normal(shape, std):
        return std * torch.randn(shape, generator=gen, device=DEVICE)

    def uniform(shape, lo, hi):
        return lo + (hi - lo) * torch.rand(shape, generator=gen, device=DEVICE)

    out = {}
    for name, ps in part_class(category, spec).param_specs(spec).items():
        if name.endswith("norm.weight"):
            t = 1 + normal(ps.shape, 0.1)
        elif name == "A_log":
            t = torch.log(uniform(ps.shape, 1.0, 16.0))
        elif name in ("dt_bias", "dt.bias"):        # step sizes from 0.001 to 0.1
            t = torch.exp(uniform(ps.shape, math.log(0.001), math.log(0.1)))
            t = t + torch.log(-torch.expm1(-t))
        elif name in ("conv.weight", "conv.bias"):
            t = normal(ps.shape, 0.3)
        elif name == "D":
            t = torch.ones(ps.shape, device=DEVICE)
        elif name in ("sink", "score_bias"):
            t = normal(ps.shape, 1.0)
        elif name in ("qkv.bias", "router.correction"):
            t = normal(ps.shape, 0.02)
        elif name == "router.weight":
            t = normal(ps.shape, 0.04)
        elif category == "head":
            t = normal(ps.shape, 0.05)
        else:
            t = normal(ps.shape, 0.02)
        out[name] = t.to(torch.bfloat16).to(dtype)
    return out


def _inputs(case, seed):
    """Everything a pass reads, as plain tensors."""
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(seed)
    dtype = DTYPES[case.get("dtype", "bfloat16")]
    category, spec = _spec(case)
    s = {"category": category, "spec": spec, "dtype": dtype,
         "params": _parameters(case, category, spec, gen, dtype), "ctx": None, "table": None}
    rows = case.get("rows")
    if rows is None:
        s["lengths"] = _lengths(case)
        s["ctx"], s["table"] = _context(s["lengths"], gen)
        rows = s["ctx"].num_tokens
    s["x"] = torch.randn(rows, case["width"], generator=gen, device=DEVICE).to(dtype)
    s["kv"] = s["state"] = None
    if category == "mixer":
        need = part_class(category, spec).cache_need(spec)
        if need.kv is not None:
            k = need.kv
            pages = s["table"].numel() + 1
            s["kv"] = torch.randn(pages, k.planes, k.num_kv_heads, PAGE, k.head_dim, generator=gen,
                                  device=DEVICE, dtype=dtype)
        if need.state is not None:
            shape = (len(s["lengths"]) + 1,) + tuple(need.state.shape)
            scale = 0.1 if case["cached"] else 0.0
            s["state"] = scale * torch.randn(shape, generator=gen, device=DEVICE)
    return s


# ------------------------------------------------------------------ one pass
def prepare(case, seed):
    if case["kind"] == "serve":
        return _prepare_serve(case, seed)
    s = _inputs(case, seed)
    s["case"] = case
    s["part"] = build_part(s["category"], s["spec"], s["params"],
                           Runtime(dtype=s["dtype"], device=torch.device(DEVICE)))
    s["cache"] = LayerCache(kv=s["kv"], page_size=PAGE, block_table=s["table"], state=s["state"])
    if case["kind"] == "head":
        rows = case["rows"]
        s["sampler"] = Sampler(case["vocab"], rows, torch.device(DEVICE))
        s["requests"] = ["request %d" % i for i in range(rows)]
        gen = torch.Generator().manual_seed(seed)
        for i, r in enumerate(s["requests"]):
            earlier = torch.randint(0, case["vocab"], (40,), generator=gen).tolist()
            s["sampler"].add_request(
                r, SamplingParams(temperature=case["temperature"], top_p=case["top_p"],
                                  repetition_penalty=case["penalty"], seed=seed % 1000 + i), i,
                earlier)
    return s


def run(s):
    kind = s["case"]["kind"]
    if kind == "serve":
        return _run_serve(s)
    if kind == "head":
        logits = s["part"].forward(s["x"])
        return {"logits": logits, "tokens": s["sampler"].sample(s["requests"], logits)}
    if s["category"] == "ffn":
        return {"y": s["part"].forward(s["x"], s["ctx"])}
    out = {"y": s["part"].forward(s["x"], s["ctx"], s["cache"])}
    if s["kv"] is not None:
        out["kv"] = s["kv"]
    if s["state"] is not None:
        out["state"] = s["state"]
    return out


def _prepare_serve(case, seed):
    raw = dict(architectures=["LlamaForCausalLM"], num_hidden_layers=case["depth"],
               hidden_size=case["width"], num_attention_heads=case["heads"],
               num_key_value_heads=case["kv_heads"], head_dim=case["dim"],
               intermediate_size=case["ff"], vocab_size=case["vocab"], tie_word_embeddings=True,
               rope_theta=500000.0, rope_scaling=LLAMA3, rms_norm_eps=1e-5,
               max_position_embeddings=131072, hidden_act="silu")
    cfg = config_from_dict(raw)
    model = load_model(None, dtype="bfloat16", device=DEVICE, config=cfg,
                       tensors=random_checkpoint(cfg, seed, std=0.02, norm_noise=0.1, device=DEVICE))
    n, prompt, new = case["requests"], case["prompt"], case["new"]
    stepper = make_stepper(model, page_size=PAGE, num_pages=n * (-(-(prompt + new) // PAGE)) + 8,
                           num_slots=n + 1)
    gen = torch.Generator().manual_seed(seed)
    prompts = [torch.randint(0, case["vocab"], (prompt - i * prompt // (2 * n),),
                             generator=gen).tolist() for i in range(n)]
    following = torch.randint(0, case["vocab"], (new, n), generator=gen).tolist()
    s = {"case": case, "model": model, "stepper": stepper, "prompts": prompts,
         "following": following}
    _run_serve(s)       # a server is warm when its users come: decode graphs are captured
    return s


def _run_serve(s):
    """Requests come in, their prompts are run, ``new`` given tokens follow one by one, and they
    leave; the logits after the prompts and after every token."""
    stepper, prompts = s["stepper"], s["prompts"]
    for i in range(len(prompts)):
        stepper.add_request(i)
    out = [stepper.step([StepEntry(i, p, (len(p) - 1,)) for i, p in enumerate(prompts)]).clone()]
    for row in s["following"]:
        out.append(stepper.step([StepEntry(i, [t], (0,)) for i, t in enumerate(row)]).clone())
    for i in range(len(prompts)):
        stepper.free_request(i)
    return out


# ------------------------------------------------------------------ what a pass cannot do without
def _visible(case, spec):
    """Pairs of a query and a key that it sees."""
    window = getattr(spec, "window", None)
    chunk = getattr(spec, "chunk", None)
    total = 0
    for cached, new in _lengths(case):
        for p in range(cached, cached + new):
            if chunk:
                total += p % chunk + 1
            elif window:
                total += min(p + 1, window + getattr(spec, "keep_first", 0))
            else:
                total += p + 1
    return total


def _matrix_numbers(case):
    category, spec = _spec(case)
    return sum(math.prod(ps.shape) for ps in part_class(category, spec).param_specs(spec).values())


def work(case):
    kind, width = case["kind"], case["width"]
    size = 4 if case.get("dtype") == "float32" else 2
    if kind == "serve":
        layer = width * (case["heads"] + 2 * case["kv_heads"]) * case["dim"] \
            + width * case["heads"] * case["dim"] + 3 * width * case["ff"]
        head = width * case["vocab"]
        n, new = case["requests"], case["new"]
        prompts = [case["prompt"] - i * case["prompt"] // (2 * n) for i in range(n)]
        kv = 2 * case["kv_heads"] * case["dim"] * 2 * case["depth"]
        tokens = sum(prompts) + n * new
        pairs = sum(p * (p + 1) // 2 + sum(p + k + 1 for k in range(new)) for p in prompts)
        bytes_ = (1 + new) * 2 * (case["depth"] * layer + head) \
            + kv * (tokens + sum(p + k for p in prompts for k in range(new))) \
            + 4 * n * (1 + new) * case["vocab"]
        flops = 2 * tokens * case["depth"] * layer + 2 * n * (1 + new) * head \
            + 4 * pairs * case["heads"] * case["dim"] * case["depth"]
        return {"bytes": bytes_, "flops": flops}
    category, spec = _spec(case)
    numbers = _matrix_numbers(case)
    if kind == "head":
        return {"bytes": numbers * 2 + case["rows"] * (width * 2 + case["vocab"] * 4),
                "flops": 2 * case["rows"] * numbers}
    if kind == "mlp":
        return {"bytes": size * (numbers + 2 * case["rows"] * width),
                "flops": 2 * case["rows"] * numbers}
    if kind == "experts":
        one = 3 * width * case["ff"]
        used = min(case["experts"], case["rows"] * case["top"])
        rest = numbers - case["experts"] * one
        return {"bytes": 2 * (rest + used * one + 2 * case["rows"] * width),
                "flops": 2 * case["rows"] * (rest + case["top"] * one)}
    lengths = _lengths(case)
    tokens = sum(new for _, new in lengths)
    bytes_ = size * (numbers + 2 * tokens * width)
    flops = 2 * tokens * numbers
    if kind in ("attention", "optioned"):
        dim = spec.head_dim
        seen = sum(min(c, _reach(spec)) for c, _ in lengths)
        bytes_ += size * 2 * spec.num_kv_heads * dim * (seen + tokens)
        flops += 4 * _visible(case, spec) * spec.num_heads * dim
    elif kind == "latent":
        row = spec.kv_rank + spec.rot_dim
        seen = sum(min(c, _reach(spec)) for c, _ in lengths)
        bytes_ += 2 * row * (seen + tokens)
        # keys and values made once a token and head, or folded into queries and outputs
        flops += 2 * _visible(case, spec) * spec.num_heads * (spec.qk_dim + spec.rot_dim + spec.v_dim)
    else:
        state = math.prod(part_class(category, spec).cache_need(spec).state.shape)
        bytes_ += 2 * 4 * len(lengths) * state
        flops += tokens * (8 * spec.num_heads * spec.qk_dim * spec.v_dim if kind == "delta"
                           else 7 * spec.inner * spec.state)
    return {"bytes": bytes_, "flops": flops}


def _reach(spec):
    window = getattr(spec, "window", None)
    return getattr(spec, "chunk", None) or (window + getattr(spec, "keep_first", 0) if window
                                            else 1 << 60)


def tolerance(case):
    """About four times what the outputs differ by from the same in 64 bits: bfloat16 rounds
    activations between a layer's products to 8 bits (0.0024 to 0.0046 on the layers), the 32-bit
    mode and the head sum in 24 bits (1.4e-6 and 3.2e-6)."""
    if case.get("dtype") == "float32":
        return {"rel": 6e-6}
    if case["kind"] == "head":
        return {"rel": 1.3e-5, "differ": 0.01}
    if case["kind"] == "serve":
        return {"rel": 0.03}
    return {"rel": 0.012}


# ------------------------------------------------------------------ the same in 64 bits
def exact(case, seed):
    if case["kind"] == "serve":
        return None
    s = _inputs(case, seed)
    s["x"] = s["x"].double()
    s["w"] = {k: v.double() for k, v in s["params"].items()}
    kind = case["kind"]
    if kind == "head":
        return {"logits": s["x"] @ s["w"]["weight"].T, "tokens": None}
    if kind == "mlp":
        return {"y": _gated(s["x"], s["w"]["gate_up.weight"], s["w"]["down.weight"])}
    if kind == "experts":
        return {"y": _exact_experts(s)}
    if kind == "attention" or kind == "optioned":
        return {"y": _exact_attention(s), "kv": None}
    if kind == "latent":
        return {"y": _exact_latent(s), "kv": None}
    if case["cached"]:
        return None         # where in a state's row what is kept is this package's affair
    return {"y": (_exact_delta if kind == "delta" else _exact_scan)(s), "state": None}


def _silu(v):
    return v * torch.sigmoid(v)


def _gated(x, gate_up, down):
    g, u = (x @ gate_up.T).chunk(2, dim=-1)
    return (_silu(g) * u) @ down.T


def _clamped(x, gate_up, down, limit, alpha):
    g, u = (x @ gate_up.T).chunk(2, dim=-1)
    g, u = g.clamp(max=limit), u.clamp(-limit, limit)
    return (g * torch.sigmoid(alpha * g) * (u + 1)) @ down.T


def _frequencies(p):
    freqs = []
    for j in range(p.rotary_dim // 2):
        f = p.theta ** (-2.0 * j / p.rotary_dim)
        if p.scaling is not None:
            sc, wave = p.scaling, 2 * math.pi / f
            old = sc.original_max_position_embeddings
            if wave > old / sc.low_freq_factor:
                f /= sc.factor
            elif wave >= old / sc.high_freq_factor:
                mix = (old / wave - sc.low_freq_factor) / (sc.high_freq_factor - sc.low_freq_factor)
                f = (1 - mix) * f / sc.factor + mix * f
        freqs.append(f)
    return torch.tensor(freqs, dtype=torch.float64, device=DEVICE)


def _rotate(x, positions, p):
    """x: [tokens, heads, dim]; feature i of the first rotary_dim turns with i + rotary_dim / 2."""
    half = p.rotary_dim // 2
    angle = positions.double()[:, None, None] * _frequencies(p)
    a, b, rest = x[..., :half], x[..., half:2 * half], x[..., 2 * half:]
    return torch.cat([a * angle.cos() - b * angle.sin(), b * angle.cos() + a * angle.sin(), rest], -1)


def _over_rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _requests(s):
    """(index, cached, new, token range) of each request."""
    at = 0
    for i, (cached, new) in enumerate(s["lengths"]):
        yield i, cached, new, slice(at, at + new)
        at += new


def _cached_rows(s, i, n):
    """The first n rows of request i: [n, planes, heads, features]."""
    pages = s["kv"][s["table"][i].long()]                   # [width, planes, heads, page, features]
    return pages.permute(0, 3, 1, 2, 4).flatten(0, 1)[:n].double()


def _mask(spec, cached, new):
    i = torch.arange(cached, cached + new, device=DEVICE)[:, None]
    j = torch.arange(cached + new, device=DEVICE)[None]
    see = j <= i
    if getattr(spec, "chunk", None):
        see &= j >= i // spec.chunk * spec.chunk
    elif spec.window:
        see &= (i - j < spec.window) | (j < getattr(spec, "keep_first", 0))
    return see


def _exact_attention(s):
    spec, w, x = s["spec"], s["w"], s["x"]
    heads, kv_heads, dim = spec.num_heads, spec.num_kv_heads, spec.head_dim
    positions = s["ctx"].positions
    proj = x @ w["qkv.weight"].T
    q_cols, k_cols = heads * dim, kv_heads * dim
    gate = proj[:, q_cols + 2 * k_cols:]
    proj = proj[:, :q_cols + 2 * k_cols]
    if spec.bias:
        proj = proj + w["qkv.bias"]
    q, k, v = (t.reshape(len(x), -1, dim) for t in proj.split([q_cols, k_cols, k_cols], dim=1))
    if spec.qk_norm_eps is not None:
        q, k = _over_rms(q, spec.qk_norm_eps), _over_rms(k, spec.qk_norm_eps)
        if spec.qk_norm_weight:
            q, k = q * w["q_norm.weight"], k * w["k_norm.weight"]
    if spec.position.kind == "rope":
        q, k = _rotate(q, positions, spec.position), _rotate(k, positions, spec.position)
    if spec.q_temp is not None:
        coef, every = spec.q_temp
        q = q * (1 + coef * torch.log((positions.double() + 1).div(every).floor() + 1))[:, None, None]
    scale = spec.scale if spec.scale is not None else dim ** -0.5
    out = torch.empty(len(x), heads, dim, dtype=torch.float64, device=DEVICE)
    for i, cached, new, at in _requests(s):
        old = _cached_rows(s, i, cached)
        keys = torch.cat([old[:, 0], k[at]]).repeat_interleave(heads // kv_heads, dim=1)
        values = torch.cat([old[:, 1], v[at]]).repeat_interleave(heads // kv_heads, dim=1)
        see = _mask(spec, cached, new)
        for h in range(heads):
            z = q[at, h] @ keys[:, h].T * scale
            if spec.softcap:
                z = spec.softcap * torch.tanh(z / spec.softcap)
            if spec.score_bias:
                z = z + w["score_bias"][h]
            if spec.weights == "sigmoid":
                p = torch.sigmoid(z) * see
            else:
                z = z.masked_fill(~see, -math.inf)
                if spec.sink == "learned":
                    z = torch.cat([z, w["sink"][h].expand(new, 1)], dim=1)
                p = torch.softmax(z, dim=1)[:, :cached + new]
            out[at, h] = p @ values[:, h]
    y = out.flatten(1)
    if spec.feature_gate:
        y = y * torch.sigmoid(gate)
    return y @ w["o.weight"].T


def _exact_latent(s):
    spec, w, x = s["spec"], s["w"], s["x"]
    heads, dim, rot, rank = spec.num_heads, spec.qk_dim, spec.rot_dim, spec.kv_rank
    positions = s["ctx"].positions
    proj = x @ w["in.weight"].T
    first = spec.q_rank if spec.q_rank is not None else heads * (dim + rot)
    q, down, gate = proj[:, :first], proj[:, first:first + rank + rot], proj[:, first + rank + rot:]
    if spec.q_rank is not None:
        q = (_over_rms(q, spec.norm_eps) * w["q_norm.weight"]) @ w["uq.weight"].T
    q = q.reshape(len(x), heads, dim + rot)
    q_rot = _rotate(q[..., dim:], positions, spec.position)
    c = _over_rms(down[:, :rank], spec.norm_eps) * w["kv_norm.weight"]
    k_rot = _rotate(down[:, None, rank:], positions, spec.position)[:, 0]
    uk, uv = (w[n].reshape(heads, -1, rank) for n in ("uk.weight", "uv.weight"))
    out = torch.empty(len(x), heads, uv.shape[1], dtype=torch.float64, device=DEVICE)
    for i, cached, new, at in _requests(s):
        old = _cached_rows(s, i, cached)[:, 0, 0]
        lat, kr = torch.cat([old[:, :rank], c[at]]), torch.cat([old[:, rank:], k_rot[at]])
        see = _mask(spec, cached, new)
        for h in range(heads):
            z = q[at, h, :dim] @ (lat @ uk[h].T).T + q_rot[at, h] @ kr.T
            p = torch.softmax((z * spec.scale).masked_fill(~see, -math.inf), dim=1)
            out[at, h] = p @ (lat @ uv[h].T)
    g = torch.sigmoid(gate)
    out = out * (g[:, :, None] if spec.gate_per_head else g.reshape(out.shape))
    return out.flatten(1) @ w["o.weight"].T


def _exact_experts(s):
    spec, w, x = s["spec"], s["w"], s["x"]
    e, ff, width = spec.num_experts, spec.expert_size, spec.hidden_size
    logits = x @ w["router.weight"].T
    z = logits[:, :e]
    scores = torch.sigmoid(z) if spec.score == "sigmoid" else torch.softmax(z, dim=1)
    choice = scores + (w["router.correction"] if spec.choice_bias else 0.0)
    if spec.groups is not None:
        count, keep = spec.groups
        best = choice.reshape(len(x), count, -1).amax(-1)
        kept = torch.zeros_like(best, dtype=torch.bool).scatter(1, best.topk(keep, dim=1).indices, True)
        choice = choice.masked_fill(~kept.repeat_interleave(e // count, dim=1), -math.inf)
    chosen = choice.topk(spec.top, dim=1).indices
    weight = scores.gather(1, chosen)
    if spec.renormalize:
        weight = weight / (weight.sum(1, keepdim=True) + spec.renorm_eps)
    weight = weight * spec.weight_scale
    clamped = spec.activation == "clamped_swish"
    y = torch.zeros_like(x)
    gate_up = w["experts.gate_up.weight"].reshape(e, 2 * ff, width)
    down = w["experts.down.weight"].reshape(e, width, ff)
    for k in range(e):
        rows, place = (chosen == k).nonzero(as_tuple=True)
        a, xe = weight[rows, place][:, None], x[rows]
        if spec.scale_input:
            y[rows] += _gated(a * xe, gate_up[k], down[k])
        elif clamped:
            y[rows] += a * _clamped(xe, gate_up[k], down[k], spec.limit, spec.swish_alpha)
        else:
            y[rows] += a * _gated(xe, gate_up[k], down[k])
    if clamped:
        shared = _clamped(x, w["shared.gate_up.weight"], w["shared.down.weight"], spec.shared_limit,
                          spec.swish_alpha)
    else:
        shared = _gated(x, w["shared.gate_up.weight"], w["shared.down.weight"])
    return y + (shared * torch.sigmoid(logits[:, e:e + 1]) if spec.shared_gate else shared)


def _convolved(x, weight, bias=None):
    """Causal convolution per channel from a sequence's start, then SiLU."""
    taps = weight.shape[1]
    padded = torch.cat([x.new_zeros(taps - 1, x.shape[1]), x])
    y = sum(padded[t:t + len(x)] * weight[:, t] for t in range(taps))
    return _silu(y if bias is None else y + bias)


def _exact_delta(s):
    spec, w, x = s["spec"], s["w"], s["x"]
    heads, groups, dim, vdim = spec.num_heads, spec.num_kv_heads, spec.qk_dim, spec.v_dim
    proj = x @ w["in.weight"].T
    channels = 2 * groups * dim + heads * vdim
    beta = torch.sigmoid(proj[:, channels:channels + heads])
    rest = proj[:, channels + heads:]
    if spec.head_decay:
        a, gate = rest[:, :heads, None], rest[:, heads:]
        bias = w["dt_bias"].reshape(heads, 1)
    else:
        a = (rest[:, :spec.decay_rank] @ w["a2.weight"].T).reshape(len(x), heads, dim)
        gate = rest[:, spec.decay_rank:] @ w["g2.weight"].T
        bias = w["dt_bias"].reshape(heads, dim)
    decay = torch.exp(-torch.exp(w["A_log"])[:, None] * torch.nn.functional.softplus(a + bias))
    out = torch.empty(len(x), heads, vdim, dtype=torch.float64, device=DEVICE)
    for _, _, new, at in _requests(s):
        y = _convolved(proj[at, :channels], w["conv.weight"])
        q, k, v = y.split([groups * dim, groups * dim, heads * vdim], dim=1)
        q, k = (t.reshape(new, groups, dim) for t in (q, k))
        q, k = (t / torch.sqrt((t * t).sum(-1, keepdim=True) + spec.unit_eps) for t in (q, k))
        q, k = ((t * f).repeat_interleave(heads // groups, dim=1) for t, f in ((q, dim ** -0.5), (k, 1.0)))
        v, b, g = v.reshape(new, heads, vdim), beta[at], decay[at]
        mem = torch.zeros(heads, dim, vdim, dtype=torch.float64, device=DEVICE)
        for t in range(new):
            mem = mem * g[t][:, :, None]
            u = b[t][:, None] * (v[t] - torch.bmm(k[t][:, None], mem)[:, 0])
            mem = torch.baddbmm(mem, k[t][:, :, None], u[:, None])
            out[at.start + t] = torch.bmm(q[t][:, None], mem)[:, 0]
    out = _over_rms(out, spec.norm_eps) * w["norm.weight"]
    gate = _silu(gate) if spec.gate_activation == "silu" else torch.sigmoid(gate)
    return (out.flatten(1) * gate) @ w["o.weight"].T


def _exact_scan(s):
    spec, w, x = s["spec"], s["w"], s["x"]
    inner, n, rank = spec.inner, spec.state, spec.dt_rank
    xz = x @ w["in.weight"].T
    a = -torch.exp(w["A_log"])
    out = torch.empty(len(x), inner, dtype=torch.float64, device=DEVICE)
    for _, _, new, at in _requests(s):
        xc = _convolved(xz[at, :inner], w["conv.weight"], w["conv.bias"])
        proj = xc @ w["x.weight"].T
        dt = torch.nn.functional.softplus(proj[:, :rank] @ w["dt.weight"].T + w["dt.bias"])
        b, c = proj[:, rank:rank + n], proj[:, rank + n:]
        mem = torch.zeros(inner, n, dtype=torch.float64, device=DEVICE)
        for t in range(new):
            mem = torch.exp(dt[t][:, None] * a) * mem + (dt[t] * xc[t])[:, None] * b[t]
            out[at.start + t] = mem @ c[t] + w["D"] * xc[t]
    return (out * _silu(xz[:, inner:])) @ w["o.weight"].T
