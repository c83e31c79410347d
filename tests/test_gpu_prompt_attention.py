"""The tcgen05 prompt attention with probabilities in three bfloat16 parts, paged and latent form, against
attention in double precision over the same bfloat16 numbers.  Pages that no token sees hold NaN."""
import math

import pytest
import torch

from test_gpu_kernels import DEV, rnd

pytestmark = pytest.mark.gpu


def i32(values):
    return torch.tensor(values, dtype=torch.int32, device=DEV)


def batch(lens_q, lens_kv):
    from mstar_b200.parts.base import StepContext

    starts = [0]
    for n in lens_q:
        starts.append(starts[-1] + n)
    pos = i32([k - q + i for q, k in zip(lens_q, lens_kv) for i in range(q)])
    return StepContext(num_tokens=starts[-1], num_entries=len(lens_q),
                       token_req=i32([r for r, q in enumerate(lens_q) for _ in range(q)]), positions=pos,
                       cache_pos=pos, qo_indptr=i32(starts), kv_len=i32(lens_kv), slots=i32(list(range(len(lens_q)))),
                       q_lens=list(lens_q), kv_lens=list(lens_kv), max_q_len=max(lens_q), max_kv_len=max(lens_kv),
                       num_decode=0), starts


def visible(q, kv, window, keep_first, chunk):
    i = torch.arange(kv - q, kv, device=DEV)[:, None]
    j = torch.arange(kv, device=DEV)[None]
    see = j <= i
    if chunk:
        return see & (j >= i // chunk * chunk)
    return see & ((i - j < window) | (j < keep_first)) if window else see


def paged(lens_q, lens_kv, page, lowest, make_row, shape, keep_first=0):
    """A cache of NaN whose visible rows (keys from lowest[r] on and the first keep_first) are filled;
    pages without a visible key are -1 in the table."""
    width = -(-max(lens_kv) // page)
    order = torch.randperm(len(lens_q) * width + 2, generator=torch.Generator().manual_seed(3)).tolist()
    cache = torch.full((len(order), *shape), float("nan"), dtype=torch.bfloat16, device=DEV)
    table = torch.full((len(lens_q), width), -1, dtype=torch.int32)
    for r, n in enumerate(lens_kv):
        for key in range(n):
            if key >= lowest[r] or key < keep_first:
                table[r, key // page] = pg = order[r * width + key // page]
                make_row(cache, pg, key % page, r, key)
    return cache, table.to(DEV)


FORMS = {
    "sink": dict(softcap=30.0, sink=True, gate="feature"),
    "window": dict(window=70, softcap=20.0),
    "keep_first": dict(window=70, keep_first=5, gate="head"),
    "keep_many": dict(window=33, keep_first=66),
    "chunk": dict(chunk=96, sigmoid=True, softcap=30.0, bias=True, gate="feature"),
    "sigmoid": dict(sigmoid=True, bias=True),
    "plain": dict(bias=True),
    "low_cap": dict(softcap=5.0, sink=True, window=100),        # scores past half of the cap
    "high_cap": dict(softcap=60.0, bias=True),                  # a cap too high to be the reference maximum
}


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("lens_q,lens_kv,nq,nkv,hd,page", [
    ([130, 17], [130, 300], 4, 1, 64, 16),       # a row tile and one row more; keys shared among CTAs
    ([50], [333], 6, 2, 128, 8),                 # a group of 3: 126 of 128 rows
    ([300], [300], 1, 1, 128, 64),               # one head a group
    ([40, 40, 64], [40, 200, 64], 16, 8, 64, 32),
    ([1, 130, 1], [290, 300, 33], 4, 1, 64, 128),    # pages of several tiles; single tokens beside a portion
    ([70, 1], [600, 257], 4, 2, 128, 256)])
def test_prompt_attention_with_options(form, lens_q, lens_kv, nq, nkv, hd, page, monkeypatch):
    from mstar_b200 import ops

    o = FORMS[form]
    window, keep, chunk = o.get("window", 0), o.get("keep_first", 0), o.get("chunk", 0)
    ctx, starts = batch(lens_q, lens_kv)
    T, G, scale = starts[-1], nq // nkv, hd ** -0.5
    q = rnd(T, nq * hd, dtype=torch.bfloat16, seed=1, scale=2.0)
    ks = [rnd(n, nkv, hd, dtype=torch.bfloat16, seed=10 + r) for r, n in enumerate(lens_kv)]
    vs = [rnd(n, nkv, hd, dtype=torch.bfloat16, seed=20 + r) for r, n in enumerate(lens_kv)]
    see = [visible(a, n, window, keep, chunk) for a, n in zip(lens_q, lens_kv)]

    def row(cache, pg, slot, r, key):
        cache[pg, 0, :, slot], cache[pg, 1, :, slot] = ks[r][key], vs[r][key]

    lowest = [max(0, n - a - window + 1) if window else (n - a) // chunk * chunk if chunk else 0
              for a, n in zip(lens_q, lens_kv)]
    cache, table = paged(lens_q, lens_kv, page, lowest, row, (2, nkv, page, hd), keep)
    sink = rnd(nq, seed=5) if o.get("sink") else None
    bias = rnd(nq, seed=6) if o.get("bias") else None
    gate = None
    if o.get("gate"):
        gate = rnd(T, 8 + nq * (hd if o["gate"] == "feature" else 1), seed=7)[:, 8:]
    args = (q, cache, table, ctx.token_req, ctx.cache_pos, nq, nkv, hd, hd, page, window, keep, scale)
    kw = dict(ctx=ctx, gate=gate, softcap=o.get("softcap"), sink=sink, chunk=chunk,
              sigmoid=bool(o.get("sigmoid")), bias=bias)
    assert ops._sink_prompt_map(q, cache, ctx, nq, nkv, hd, hd, page) is not None
    got = ops.sink_attention(*args, **kw)
    monkeypatch.setattr(ops, "prompt_splits", lambda *a: 1)
    alone = ops.sink_attention(*args, **kw)
    monkeypatch.setattr(ops, "prompt_splits", lambda *a: 7)
    shared = ops.sink_attention(*args, **kw)
    ops.check_error_word(DEV)

    want = torch.empty(T, nq, hd, dtype=torch.float64, device=DEV)
    size = torch.empty_like(want)
    for r, s in enumerate(see):
        for h in range(nq):
            at = slice(starts[r], starts[r + 1])
            z = q.view(T, nq, hd)[at, h].double() @ ks[r][:, h // G].double().T * scale
            if o.get("softcap"):
                z = o["softcap"] * torch.tanh(z / o["softcap"])
            if bias is not None:
                z = z + bias[h].double()
            if o.get("sigmoid"):
                p = torch.sigmoid(z) * s
            else:
                z = z.masked_fill(~s, -math.inf)
                if sink is not None:
                    z = torch.cat([z, sink[h].double().expand(len(z), 1)], dim=1)
                p = torch.softmax(z, dim=1)[:, :s.shape[1]]
            want[at, h] = p @ vs[r][:, h // G].double()
            size[at, h] = p @ vs[r][:, h // G].double().abs()
    if gate is not None:
        g = torch.sigmoid(gate.double()).reshape(T, nq, -1)
        want, size = want * g, size * g
    # the result's rounding to bfloat16, and what float scores (sums of hd products, then an
    # exponential) and probabilities of 16 bits leave of the sum's terms
    bound = 2 ** -8 * want.abs() + 2 ** -13 * size + 1e-6
    for y in (got, alone, shared):
        assert ((y.view(T, nq, hd).double() - want).abs() <= bound).all()


@pytest.mark.parametrize("window", [0, 70])
@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("lens_q,lens_kv,heads,dim,rank,rot,page", [
    ([130, 33], [130, 300], 3, 64, 32, 32, 16),
    ([200], [1000], 2, 128, 64, 64, 8),
    ([64, 64, 65], [64, 64, 200], 1, 128, 40, 8, 4)])
def test_latent_prompt_attention(window, gated, lens_q, lens_kv, heads, dim, rank, rot, page, monkeypatch):
    from mstar_b200 import ops

    ctx, starts = batch(lens_q, lens_kv)
    T, scale = starts[-1], (dim + rot) ** -0.5
    q = rnd(T, heads, dim + rot, dtype=torch.bfloat16, seed=1)
    rows = [rnd(n, rank + rot, dtype=torch.bfloat16, seed=10 + r) for r, n in enumerate(lens_kv)]
    w_kv = rnd(2 * heads * dim, rank, dtype=torch.bfloat16, seed=2, scale=rank ** -0.5)
    gate = rnd(T, heads + 3, seed=7)[:, 3:] if gated else None

    def row(cache, pg, slot, r, key):
        cache[pg, 0, 0, slot] = rows[r][key]

    lowest = [max(0, n - a - window + 1) if window else 0 for a, n in zip(lens_q, lens_kv)]
    cache, table = paged(lens_q, lens_kv, page, lowest, row, (1, 1, page, rank + rot))
    assert ops.latent_prompt_takes(q, cache, dim, dim, rank, rot)
    groups = ops.latent_prompt_groups(lens_q, lens_kv, window, heads * dim)
    assert groups and sum(g[1] for g in groups) == len(lens_q)
    want = torch.empty(T, heads, dim, dtype=torch.float64, device=DEV)
    size = torch.empty_like(want)
    wk, wv = w_kv.double().view(2, heads, dim, rank)
    for r in range(len(lens_q)):
        see = visible(lens_q[r], lens_kv[r], window, 0, 0)
        at = slice(starts[r], starts[r + 1])
        lat, kr = rows[r][:, :rank].double(), rows[r][:, rank:].double()
        for h in range(heads):
            qd = q[at, h].double()
            z = (qd[:, :dim] @ (lat @ wk[h].T).T + qd[:, dim:] @ kr.T) * scale
            p = torch.softmax(z.masked_fill(~see, -math.inf), dim=1)
            want[at, h], size[at, h] = p @ (lat @ wv[h].T), p @ (lat @ wv[h].T).abs()
    if gated:
        g = torch.sigmoid(gate.double())[:, :, None]
        want, size = want * g, size * g
    bound = 2 ** -8 * want.abs() + 2 ** -13 * size + 1e-6
    few = [(i, 1, ops.latent_prompt_groups([a], [n], window, heads * dim)[0][2]) for i, (a, n) in enumerate(zip(lens_q, lens_kv))]
    for parts, splits in ((groups, None), (few, None), (groups, 1), (groups, 5)):
        if splits:
            monkeypatch.setattr(ops, "prompt_splits", lambda *a, n=splits: n)
        out = torch.full((T, heads * dim), float("nan"), dtype=torch.bfloat16, device=DEV)
        ops.latent_attention_prompt(q, cache, table, ctx, parts, w_kv, heads, dim, rank, rot, page, window, scale,
                                    out, gate=gate)
        ops.check_error_word(DEV)
        assert ((out.view(T, heads, dim).double() - want).abs() <= bound).all()


@pytest.mark.parametrize("hd,nq,nkv", [(128, 8, 4), (64, 16, 4)])
def test_capped_rows_have_the_bits_of_what_they_see(hd, nq, nkv):
    """Later tokens of a request, the next request and what lies on a page behind the last key change no bit of a
    row, though the two forms of tanh that its scores' sizes choose between differ."""
    from mstar_b200 import ops

    lens, page, scale = [200, 61], 64, hd ** -0.5
    ctx, starts = batch(lens, lens)
    T, half = starts[-1], 130
    q = rnd(T, nq * hd, dtype=torch.bfloat16, seed=1)
    kv = rnd(sum(-(-n // page) for n in lens), 2, nkv, page, hd, dtype=torch.bfloat16, seed=2)
    table = torch.tensor([[3, 1, 2, 0], [4, 0, 0, 0]], dtype=torch.int32, device=DEV)

    def run(queries, cache):
        out = ops.sink_attention(queries, cache, table, ctx.token_req, ctx.cache_pos, nq, nkv, hd, hd, page, 0, 0,
                                 scale, ctx=ctx, softcap=30.0)
        ops.check_error_word(DEV)
        return out

    want = run(q, kv)
    q2, kv2 = q.clone(), kv.clone()
    q2[half:] *= 40                              # from token `half` of the first request on
    kv2[2, 0, :, half - 128:] *= 40              # ... their keys
    kv2[0, 0] *= 40
    kv2[4, 0] *= 40                              # the second request's keys
    got = run(q2, kv2)
    assert torch.equal(got[:half], want[:half]) and not torch.equal(got[half:], want[half:])
    kv3 = kv.clone()
    kv3[0, 0, :, 200 - 192:] *= 40               # behind the first request's last key
    kv3[4, 0, :, 61:] *= 40
    assert torch.equal(run(q, kv3), want)


def cancelling(p, seed, reserve=4):
    """bfloat16 values [keys, probes] whose sums with the weights p [probes, keys] (double) nearly vanish: random
    ones, then corrections by reserved keys, each of which leaves 2^-9 of what is left.  And the size of a sum
    whose terms have independent errors: the root of the sum of their squares."""
    v = rnd(p.shape[1], p.shape[0], dtype=torch.bfloat16, seed=seed)
    rows = torch.arange(len(p), device=DEV)
    spare = p.argsort(dim=1, descending=True)[:, 2:2 + reserve]     # keys with much weight
    for i in range(reserve):
        v[spare[:, i], rows] = 0
    for i in range(reserve):
        left = (p * v.double().T).sum(1)
        v[spare[:, i], rows] = (-left / p[rows, spare[:, i]]).to(torch.bfloat16)
    assert ((p * v.double().T).sum(1).abs() < 2 ** -26 * p.sum(1)).all()
    return v, (p * v.double().T).square().sum(1).sqrt()


# What is left of sums that vanish is the error of their terms.  That of a probability: the rounding of a base-2
# exponent of at most 8 (two roundings of 2^-22 at most, times ln 2), the exponential's 2^-22: some 2^-22 in the
# mean.  A third bfloat16 part leaves 2^-27 of it; without one the second part's rounding leaves 2^-18.8 in the mean.
TERM = 2 ** -20.5


@pytest.mark.parametrize("form", ["plain", "sink", "cap", "low_cap", "sigmoid"])
@pytest.mark.parametrize("hd,splits", [(64, 1), (128, 1), (128, 3)])
def test_probabilities_keep_24_bits(form, hd, splits, monkeypatch):
    from mstar_b200 import ops

    T, past, page = 40, 150, 16
    N, scale, nq = T + past, hd ** -0.5, 2
    ctx, _ = batch([T], [N])
    q, k = rnd(T, nq * hd, dtype=torch.bfloat16, seed=1), rnd(N, hd, dtype=torch.bfloat16, seed=2)
    cap = {"cap": 50.0, "low_cap": 10.0}.get(form)
    sink = rnd(nq, seed=5) if form == "sink" else None
    z = q.view(T, nq, hd)[:, 0].double() @ k.double().T * scale         # the probes: head 0, a feature a token
    if cap:
        z = cap * torch.tanh(z / cap)
    p = torch.sigmoid(z) if form == "sigmoid" else torch.exp(z)
    p = p * visible(T, N, 0, 0, 0)
    v, size = cancelling(p, 3)
    v = torch.cat([v, rnd(N, hd - T, dtype=torch.bfloat16, seed=4)], dim=1)
    total = torch.ones_like(size) if form == "sigmoid" else p.sum(1) + (sink[0].double().exp() if sink is not None else 0)

    def row(cache, pg, slot, r, key):
        cache[pg, 0, 0, slot], cache[pg, 1, 0, slot] = k[key], v[key]

    cache, table = paged([T], [N], page, [0], row, (2, 1, page, hd))
    assert ops._sink_prompt_map(q, cache, ctx, nq, 1, hd, hd, page) is not None
    monkeypatch.setattr(ops, "prompt_splits", lambda *a: splits)
    got = ops.sink_attention(q, cache, table, ctx.token_req, ctx.cache_pos, nq, 1, hd, hd, page, 0, 0, scale, ctx=ctx,
                             softcap=cap, sink=sink, sigmoid=form == "sigmoid")
    ops.check_error_word(DEV)
    left = got.view(T, nq, hd)[:, 0].double().diagonal(dim1=0, dim2=1) * total / size
    assert left.square().mean().sqrt() < TERM


@pytest.mark.parametrize("dim,splits", [(64, 1), (128, 1), (64, 3)])
def test_latent_probabilities_keep_24_bits(dim, splits, monkeypatch):
    """With up-projections that pick latents, keys and values are bfloat16 numbers and the probabilities the only
    ones that are not."""
    from mstar_b200 import ops

    T, past, page, rank, rot = 40, 150, 16, 2 * dim, 32
    N, scale = T + past, (dim + rot) ** -0.5
    ctx, _ = batch([T], [N])
    q = rnd(T, 1, dim + rot, dtype=torch.bfloat16, seed=1)
    rows = rnd(N, rank + rot, dtype=torch.bfloat16, seed=2)
    w_kv = torch.eye(2 * dim, dtype=torch.bfloat16, device=DEV)          # latents: the key's features, the value's
    z = (q[:, 0, :dim].double() @ rows[:, :dim].double().T + q[:, 0, dim:].double() @ rows[:, rank:].double().T) * scale
    p = torch.exp(z) * visible(T, N, 0, 0, 0)
    v, size = cancelling(p, 3)
    rows[:, dim:dim + T] = v

    def row(cache, pg, slot, r, key):
        cache[pg, 0, 0, slot] = rows[key]

    cache, table = paged([T], [N], page, [0], row, (1, 1, page, rank + rot))
    assert ops.latent_prompt_takes(q, cache, dim, dim, rank, rot)
    monkeypatch.setattr(ops, "prompt_splits", lambda *a: splits)
    out = torch.empty(T, dim, dtype=torch.bfloat16, device=DEV)
    ops.latent_attention_prompt(q, cache, table, ctx, [(0, 1, N)], w_kv, 1, dim, rank, rot, page, 0, scale, out)
    ops.check_error_word(DEV)
    left = out.double().diagonal(dim1=0, dim2=1) * p.sum(1) / size
    assert left.square().mean().sqrt() < TERM


def latent_layer(seed, heads=4, window=None, gate_per_head=False, q_rank=None, hidden=128, dim=64, rot=32, rank=64):
    from mstar_b200.config.layout import LatentAttentionSpec, PositionSpec
    from mstar_b200.parts.base import Runtime
    from mstar_b200.parts.registry import build_part, part_class

    spec = LatentAttentionSpec(hidden_size=hidden, num_heads=heads, qk_dim=dim, rot_dim=rot, v_dim=dim, kv_rank=rank,
                               position=PositionSpec(kind="rope", head_dim=rot, rotary_dim=rot, theta=1e4),
                               window=window, gate_per_head=gate_per_head, q_rank=q_rank)
    params = {n: rnd(*ps.shape, dtype=torch.bfloat16, seed=seed + i, scale=ps.shape[-1] ** -0.5)
              if len(ps.shape) > 1 else 1 + rnd(*ps.shape, dtype=torch.bfloat16, seed=seed + i, scale=0.1)
              for i, (n, ps) in enumerate(part_class("mixer", spec).param_specs(spec).items())}
    return build_part("mixer", spec, params, Runtime(dtype=torch.bfloat16, device=torch.device(DEV))), rank + rot


def latent_forward(part, row, lens_q, lens_kv, x, page=16):
    """The layer's outputs over requests whose earlier rows are random (the same for a request in every batch:
    ``lens_kv`` and ``x`` by request name)."""
    from mstar_b200.parts.base import LayerCache

    names = list(lens_q)
    ctx, starts = batch([lens_q[n] for n in names], [lens_kv[n] for n in names])
    ctx.num_decode = next((i for i, n in enumerate(names) if lens_q[n] > 1), len(names))
    width = max(-(-n // page) for n in lens_kv.values())
    cache = torch.empty(len(names) * width, 1, 1, page, row, dtype=torch.bfloat16, device=DEV)
    for i, n in enumerate(names):
        cache[i * width:(i + 1) * width] = rnd(width, 1, 1, page, row, dtype=torch.bfloat16, seed=100 + n)
    table = torch.arange(len(names) * width, dtype=torch.int32, device=DEV).view(-1, width)
    y = part.forward(torch.cat([x[n] for n in names]), ctx, LayerCache(kv=cache, page_size=page, block_table=table))
    return {n: y[starts[i]:starts[i + 1]].double() for i, n in enumerate(names)}


# both forms round to bfloat16 between the layer's products: 0.003 of the result each
def same(got, want):
    return (got - want).norm() <= 0.012 * want.norm()


@pytest.mark.parametrize("q_rank", [None, 48])
def test_latent_layer_with_a_gate_a_head(q_rank, monkeypatch):
    """The first product gives the gate in bfloat16 where the queries come straight from it, else in float."""
    from mstar_b200 import ops

    part, row = latent_layer(1, heads=8, gate_per_head=True, q_rank=q_rank)
    x = {0: rnd(130, 128, dtype=torch.bfloat16, seed=50)}
    calls = []
    prompt = ops.latent_attention_prompt
    monkeypatch.setattr(ops, "latent_attention_prompt", lambda *a, **k: (calls.append(1), prompt(*a, **k)))
    got = latent_forward(part, row, {0: 130}, {0: 200}, x)[0]
    ops.check_error_word(DEV)
    assert calls
    monkeypatch.setattr(ops, "latent_prompt_takes", lambda *a: False)
    assert same(got, latent_forward(part, row, {0: 130}, {0: 200}, x)[0])


@pytest.mark.parametrize("window", [None, 70])
@pytest.mark.parametrize("gate_per_head", [False, True])
def test_latent_layer_in_mixed_steps(window, gate_per_head, monkeypatch):
    """Single tokens, long portions and a short one between them, each as by itself in the folded form; with the
    keys and values of all heads made at once and of three at a time."""
    from mstar_b200 import ops

    part, row = latent_layer(1, heads=8, window=window, gate_per_head=gate_per_head)
    assert part.uv.data_ptr() == part.w_kv[8 * 64:].data_ptr()       # no second copy
    lens_q, lens_kv = {0: 1, 1: 1, 2: 100, 3: 20, 4: 70}, {0: 50, 1: 300, 2: 100, 3: 220, 4: 400}
    x = {n: rnd(q, 128, dtype=torch.bfloat16, seed=50 + n) for n, q in lens_q.items()}
    seen = []
    monkeypatch.setattr(ops, "LATENT_PROMPT_SHORT_KEYS", 50)
    prompt = ops.latent_attention_prompt
    monkeypatch.setattr(ops, "latent_attention_prompt", lambda *a, **k: (seen.append(a[4]), prompt(*a, **k)))
    got = latent_forward(part, row, lens_q, lens_kv, x)
    monkeypatch.setattr(ops, "latent_prompt_room", lambda *a: 3 * 16 * 64 * 400)
    three = latent_forward(part, row, lens_q, lens_kv, x)
    ops.check_error_word(DEV)
    assert [[g[:2] for g in groups] for groups in seen] == [[(2, 1), (4, 1)]] * 2
    monkeypatch.setattr(ops, "latent_prompt_takes", lambda *a: False)
    for n in lens_q:
        alone = latent_forward(part, row, {n: lens_q[n]}, lens_kv, x)[n]
        assert same(got[n], alone) and same(three[n], alone)
