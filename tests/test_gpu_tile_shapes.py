"""Kernels that cut their work into tiles by size, at the sizes where a tile's edge or a choice
between two shapes lies, against plain double precision."""
import functools

import pytest
import torch

from test_gpu_kernels import DEV, paged_case, rnd

pytestmark = pytest.mark.gpu


# rows at every border between the tile shapes, widths that end inside a tile, K no multiple of the
# k-block or of the 16-byte loads, operands that start off 16 bytes
@pytest.mark.parametrize("m,n,k,off", [(8, 33, 129, 0), (9, 16, 64, 0), (32, 5000, 100, 0), (33, 40, 132, 1),
                                       (700, 1700, 36, 0), (65, 3, 7, 0), (1, 17, 1, 0)])
def test_sgemm_at_the_borders_of_its_tiles(m, n, k, off):
    from mstar_b200 import ops

    a = rnd(m, k + off, seed=3)[:, off:]
    w = rnd(n, k + off, seed=4)[:, off:]
    got = ops.sgemm_nt(a, w)
    want = a.double() @ w.double().T
    # K products of magnitude about 1, rounded once each: sqrt(K) half-ulps, times a margin of 30
    assert (got.double() - want).abs().max() < 30 * 2 ** -24 * k ** 0.5 * 4
    # every shape sums in the same order: a row alone has the same bits
    assert torch.equal(ops.sgemm_nt(a[m - 1:], w), got[m - 1:])


def _sgemm(a, w, *tile):
    """The FMA kernel, or with (bn, cluster) the tensor-core kernel with that tile; None: refused."""
    from mstar_b200 import ops
    from mstar_b200.ops import lib

    out = torch.full((a.shape[0], w.shape[0]), float("nan"), device=DEV)
    args = (a.data_ptr(), w.data_ptr(), out.data_ptr(), a.shape[0], w.shape[0], a.shape[1], a.stride(0),
            w.stride(0), out.stride(0)) + tile
    word = ops.tcgen05_error_word(DEV).data_ptr() if tile else 0
    fn = lib.get("gemm_f32").mstar_sgemm_parts if tile else lib.get("gemm_f32").mstar_sgemm_nt
    code = fn(*args, word, torch.cuda.current_stream().cuda_stream)
    assert code in (0, -1)
    return out if code == 0 else None


# one row, a row past every tile width, the last tile of W shifted back by all but one row, K that ends inside a block,
# inside a pair of them and on its border, an odd number of pairs; slices of one pair (up to 2,048) and of several
@pytest.mark.parametrize("m,n,k,pad", [(1, 128, 1024, 0), (17, 129, 1028, 4), (80, 300, 1500, 0), (81, 255, 2112, 0),
                                       (33, 256, 4100, 8), (200, 640, 1024, 0), (49, 200, 2048, 0), (90, 130, 9000, 0),
                                       (18, 9500, 516, 0)])
@pytest.mark.parametrize("one_sign", [False, True])
def test_sgemm_by_parts(m, n, k, pad, one_sign):
    """Three bfloat16 parts a float: no further from 64 bits than the FMA kernel, operands of one sign (whose sums are
    all cut off to the same side) among them, the same bits from every tile, however K is shared, and for a row alone."""
    from mstar_b200 import ops

    a, w = rnd(m, k + pad, seed=5)[:, :k], rnd(n, k + pad, seed=6)[:, :k]
    if one_sign:
        a.abs_(), w.abs_()
    want = a.double() @ w.double().T
    got = ops.sgemm_nt(a, w)
    far = lambda c: ((c.double() - want).norm() / want.norm()).item()
    assert far(got) <= far(_sgemm(a, w))
    # an element of one sign: eight sums of growing numbers cut off, half a last place (2^-24 and less) each in the mean,
    # then 24 at most that are rounded
    assert not one_sign or far(got) < 2 ** -24 * (8 / 2 + 24 ** 0.5 / 4)
    # every sum into an accumulator cuts off at most a last place (2^-23) of what is there, every sum of
    # slices rounds: 8 a pair, and 24 at most
    assert ((got.double() - want).abs() <= 2 ** -23 * (8 + 24) * (a.double().abs() @ w.double().abs().T)).all()
    assert torch.equal(ops.sgemm_nt(a[m - 1:], w), got[m - 1:])
    tiles = [_sgemm(a, w, bn, cluster) for bn in (16, 32, 48, 64, 80) for cluster in (1, 2, 4, 8)]
    assert all(torch.equal(t, got) for t in tiles if t is not None) and sum(t is not None for t in tiles) >= 6
    ops.check_error_word(DEV)


@pytest.mark.parametrize("m,k", [(5, 1024), (100, 2048), (40, 4096)])
def test_sgemm_by_parts_keeps_infinities(m, k):
    from mstar_b200 import ops

    a, w = rnd(m, k, seed=7), rnd(256, k, seed=8).bfloat16().float()     # parts of w that are zero
    a[1, 3], a[2, 100], a[3, 40], a[3, 300] = float("inf"), float("nan"), float("inf"), -float("inf")
    a[4, 7], w[9, 7] = 3.4e38, 0.5               # its first part would round to an infinity
    w[11, 5], w[12, 6] = -float("inf"), float("nan")
    got, want = ops.sgemm_nt(a, w), _sgemm(a, w)
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
    both = want.isfinite()
    assert torch.equal(got[want.isinf()], want[want.isinf()]) and both[0].sum() == 254 and both[4].any()
    torch.testing.assert_close(got[both], want[both], rtol=1e-5, atol=1e-3)


@pytest.mark.parametrize("m,k", [(5, 1024), (100, 2048), (40, 4096)])
def test_sgemm_by_parts_of_products_past_the_largest_float(m, k):
    """Finite operands: where products with the lesser parts pass it too, they may be infinities of the other sign."""
    from mstar_b200 import ops

    a, w = rnd(m, k, seed=7), rnd(256, k, seed=8)
    a[1, 3], a[2, 3], w[:, 3] = 1.3e23, -3.7e30, 2.9e20 * (1 + rnd(256, seed=9).abs())
    a[3, 40], w[:, 40] = 1e25, 1e25 * rnd(256, seed=10).sign()
    got, want = ops.sgemm_nt(a, w), _sgemm(a, w)
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf()) and want[1:4].isinf().all()
    assert torch.equal(got[want.isinf()], want[want.isinf()])


@pytest.mark.parametrize("lens_q,lens_kv,nq,nkv,hd,page,window", [
    ([70, 9], [70, 200], 4, 1, 64, 16, 0),          # several blocks, a border between requests in one
    ([33, 4, 64], [100, 4, 129], 6, 2, 128, 8, 0),  # a group of 3: 63 of 64 rows
    ([40, 20], [150, 20], 2, 2, 64, 16, 37),        # a window that ends inside a tile
    ([16], [16], 32, 1, 64, 4, 0)])                 # two tokens a block
def test_float_attention_of_portions(lens_q, lens_kv, nq, nkv, hd, page, window, monkeypatch):
    """The float kernel whose blocks take several tokens, against plain attention and against the
    kernel of a block per token; rows of a request do not depend on the others of the batch."""
    from mstar_b200 import ops

    one_token, want, _ = paged_case(lens_q, lens_kv, nq, nkv, hd, page, torch.float32, 5, window)
    monkeypatch.setattr(ops, "paged_attention_generic",
                        functools.partial(ops.paged_attention_generic, entries=len(lens_q)))
    got, want, _ = paged_case(lens_q, lens_kv, nq, nkv, hd, page, torch.float32, 5, window)
    assert (got - want).abs().max() < 1e-5
    assert (got - one_token).abs().max() < 2e-6


# windows that leave a group of threads no tile, or begin and end inside tiles of both; rows of many tiles; requests
# that meet inside a block
@pytest.mark.parametrize("lens_q,lens_kv,nq,nkv,hd,page,window", [
    ([30], [190], 4, 1, 64, 16, 20), ([70, 3, 50], [500, 67, 300], 4, 2, 128, 16, 130), ([260], [260], 8, 2, 64, 16, 0),
    ([5, 6, 7, 9, 4], [5, 70, 64, 137, 4], 2, 1, 128, 4, 0)])
def test_float_attention_of_tiles_in_two_groups(lens_q, lens_kv, nq, nkv, hd, page, window, monkeypatch):
    from mstar_b200 import ops

    one_token, want, _ = paged_case(lens_q, lens_kv, nq, nkv, hd, page, torch.float32, 7, window)
    monkeypatch.setattr(ops, "paged_attention_generic",
                        functools.partial(ops.paged_attention_generic, entries=len(lens_q)))
    got, want, _ = paged_case(lens_q, lens_kv, nq, nkv, hd, page, torch.float32, 7, window)
    # products of some 8 rounded to 24 bits in the scores, weights that add up to one
    assert (got - want).abs().max() < 4e-6


# one key, a warp's keys and one more, a round of 512 keys and one more, several rounds; groups of one to nine
# heads; a window that begins inside a page
@pytest.mark.parametrize("lens_kv,nq,nkv,hd,page,window", [
    ([1, 65, 64], 8, 2, 64, 16, 0), ([513, 512, 33], 3, 1, 128, 16, 0), ([1300, 7], 9, 1, 64, 8, 0),
    ([700, 40], 4, 4, 128, 64, 37), ([1200], 10, 2, 64, 4, 600)])
def test_float_attention_of_single_tokens(lens_kv, nq, nkv, hd, page, window):
    ones = [1] * len(lens_kv)
    got, want, _ = paged_case(ones, lens_kv, nq, nkv, hd, page, torch.float32, 6, window)
    # products of some 8 rounded to 24 bits in the scores, weights that add up to one
    assert (got - want).abs().max() < 4e-6


def test_float_attention_of_portions_leaves_unseen_values_out():
    """A later token's value that is not finite reaches no earlier token of the same block."""
    from mstar_b200 import ops

    T, hd = 24, 64
    q = rnd(T, hd, seed=1)
    kv = rnd(2, 2, 1, 16, hd, seed=2)
    kv[1, 1, 0, 7] = float("inf")                   # key 23, the last
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    out = torch.empty(T, hd, device=DEV)
    ops.paged_attention_generic(q, hd, out, kv, i32([[0, 1]]), i32([0] * T), i32(list(range(T))), T, 1,
                                1, hd, 16, 0, hd ** -0.5, entries=1)
    assert torch.isfinite(out[:-1]).all() and not torch.isfinite(out[-1]).any()


# a key a token, a tile and one more, a block a tile; heads that fill a block and that don't; no rotated features
@pytest.mark.parametrize("kv,heads,rank,rot", [([1, 33, 32], 5, 64, 16), ([400, 7], 16, 512, 64), ([90], 17, 96, 32),
                                               ([65], 3, 256, 0)])
def test_latent_attention_of_single_tokens(kv, heads, rank, rot):
    """Against double precision; queries whose rows lie off 16 bytes give the same bits."""
    from mstar_b200 import ops

    T, page, D = len(kv), 16, rank + rot
    width = -(-max(kv) // page)
    cache = rnd(T * width, 1, 1, page, D, dtype=torch.bfloat16, seed=1)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    table = torch.randperm(T * width, device=DEV).to(torch.int32).view(T, width)
    q_abs, wide = 0.3 * rnd(T, heads, rank, seed=2), 0.3 * rnd(T, heads, rot + 9, dtype=torch.bfloat16, seed=3)
    run = lambda q_rot: ops.latent_attention(q_abs, q_rot, cache, table, i32(list(range(T))), i32([n - 1 for n in kv]),
                                             heads, rank, rot, page, 0, 0.1, max_keys=max(kv))
    off = wide[:, :, 1:1 + rot]                      # rows of an odd number of elements
    got = run(off.contiguous())
    assert torch.equal(run(off), got)
    for t, n in enumerate(kv):
        rows = cache[table[t].long()].view(-1, D)[:n].double()
        q = torch.cat([q_abs[t].double(), off[t].double()], 1)
        want = torch.softmax(q @ rows.T * 0.1, -1) @ rows[:, :rank]
        # queries in two bfloat16 parts (2^-16), scores of about 2, weights that add up to one, values of up to 5
        assert (got[t].double() - want).abs().max() < 2 ** -16 * 2 * 5


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("where,value", [("q", float("inf")), ("key", float("nan")), ("key", -float("inf")),
                                         ("value", float("inf")), ("value", 3.4e38), ("none", 0.0)])
def test_float_attention_of_portions_keeps_what_is_not_finite(hd, where, value):
    """As the kernel of a block per token has it; the largest floats, whose first part is not finite, too."""
    from mstar_b200 import ops

    T, heads = 150, 2
    q, kv = rnd(T, heads * hd, seed=1), rnd(10, 2, 1, 16, hd, seed=2)
    if where == "q":
        q[70, 3] = value
    elif where != "none":
        kv[4, int(where == "value"), 0, 5, 3] = value            # key 69
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    outs = []
    for entries in (1, T):                                  # (as many entries as tokens: a block per token)
        out = torch.empty(T, heads * hd, device=DEV)
        ops.paged_attention_generic(q, heads * hd, out, kv, i32([list(range(10))]), i32([0] * T), i32(list(range(T))), T,
                                    heads, 1, hd, 16, 0, hd ** -0.5, entries=entries)
        outs.append(out)
    got, want = outs
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
    both = want.isfinite()
    assert both.any(dim=1)[:69].all()
    torch.testing.assert_close(got[both], want[both], rtol=2e-5, atol=2e-6)


@pytest.mark.parametrize("hd,window", [(64, 0), (128, 0), (64, 20)])
@pytest.mark.parametrize("where,value", [("q", float("nan")), ("key", float("inf")), ("value", float("nan")),
                                         ("key", 1e30)])
def test_float_attention_of_portions_keeps_the_bits_of_rows_that_see_finite_numbers(hd, window, where, value):
    """An operand that is not finite (or scores past the largest float) changes the bits of no row that does not see it,
    of its own request or of another in the same block of 64 rows."""
    from mstar_b200 import ops

    lens, heads, page = [21, 40, 30], 2, 16                      # 32 tokens a block: each meets two requests
    T = sum(lens)
    q, kv = rnd(T, heads * hd, seed=1), rnd(9, 2, 1, page, hd, seed=2)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    table = i32([[0, 1, 2], [3, 4, 5], [6, 7, 8]])
    req, pos = [r for r, n in enumerate(lens) for _ in range(n)], [t for n in lens for t in range(n)]

    def run():
        out = torch.empty(T, heads * hd, device=DEV)
        ops.paged_attention_generic(q, heads * hd, out, kv, table, i32(req), i32(pos), T, heads, 1, hd, page, window,
                                    hd ** -0.5, entries=len(lens))
        return out

    want = run()
    at = 12                                                      # of the second request
    if where == "q":
        q[lens[0] + at, 3] = value
    else:
        kv[3, int(where == "value"), 0, at, 3] = value
        if value == 1e30:
            q[lens[0] + at:lens[0] + lens[1], 3::hd] = -1e30     # the rows that see the key
    got = run()
    sees = torch.tensor([r == 1 and (t == at if where == "q" else t >= at and not (window and t >= at + window))
                         for r, t in zip(req, pos)], device=DEV)
    if value == 1e30:
        sees = torch.tensor([r == 1 and t >= at for r, t in zip(req, pos)], device=DEV)     # (their queries changed)
    assert torch.equal(got[~sees], want[~sees])
    if value != 1e30:
        rows = got[sees].view(-1, heads, hd)                     # (a key of plus infinity may have a score of minus infinity)
        assert not torch.isfinite(rows).all() and (where == "key" or not torch.isfinite(rows).all(2).all(1).any())
    else:                                                        # a score of minus infinity: the key has no weight
        assert torch.isfinite(got[sees]).all()


@pytest.mark.parametrize("tokens,width,ff,experts,identity,top,form,on_input", [
    (200, 72, 8, 2, 0, 2, "silu", False),         # k-blocks that end early, one narrow column tile
    (300, 128, 264, 5, 1, 3, "silu", True),       # column tiles that end inside, identity experts
    (129, 264, 136, 3, 0, 1, "relu2", False),
    (771, 136, 136, 3, 0, 1, "silu", True),       # groups of a row tile and a few rows more
    (5000, 264, 520, 3, 0, 1, "silu", False),     # a second round of tiles cut in two
    (4200, 72, 1096, 3, 0, 1, "relu2", True),     # and in four
    (2100, 64, 16, 7, 2, 6, "clamped", False),    # more rows than the sort keeps in registers, top > 4
    (64, 64, 64, 40, 0, 1, "silu", True)])        # experts without rows
def test_grouped_experts_at_the_borders_of_their_tiles(tokens, width, ff, experts, identity, top, form, on_input):
    """The grouped tensor-core experts against the sum in double precision from the same bfloat16
    numbers; the only rounding on the way is that of the hidden units to bfloat16."""
    from mstar_b200 import ops

    gated, clamp = form != "relu2", (1.5, 1.702) if form == "clamped" else None
    x = rnd(tokens, width, dtype=torch.bfloat16, seed=1)
    w_up = rnd(experts * (2 if gated else 1) * ff, width, dtype=torch.bfloat16, seed=2, scale=0.2)
    w_down = rnd(experts * width, ff, dtype=torch.bfloat16, seed=3, scale=0.2)
    add = rnd(tokens, width, dtype=torch.bfloat16, seed=4)
    gate = rnd(tokens, 1, seed=5)
    chosen, weight = ops.route_topk(rnd(tokens, experts + identity, seed=6), top, softmax=True)
    got = ops.experts_grouped(x, w_up, w_down, chosen, weight, experts + identity, ff, on_input, add,
                              gated=gated, real=experts, clamp=clamp, add_gate=gate).double()
    ops.check_error_word(DEV)
    xd, ud, dd, w = x.double(), w_up.double().view(experts, -1, width), w_down.double().view(experts, width, ff), weight.double()
    want = add.double() * torch.sigmoid(gate.double())
    size = want.abs()
    for e in range(experts + identity):
        rows, place = (chosen == e).nonzero(as_tuple=True)
        a = w[rows, place][:, None]
        if e >= experts:
            y = a * xd[rows]
        else:
            h = (xd[rows] * a if on_input else xd[rows]) @ ud[e].T
            if gated:
                g, u = h.chunk(2, dim=1)
                if clamp:
                    g, u = g.clamp(max=clamp[0]), u.clamp(-clamp[0], clamp[0]) + 1
                    h = g * torch.sigmoid(clamp[1] * g) * u
                else:
                    h = g * torch.sigmoid(g) * u
            else:
                h = h.clamp(min=0) ** 2
            b = 1.0 if on_input else a
            y = b * (h @ dd[e].T)
            size[rows] += b * (h.abs() @ dd[e].abs().T)      # what the hidden units' rounding can do
        want[rows] += y
    assert ((got - want).abs() <= 2 ** -8 * (size + want.abs()) + 1e-5).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,inter", [(3, 8), (5, 2056), (2, 12), (70, 4104), (17000, 16)])
def test_gated_products_by_eight_and_one_by_one(dtype, rows, inter):
    """Widths of whole 16-byte pieces and others, zeros and large gates among them."""
    from mstar_b200 import ops

    x = rnd(rows, 2 * inter, dtype=dtype, seed=1, scale=3.0)
    x[0, :4] = torch.tensor([0.0, -200.0, 200.0, -90.0], dtype=dtype, device=DEV)
    g, u = x.double().chunk(2, dim=1)
    clipped = g.clamp(max=2.0)
    for kind, z, want in (("silu", g, g * torch.sigmoid(g) * u),
                          ("clamped_swish", 1.75 * clipped, clipped * torch.sigmoid(1.75 * clipped) * (u.clamp(-2, 2) + 1))):
        got = ops.silu_mul(x, kind=kind, limit=2.0, alpha=1.75).double()
        # half an ulp of a bfloat16 result; in float the exponent's argument z is rounded (half an
        # ulp of z, which the exponential makes a relative error), expf, the sum, the quotient and the
        # product are off by 2 ulp at most each
        off = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -24 * (z.abs() + 16)
        assert ((got - want).abs() <= off * want.abs() + 1e-30).all()
    y = rnd(rows, 2 * inter, dtype=dtype, seed=2)
    gate = rnd(rows, 2, seed=3)
    want = (y.double().view(rows, 2, inter) * torch.sigmoid(gate.double())[:, :, None]).view(rows, -1)
    got = ops.head_gate_mul(y, gate, 2, out_dtype=torch.bfloat16).double()
    assert ((got - want).abs() <= 2.0 ** -8 * want.abs() + 1e-30).all()


@pytest.mark.parametrize("g", [-86.0, -87.5, -88.0, -88.5])
def test_gates_whose_exponential_nears_the_largest_float(g):
    """The denominator 1 + exp(-g) lies around 2^126 and above, the product within bfloat16's range."""
    from mstar_b200 import ops

    x = torch.full((17000, 16), g, dtype=torch.bfloat16, device=DEV)      # (enough for eight columns a thread)
    x[:, 8:] = 2.0 ** 20
    want = g / (1 + torch.tensor(-g, dtype=torch.float64).exp()) * 2.0 ** 20
    got = ops.silu_mul(x).double()
    assert ((got - want).abs() <= 2.0 ** -8 * abs(want)).all()


@pytest.mark.parametrize("lens,heads,kv_heads,dim,vdim", [
    ([70], 2, 1, 32, 8),                    # a piece of 6 tokens at the end, 8 columns
    ([64, 1, 33], 2, 2, 64, 20),            # columns that end inside a block, an entry of one token
    ([100], 1, 1, 256, 16)])
def test_delta_rule_in_pieces_with_decays_per_channel(lens, heads, kv_heads, dim, vdim):
    """Against the recurrence in double precision, with decays from 1 down to numbers whose products
    over a piece underflow, and a state to start from."""
    from mstar_b200 import ops

    T, taps = sum(lens), 2
    q, k = (torch.nn.functional.normalize(rnd(T, kv_heads, dim, seed=s), dim=-1).view(T, -1) for s in (1, 2))
    v, beta = rnd(T, heads * vdim, seed=3), torch.sigmoid(rnd(T, heads, seed=4))
    decay = torch.exp(-torch.exp(4 * rnd(T, heads * dim, seed=5) - 3))
    size = ops.gated_delta_state_size(heads, kv_heads, dim, vdim, taps)
    state = 0.3 * rnd(len(lens), size, seed=6)
    offset = (taps - 1) * (2 * kv_heads * dim + heads * vdim)
    S = state[:, offset:offset + heads * vdim * dim].double().view(-1, heads, vdim, dim).transpose(2, 3).clone()
    starts = [0]
    for n in lens:
        starts.append(starts[-1] + n)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    got = ops.delta_scan(q, k, v, beta, decay, i32(starts), i32(list(range(len(lens)))), state, len(lens), heads,
                         kv_heads, dim, vdim, taps, max_q_len=max(lens)).view(T, heads, vdim)
    ops.check_error_word(DEV)
    per = heads // kv_heads
    qd, kd = (x.double().view(T, kv_heads, dim).repeat_interleave(per, dim=1) for x in (q, k))
    vd, gd, bd = v.double().view(T, heads, vdim), decay.double().view(T, heads, dim), beta.double()
    for e in range(len(lens)):
        for t in range(starts[e], starts[e + 1]):
            S[e] *= gd[t][:, :, None]
            u = bd[t][:, None] * (vd[t] - (kd[t][:, None] @ S[e])[:, 0])
            S[e] += kd[t][:, :, None] * u[:, None]
            want = (qd[t][:, None] @ S[e])[:, 0]
            # sums of dim products of numbers of about 1, once a token, over at most 16 tokens' corrections
            assert (got[t].double() - want).abs().max() < 2 ** -24 * 64 * dim ** 0.5
    end = state[:, offset:offset + heads * vdim * dim].double().view(-1, heads, vdim, dim).transpose(2, 3)
    assert (end - S).abs().max() < 2 ** -24 * 64 * dim ** 0.5


@pytest.mark.parametrize("head_decay", [False, True])
@pytest.mark.parametrize("dim,vdim", [(32, 32), (64, 48), (128, 128), (256, 64)])
def test_delta_rule_in_pieces_rounds_to_nearest(dim, vdim, head_decay):
    """Under decays that leave a few tokens in the state, its errors favour neither side (sums that are
    cut off come out 2^-25 of themselves too small)."""
    from mstar_b200 import ops

    T, heads = 64, 2
    q, k = (torch.nn.functional.normalize(rnd(T, heads, dim, seed=s), dim=-1).view(T, -1) for s in (1, 2))
    v, beta = rnd(T, heads * vdim, seed=3), torch.sigmoid(rnd(T, heads, seed=4))
    decay = torch.exp(-torch.exp(2 * rnd(T, heads * (1 if head_decay else dim), seed=5)))
    state = torch.zeros(1, ops.gated_delta_state_size(heads, heads, dim, vdim, 1), device=DEV)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    ops.delta_scan(q, k, v, beta, decay, i32([0, T]), i32([0]), state, 1, heads, heads, dim, vdim, 1, max_q_len=T)
    kd, gd = k.double().view(T, heads, dim), decay.double().view(T, heads, -1)
    S = torch.zeros(heads, dim, vdim, dtype=torch.float64, device=DEV)
    for t in range(T):
        S *= gd[t][:, :, None]
        u = beta[t].double()[:, None] * (v[t].double().view(heads, vdim) - (kd[t][:, None] @ S)[:, 0])
        S += kd[t][:, :, None] * u[:, None]
    far = (state.view(heads, vdim, dim).transpose(1, 2).double() - S) / S
    far = far[S.abs() > S.abs().mean() / 8]
    # a column of the last token's u is off by 2^-24 at most either way: 2^-24 / sqrt(heads * vdim) in the mean,
    # times a margin of 2
    assert far.mean().abs() < 2 ** -23 / (heads * vdim) ** 0.5


@pytest.mark.parametrize("head_decay", [False, True])
@pytest.mark.parametrize("heads,dim,vdim", [(1, 32, 8), (2, 128, 40), (80, 64, 32)])     # 8 and 16 columns a block
def test_delta_rule_in_pieces_leaves_later_values_out(head_decay, heads, dim, vdim):
    """A value that is not finite reaches no earlier token's output, wherever it lies in its piece."""
    from mstar_b200 import ops

    T, taps = 70, 2
    q, k = (torch.nn.functional.normalize(rnd(T, heads, dim, seed=s), dim=-1).view(T, -1) for s in (1, 2))
    v, beta = rnd(T, heads * vdim, seed=3), torch.sigmoid(rnd(T, heads, seed=4))
    decay = torch.sigmoid(rnd(T, heads * (1 if head_decay else dim), seed=5) + 3)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)

    def run(values):
        state = 0.3 * rnd(1, ops.gated_delta_state_size(heads, heads, dim, vdim, taps), seed=6)
        return ops.delta_scan(q, k, values, beta, decay, i32([0, T]), i32([0]), state, 1, heads, heads, dim, vdim, taps,
                              max_q_len=T)

    want = run(v)
    for t in (1, 7, 31, 34, 69):
        bad = v.clone()
        bad[t] = float("inf")
        got = run(bad)
        assert torch.equal(got[:t], want[:t]) and not torch.isfinite(got[t]).any()
    ops.check_error_word(DEV)


@pytest.mark.parametrize("head_decay", [False, True])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_delta_inputs_by_runs_of_tokens(head_decay, dtype):
    """Enough tokens for a warp to take eight in a row, entries that meet inside such a run or are shorter than the
    convolution, no multiple of eight in all: against double precision, and each entry by itself (a token a warp there,
    and an entry that begins a run) with the same bits."""
    from mstar_b200 import ops

    lens, heads, kv_heads, dim, taps = [300, 2, 5, 241, 1], 8, 4, 128, 4
    T, qk, vv = sum(lens), kv_heads * dim, heads * dim
    channels = 2 * qk + vv
    proj = rnd(T, channels + 2 * heads + 8, seed=1)
    w = (0.3 * rnd(channels, taps, seed=2)).to(dtype)
    decays = heads if head_decay else heads * dim
    a_proj = None if head_decay else rnd(T, decays, seed=3)
    bias, rate = rnd(decays, seed=4) - 3, torch.rand(heads, device=DEV) * 15 + 1
    state = rnd(len(lens), ops.gated_delta_state_size(heads, kv_heads, dim, dim, taps), seed=5)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    starts = [sum(lens[:e]) for e in range(len(lens) + 1)]

    def run(first, last, slots):
        rows = slice(starts[first], starts[last])
        req = [e for e in range(last - first) for _ in range(lens[first + e])]
        return ops.delta_prepare(proj[rows], w, None if head_decay else a_proj[rows], bias, rate, i32(req),
                                 i32([s - starts[first] for s in starts[first:last + 1]]), i32(slots), state, heads,
                                 kv_heads, dim, dim, taps, 1e-6)

    got = run(0, len(lens), list(range(len(lens))))
    for e in range(len(lens)):
        alone = run(e, e + 1, [e])
        assert all(torch.equal(x[starts[e]:starts[e + 1]], y) for x, y in zip(got, alone)), e
    past = state[:, :(taps - 1) * channels].double().view(-1, taps - 1, channels)
    x = torch.cat([torch.cat([past[e], proj[starts[e]:starts[e + 1], :channels].double()]).unfold(0, taps, 1)
                   for e in range(len(lens))])
    y = torch.nn.functional.silu((x * w.double()).sum(2))
    unit = lambda z: (z / (z.pow(2).sum(2, keepdim=True) + 1e-6).sqrt()).view(T, -1)
    b = proj[:, channels:channels + heads].double()
    z = proj[:, channels + heads:channels + 2 * heads].double() if head_decay else a_proj.double()
    step = torch.nn.functional.softplus(z + bias.double()).view(T, heads, -1)
    want = (unit(y[:, :qk].view(T, kv_heads, dim)) * dim ** -0.5, unit(y[:, qk:2 * qk].view(T, kv_heads, dim)),
            y[:, 2 * qk:], torch.sigmoid(b), torch.exp(-rate.double()[:, None] * step).view(T, -1))
    for g, v in zip(got, want):
        # four products and a SiLU, each rounded once or twice, of sums of about 1 (exponents of up to some 50)
        assert (g.double() - v).abs().max() < 2 ** -24 * 64


@pytest.mark.parametrize("decay_rank,gate_rank", [(12, 64), (8, 8), (64, 20), (128, 128)])
def test_low_rank_inputs_of_the_delta_rule_are_matrices_of_their_own(decay_rank, gate_rank, monkeypatch):
    """On 16 bytes and without gaps between rows, as the package's own products want them, whatever the ranks are."""
    import types

    from mstar_b200.parts import gated_delta

    part = object.__new__(gated_delta.GatedDelta)
    part.spec = types.SimpleNamespace(head_decay=False, full_gate=False, num_heads=2, v_dim=16, decay_rank=decay_rank,
                                      gate_rank=gate_rank)
    part.runtime = types.SimpleNamespace(dtype=torch.bfloat16)
    part.w_a2, part.w_g2 = rnd(32, decay_rank, dtype=torch.bfloat16), rnd(32, gate_rank, dtype=torch.bfloat16)
    linear, inputs = gated_delta.ops.linear, []
    monkeypatch.setattr(gated_delta.ops, "linear", lambda x, w, **kw: inputs.append(x) or linear(x, w, **kw))
    proj = rnd(9, 101 + decay_rank + gate_rank + 4, seed=2)
    part._decay_and_gate(proj, 101)
    want = proj[:, 101:101 + decay_rank + gate_rank].bfloat16().split([decay_rank, gate_rank], dim=1)
    for got, w in zip(inputs, want):
        assert torch.equal(got, w) and got.is_contiguous() and got.data_ptr() % 16 == 0


@pytest.mark.parametrize("heads,kv_heads,dim,rotary", [(4, 2, 64, 64), (3, 1, 128, 64), (2, 2, 64, 16)])
def test_float_rotation_of_few_and_many_tokens(heads, kv_heads, dim, rotary):
    """63 tokens a pair a thread, 64 by eights: the same bits, in the rows and in the cache."""
    from mstar_b200 import ops

    page, T = 16, 64
    qkv, freq = rnd(T, (heads + 2 * kv_heads) * dim, seed=1), torch.rand(rotary // 2, device=DEV)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    table, pos, cached = i32([list(range(40))]), [5 + 9 * t for t in range(T)], []
    for n in (T, T - 1):
        rows, kv = qkv[:n].clone(), torch.zeros(40, 2, kv_heads, page, dim, device=DEV)
        ops.rope_kv_write(rows, i32(pos[:n]), i32(pos[:n]), i32([0] * n), table, freq, kv, heads, kv_heads, dim, rotary,
                          False, page)
        if n == T:
            kv[pos[-1] // page, :, :, pos[-1] % page] = 0        # the token that the other run leaves out
        cached.append((rows[:T - 1, :heads * dim], kv))
    assert all(torch.equal(x, y) for x, y in zip(*cached)) and cached[0][1].any()


# on both sides of the counts from which rows go a number a thread
@pytest.mark.parametrize("rows,hidden", [(1024, 64), (1025, 64), (1025, 2056), (512, 2056), (513, 2056), (513, 4096)])
def test_rows_by_eights_and_one_by_one(rows, hidden):
    from mstar_b200 import ops

    table, ids = rnd(50, hidden, dtype=torch.bfloat16, seed=1), torch.arange(rows, device=DEV, dtype=torch.int32) % 50
    assert torch.equal(ops.embed_rows(table, ids, scale=0.5), table.float()[ids.long()] * 0.5)
    resid, delta = rnd(50, hidden, seed=2), rnd(50, hidden, dtype=torch.bfloat16, seed=3)
    assert torch.equal(ops.gather_add_rows(resid, delta, ids), (resid + delta.float())[ids.long()])


@pytest.mark.parametrize("temperature,opts", [(0.6, {"top_p": 0.8}), (3.0, {"top_p": 0.95}), (0.05, {"top_p": 0.999}),
                                              (1.0, {"top_p": 1e-6}), (1.5, {"top_k": 3000, "top_p": 0.9}),
                                              (1.0, {"top_k": 700})])
def test_sampling_where_the_threshold_is_hard_to_find(temperature, opts):
    """The kept set and the draw where the first round's bins tell little: equal logits, two values, one logit far
    above the others, a range past the largest float, minus infinities, many logits in a bin, few logits in all."""
    import plain_llama as P
    from mstar_b200 import ops

    vocab = 20011
    x = rnd(8, vocab, seed=3, scale=2.0)
    x[0] = 1.5
    x[1] = (x[1] > 0).float()
    x[2, 77] = 1e30
    x[3, 5], x[3, 6] = 3e38, -3e38
    x[4, ::2] = -float("inf")
    x[5] = 10 + x[5] * 1e-4
    x[6] = torch.round(x[6] * 8) / 8
    seeds, offsets = torch.arange(50, 58, device=DEV), torch.arange(8, device=DEV)
    full = lambda v, dt: torch.full((8,), v, dtype=dt, device=DEV)
    extra = {k: full(v, torch.int32 if k == "top_k" else torch.float32) for k, v in opts.items()}
    got = ops.sample(x, full(temperature, torch.float32), seed=seeds, offset=offsets, **extra).tolist()
    for r, tok in enumerate(got):
        p = P.plain_sampling_distribution(x[r].cpu(), temperature, **opts)
        assert p[tok] > 0, f"row {r}: token {tok} is outside the kept set"
        cdf, u = torch.cumsum(p, 0), P.plain_uniform(50 + r, r)
        assert (cdf[tok - 1].item() if tok else 0.0) - 1e-4 <= u <= cdf[tok].item() + 1e-4, (r, tok, u)


@pytest.mark.parametrize("opts", [{"top_p": 0.9}, {"top_k": 900}])
def test_sampling_of_more_tied_logits_than_a_list_holds(opts):
    """Logits in steps of an eighth over rows of 157 k, at offsets at which their keys take one, two and three rounds."""
    import plain_llama as P
    from mstar_b200 import ops

    vocab = 156940
    x = torch.round(3 * rnd(6, vocab, seed=3) * 8) / 8
    for r, (scale, off) in enumerate(((1, 0), (1, 3000), (1e-3, 1), (1, -40), (1e-6, 1), (64, 0))):
        x[r] = x[r] * scale + off
    seeds, offsets = torch.arange(50, 56, device=DEV), torch.arange(6, device=DEV)
    temperature = torch.tensor([1, 1, 1e-3, 1, 1e-6, 64], device=DEV)
    extra = {k: torch.full((6,), v, dtype=torch.int32 if k == "top_k" else torch.float32, device=DEV) for k, v in opts.items()}
    got = ops.sample(x, temperature, seed=seeds, offset=offsets, **extra).tolist()
    for r, tok in enumerate(got):
        p = P.plain_sampling_distribution(x[r].cpu(), temperature[r].item(), **opts)
        assert p[tok] > 0, f"row {r}: token {tok} is outside the kept set"
        cdf, u = torch.cumsum(p.double(), 0), P.plain_uniform(50 + r, r)
        assert (cdf[tok - 1].item() if tok else 0.0) - 1e-4 <= u <= cdf[tok].item() + 1e-4, (r, tok, u)


def test_delta_rule_in_pieces_with_more_blocks_than_fit():
    """So many blocks an SM (34,816 in all) that a share of its shared memory holds no piece."""
    from mstar_b200 import ops

    entries, heads, dim, taps = 34, 64, 256, 1
    T = 64 + entries - 1
    starts = torch.tensor([0] + list(range(64, T + 1)), dtype=torch.int32, device=DEV)
    q, k = (torch.nn.functional.normalize(rnd(T, dim, seed=s), dim=-1) for s in (1, 2))
    v, beta = rnd(T, heads * dim, seed=3), torch.sigmoid(rnd(T, heads, seed=4))
    decay = torch.sigmoid(rnd(T, heads, seed=5) + 3)
    state = torch.zeros(entries, ops.gated_delta_state_size(heads, 1, dim, dim, taps), device=DEV)
    slots = torch.arange(entries, dtype=torch.int32, device=DEV)
    got = ops.delta_scan(q, k, v, beta, decay, starts, slots, state, entries, heads, 1, dim, dim, taps, max_q_len=64)
    ops.check_error_word(DEV)
    # an entry of one token from an empty state: o = (q . k) beta v
    want = (q * k).sum(1)[64:, None, None] * (beta[:, :, None] * v.view(T, heads, dim))[64:]
    assert (got.view(T, heads, dim)[64:] - want).abs().max() < 2 ** -24 * 64 * dim ** 0.5


# pieces of a given size; then a few tokens (8 at most), whole portions, portions cut by their own length
@pytest.mark.parametrize("lens,inner,piece", [([512, 7, 530], 64, "256"), ([600], 32, "0"), ([513], 96, "16"),
                                              ([1, 8, 2, 1], 64, None), ([9, 1], 32, None), ([192, 191, 1], 64, None)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_selective_scan_of_long_portions(lens, inner, piece, dtype, monkeypatch):
    """The scan for 16 states a channel, whole and in pieces, against the recurrence in double precision."""
    from mstar_b200 import ops

    if piece is not None:
        monkeypatch.setenv("MSTAR_SCAN_PIECE", piece)
    T, rank, N, taps = sum(lens), 4, 16, 3
    xc, xz = rnd(T, inner, dtype=dtype, seed=1), rnd(T, 2 * inner, dtype=dtype, seed=2)
    proj, w_dt = rnd(T, rank + 2 * N, seed=3), rnd(inner, rank, seed=4)
    bias, a, d = rnd(inner, seed=5) - 3, -torch.exp(rnd(inner, N, seed=6)), rnd(inner, seed=7)
    state = rnd(len(lens), ops.selective_scan_state_size(inner, N, taps), seed=8)
    S = state[:, (taps - 1) * inner:].double().view(-1, inner, N).clone()
    window = state[:, :(taps - 1) * inner].view(-1, taps - 1, inner).clone()
    starts = [0]
    for n in lens:
        starts.append(starts[-1] + n)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    got = ops.selective_scan(xc, xz, proj, w_dt, bias, a, d, i32(starts), i32(list(range(len(lens)))), state, len(lens),
                             inner, N, rank, taps, max_q_len=max(lens)).double()
    dt = torch.nn.functional.softplus(proj[:, :rank].double() @ w_dt.double().T + bias.double())
    x, z, p = xc.double(), xz[:, inner:].double(), proj.double()
    want, size = torch.empty_like(got), torch.empty_like(got)
    for e in range(len(lens)):
        for t in range(starts[e], starts[e + 1]):
            S[e] = torch.exp(dt[t][:, None] * a.double()) * S[e] + (dt[t] * x[t])[:, None] * p[t, rank:rank + N]
            want[t] = S[e] @ p[t, rank + N:] + d.double() * x[t]
            size[t] = S[e].abs() @ p[t, rank + N:].abs() + (d.double() * x[t]).abs()
    gate = z * torch.sigmoid(z)
    # a state is a sum of decayed inputs whose exponents are rounded (2^-24 of up to 100) and whose exponentials are
    # off by 2 ulp; the result is rounded to its type
    off = 2.0 ** -8 if dtype == torch.bfloat16 else 0.0
    assert ((got - want * gate).abs() <= off * (want * gate).abs() + 2 ** -17 * size * gate.abs() + 1e-6).all()
    end = state[:, (taps - 1) * inner:].double().view(-1, inner, N)
    assert ((end - S).abs() <= 2 ** -17 * S.abs() + 1e-5).all()
    for e in range(len(lens)):                       # the convolution's window moved on
        seen = torch.cat([window[e], xz[starts[e]:starts[e + 1], :inner].float()])
        assert torch.equal(state[e, :(taps - 1) * inner].view(taps - 1, inner), seen[-(taps - 1):])


# off 1: rows off 16 bytes, the kernel for any number of states, which cuts where the batch's longest is long
@pytest.mark.parametrize("alone,beside,off", [
    (alone, beside, off) for alone, beside in ((600, [4200, 3]), (520, [520] * 9), (2047, [513]), (1024, [1] * 20))
    for off in (0, 1)] + [(1, [9], 0), (5, [300], 0), (150, [700], 0)])
def test_selective_scan_of_a_portion_does_not_depend_on_the_batch(alone, beside, off):
    """A portion's bits by itself and among others: how it is cut follows from its own length."""
    from mstar_b200 import ops

    inner, rank, N, taps = 2048, 4, 16, 4
    lens = beside[:1] + [alone] + beside[1:]
    T, at = sum(lens), lens[0]
    xc, xz = rnd(T, inner, dtype=torch.bfloat16, seed=1), rnd(T, 2 * inner + off, dtype=torch.bfloat16, seed=2)[:, :2 * inner]
    proj, w_dt = rnd(T, rank + 2 * N, seed=3), rnd(inner, rank, seed=4)
    bias, a, d = rnd(inner, seed=5) - 3, -torch.exp(rnd(inner, N, seed=6)), rnd(inner, seed=7)
    state = rnd(len(lens), ops.selective_scan_state_size(inner, N, taps), seed=8)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)

    def run(rows, sizes, slots):
        starts = [0]
        for n in sizes:
            starts.append(starts[-1] + n)
        moved = state.clone()
        y = ops.selective_scan(xc[rows].contiguous(), xz[rows], proj[rows].contiguous(), w_dt, bias, a, d, i32(starts),
                               i32(slots), moved, len(sizes), inner, N, rank, taps, max_q_len=max(sizes))
        return y, moved[1]

    whole, end = run(slice(0, T), lens, list(range(len(lens))))
    one, one_end = run(slice(at, at + alone), [alone], [1])
    assert torch.equal(whole[at:at + alone], one) and torch.equal(end, one_end)


@pytest.mark.parametrize("lens,inner", [([1, 2, 3, 1700, 5, 6], 1032), ([2401], 64), ([3] * 800, 64)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_convolution_of_several_tokens_a_thread(lens, inner, dtype):
    """Portions that begin and end inside a thread's tokens and a number of tokens it does not divide,
    against the convolution in double precision."""
    from mstar_b200 import ops

    T, taps, N = sum(lens), 4, 16
    xz, w, bias = rnd(T, 2 * inner, dtype=dtype, seed=1), rnd(inner, taps, dtype=dtype, seed=2), rnd(inner, dtype=dtype, seed=3)
    state = rnd(len(lens), ops.selective_scan_state_size(inner, N, taps), seed=4)
    starts = [0]
    for n in lens:
        starts.append(starts[-1] + n)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    req = torch.repeat_interleave(torch.arange(len(lens)), torch.tensor(lens)).to(torch.int32).to(DEV)
    got = ops.conv_silu(xz, w, bias, req, i32(starts), i32(list(range(len(lens)))), state, inner, taps,
                        weight_t=w.float().T.contiguous(), bias_f32=bias.float()).double()
    for e in range(len(lens)):
        x = torch.cat([state[e, :(taps - 1) * inner].view(taps - 1, inner), xz[starts[e]:starts[e + 1], :inner].float()]).double()
        y, size = bias.double().expand(lens[e], inner), bias.double().abs().expand(lens[e], inner)
        for k in range(taps):
            y = y + w[:, k].double() * x[k:k + lens[e]]
            size = size + (w[:, k].double() * x[k:k + lens[e]]).abs()
        want = y * torch.sigmoid(y)
        # five float sums whose errors the activation's slope (1.1 at most) passes on, an exponential and a quotient
        # of 2 ulp each, and the result's rounding
        off = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -20
        assert ((got[starts[e]:starts[e + 1]] - want).abs() <= off * want.abs() + 2 ** -21 * size).all()


@pytest.mark.parametrize("rows,hidden", [(2501, 1024), (1101, 2056), (901, 4096), (5001, 264)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("add", [False, True])
def test_norm_of_many_rows_has_the_bits_of_the_norm_of_one(rows, hidden, dtype, add):
    from mstar_b200 import ops

    x, w = rnd(rows, hidden, seed=1), rnd(hidden, dtype=dtype, seed=2)
    delta = rnd(rows, hidden, dtype=dtype, seed=3) if add else None
    whole = x.clone()
    got = ops.add_rmsnorm(whole, delta, w, 1e-6, dtype)
    for r in list(range(0, rows, 97)) + [rows - 1]:
        one = x[r:r + 1].clone()
        y = ops.add_rmsnorm(one, delta[r:r + 1] if add else None, w, 1e-6, dtype)
        assert torch.equal(y[0], got[r]) and torch.equal(one[0], whole[r])


# the last one goes a feature at a time, the others four a lane
@pytest.mark.parametrize("nq,nkv,hd,vd,rot,interleaved,norm,form", [
    (16, 4, 128, 128, 128, False, True, "bias"), (3, 1, 20, 12, 16, False, True, "first"),
    (9, 9, 64, 64, 6, True, False, "plain"), (4, 2, 100, 100, 8, False, True, "keys"),
    (2, 2, 8, 128, 0, False, False, "bias"), (5, 1, 36, 20, 20, False, True, "bias")])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_attention_inputs_by_four_features(nq, nkv, hd, vd, rot, interleaved, norm, form, dtype):
    """Bias, head norm, temperature, rotation and the cache's pages, against double precision."""
    from mstar_b200 import ops

    T, page, pages, eps = 37, 4, 12, 1e-6
    keys = form == "keys"
    qkv = rnd(T, (nq + nkv) * hd + (0 if keys else nkv * vd) + 4, seed=1)
    width = qkv.shape[1] - 4
    bias = rnd(width, seed=2) if form == "bias" else None
    wq, wk = (rnd(hd, seed=3), rnd(hd, seed=4)) if norm else (None, None)
    first = (rnd(T, nkv * vd, seed=5), 0.3) if form == "first" else None
    freq = (10000.0 ** -(torch.arange(rot // 2, dtype=torch.float64) / max(rot // 2, 1))).to(DEV)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    table = torch.randperm(pages, generator=torch.Generator().manual_seed(0)).to(torch.int32).to(DEV)[None]
    at = list(range(2, 2 + T))
    cache = torch.zeros(pages, ops.sink_page_elements(nkv, page, hd, vd), dtype=dtype, device=DEV)
    positions = [1000 + 7 * i for i in range(T)]
    q = ops.sink_prepare(qkv, bias, wq, wk, freq, i32(positions), i32(at), i32([0] * T), table, cache, nq, nkv, hd, vd,
                         rot, page, eps, dtype, value_from_key=keys, interleaved=interleaved, q_temp=(0.1, 64),
                         first_values=first)
    x = qkv[:, :width].double() + (bias.double() if bias is not None else 0.0)
    heads, values = x[:, :(nq + nkv) * hd].view(T, nq + nkv, hd), x[:, (nq + nkv) * hd:].view(T, -1, vd)
    if keys:
        values = heads[:, nq:]
    if first is not None:
        values = 0.3 * first[0].double().view(T, nkv, vd) + 0.7 * values
    if norm:
        heads = heads * torch.rsqrt((heads * heads).mean(-1, keepdim=True) + eps)
        heads = heads * torch.cat([wq.double().expand(nq, hd), wk.double().expand(nkv, hd)])
    pos = torch.tensor(positions, dtype=torch.float64, device=DEV)
    temp = 1 + 0.1 * torch.log(torch.floor((pos + 1) / 64) + 1)
    heads = torch.cat([heads[:, :nq] * temp[:, None, None], heads[:, nq:]], dim=1)
    want, partner = heads.clone(), torch.zeros_like(heads)
    if rot:
        c, s = (f(pos[:, None] * freq)[:, None] for f in (torch.cos, torch.sin))
        lo = slice(0, rot, 2) if interleaved else slice(0, rot // 2)
        hi = slice(1, rot, 2) if interleaved else slice(rot // 2, rot)
        a, b = heads[:, :, lo], heads[:, :, hi]
        want[:, :, lo], want[:, :, hi] = a * c - b * s, b * c + a * s
        partner[:, :, lo], partner[:, :, hi] = b, a
    # a feature and its partner, rounded a few times each on their way, times sines and cosines of angles that are
    # right to 2e-7; and the result's rounding
    off = 2.0 ** -8 if dtype == torch.bfloat16 else 0.0
    bound = off * want.abs() + 2 ** -19 * (heads.abs() + partner.abs()) + 1e-6
    assert ((q.view(T, nq, hd).double() - want[:, :nq]).abs() <= bound[:, :nq]).all()
    for t in range(T):
        row = cache[table[0, at[t] // page]].double()
        k = row[:nkv * page * hd].view(nkv, page, hd)[:, at[t] % page]
        v = row[nkv * page * hd:].view(nkv, page, vd)[:, at[t] % page]
        assert ((k - want[t, nq:]).abs() <= bound[t, nq:]).all()
        assert ((v - values[t]).abs() <= off * values[t].abs() + 2 ** -20 * (values[t].abs() + 4)).all()


# the last two go a feature at a time (sizes; a view that starts off 16 bytes), the others four a thread
@pytest.mark.parametrize("rank,rot,rot_dims,q_rank,heads,qk_dim,interleaved,off", [
    (512, 64, 64, 1024, 16, 128, False, 0), (1024, 8, 8, 2048, 1, 4, True, 0), (20, 12, 8, 1028, 3, 16, True, 0),
    (64, 40, 16, 4, 5, 20, False, 0), (30, 10, 6, 34, 3, 18, False, 0), (64, 16, 16, 64, 2, 16, True, 1)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_latent_cache_fill_by_four_features(rank, rot, rot_dims, q_rank, heads, qk_dim, interleaved, off, dtype):
    """Norms, rotation of the shared key part and of the queries, and the cache's rows, against double precision."""
    from mstar_b200 import ops

    T, page, pages, eps, per = 21, 4, 8, 1e-6, qk_dim + rot
    proj = rnd(T, q_rank + rank + rot + 4, seed=1)[:, off:]
    lat_q, dkv = proj[:, :q_rank], proj[:, q_rank:q_rank + rank + rot]
    q = rnd(T, heads * per, dtype=dtype, seed=2)
    wq, wk = rnd(q_rank, seed=3), rnd(rank, seed=4)
    freq = (10000.0 ** -(torch.arange(rot_dims // 2, dtype=torch.float64) / (rot_dims // 2))).to(DEV)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    table = torch.randperm(pages, generator=torch.Generator().manual_seed(0)).to(torch.int32).to(DEV)[None]
    cache = torch.zeros(pages, 1, 1, page, rank + rot, dtype=dtype, device=DEV)
    positions = [5000 + 3 * i for i in range(T)]
    rotated = q.clone()
    got = ops.latent_fill(rotated, dkv, wk, freq, i32(positions), i32(list(range(3, 3 + T))), i32([0] * T), table, cache,
                          heads, qk_dim, rot, rot_dims, rank, page, eps, interleaved=interleaved, q_latent=lat_q,
                          q_latent_weight=wq)
    angle = torch.tensor(positions, dtype=torch.float64, device=DEV)[:, None] * freq

    def turned(x):
        """[T, heads, rot], and the size of what its terms were"""
        lo = slice(0, rot_dims, 2) if interleaved else slice(0, rot_dims // 2)
        hi = slice(1, rot_dims, 2) if interleaved else slice(rot_dims // 2, rot_dims)
        y, size, c, s = x.clone(), x.abs(), torch.cos(angle)[:, None], torch.sin(angle)[:, None]
        y[:, :, lo], y[:, :, hi] = x[:, :, lo] * c - x[:, :, hi] * s, x[:, :, hi] * c + x[:, :, lo] * s
        size[:, :, lo] = size[:, :, hi] = x[:, :, lo].abs() + x[:, :, hi].abs()
        return y, size

    # sums of squares and products of some four roundings each; and the result's rounding
    end = 2.0 ** -8 if dtype == torch.bfloat16 else 0.0
    close = lambda y, want, size: ((y.double() - want).abs() <= end * want.abs() + 2 ** -20 * size + 1e-9).all()
    over = lambda x: x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)
    want = over(lat_q.double()) * wq.double()
    assert close(got, want, want.abs())
    x = q.double().view(T, heads, per)
    y, size = turned(x[:, :, qk_dim:])
    assert close(rotated.view(T, heads, per)[:, :, qk_dim:], y, size)
    assert torch.equal(rotated.view(T, heads, per)[:, :, :qk_dim], q.view(T, heads, per)[:, :, :qk_dim])
    lat = over(dkv[:, :rank].double()) * wk.double()
    key, size = turned(dkv[:, None, rank:].double())
    for t in range(T):
        row = cache[table[0, (3 + t) // page], 0, 0, (3 + t) % page]
        assert close(row[:rank], lat[t], lat[t].abs()) and close(row[rank:], key[t, 0], size[t, 0])


@pytest.mark.parametrize("kind", ["spread", "crowded", "equal", "masked"])
@pytest.mark.parametrize("opts", [dict(top_p=0.7), dict(top_k=700), dict(top_k=400, top_p=0.6), dict(top_k=5, top_p=0.99)])
def test_sampling_thresholds_by_a_list_and_by_rounds(kind, opts):
    """Few logits in the first round's bin (their list decides) and many (further rounds): a crowd beside one
    far-off logit, ties, and rows of which little is left."""
    import plain_llama as P
    from test_gpu_kernels import draw

    vocab, rows = 20003, 24
    logits = rnd(1, vocab, seed=31, scale=2.0)
    if kind == "crowded":
        logits[0, 7] = -4000.0
    elif kind == "equal":
        logits[:] = 1.25
    elif kind == "masked":
        logits[0, torch.arange(vocab, device=DEV) % 61 != 0] = -float("inf")
    seeds, offsets = [17] * rows, list(range(rows))
    got = draw(logits.repeat(rows, 1).contiguous(), 0.8, seeds, offsets, **opts).tolist()
    p = P.plain_sampling_distribution(logits[0].cpu(), 0.8, **opts)
    cdf = torch.cumsum(p.double(), 0)
    for r, tok in enumerate(got):
        assert p[tok] > 0, f"row {r}: token {tok} is outside the kept set"
        u = P.plain_uniform(seeds[r], offsets[r])
        assert (cdf[tok - 1].item() if tok else 0.0) - 3e-4 <= u <= cdf[tok].item() + 3e-4, (r, tok, u)
