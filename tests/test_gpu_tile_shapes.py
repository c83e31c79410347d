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
