"""Kernels that cut their work into tiles by size, at the sizes where a tile's edge or a choice
between two shapes lies, against plain double precision."""
import pytest
import torch

from test_gpu_kernels import rnd

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
