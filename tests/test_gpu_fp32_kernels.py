"""The 32-bit path's products at the edges of their tiles, ranges, groups and splits.

They promise the same bits for a row however the work is cut; the values are checked against float64."""

import math

import pytest
import torch

from test_gpu_kernels import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, k", [(1, 4), (31, 32), (33, 36), (64, 1024), (65, 1028), (257, 2560), (100, 4100), (70, 9728), (33, 8200), (5, 37)])
def test_f32_product_has_the_same_bits_in_every_batch(n, k):
    """Up to 2, 4, 8 and 16 tokens, tiles of 32 and of 64, split over blocks or not, K that TMA takes or not (37)."""
    gen = torch.Generator().manual_seed(n * 10007 + k)
    tokens = 257
    a, w = torch.randn(tokens, k, generator=gen).cuda(), torch.randn(n, k, generator=gen).cuda()
    full = torch.empty(tokens, n, device="cuda")
    ops().gemm_simt(a, w, full)
    # a chain of at most k / 4 + 32 multiply-adds, then 3 + 7 sums, each rounded to 2^-24 of the partial sum's bound
    bound = (k / 4 + 44) * 2.0 ** -24 * (a.abs().double() @ w.abs().double().T)
    assert ((full.double() - a.double() @ w.double().T).abs() <= bound).all()
    for lo, hi in ((0, 1), (3, 5), (5, 8), (8, 12), (0, 8), (7, 16), (1, 17), (0, 17), (40, 73), (0, 64), (100, 165), (56, 256)):
        part = torch.empty(hi - lo, n, device="cuda")
        ops().gemm_simt(a[lo:hi], w, part)
        assert torch.equal(part, full[lo:hi]), (lo, hi)
