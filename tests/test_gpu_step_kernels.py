"""Kernels of whole steps at the edges of their tiles, groups, segments and splits, against float64."""

import math

import pytest
import torch

from test_gpu_kernels import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 7, 16])
@pytest.mark.parametrize("inter, k", [(64, 512), (64, 4096), (74 * 64, 520), (75 * 64, 512), (19 * 64, 1000)])
def test_few_token_gated_product_split_over_a_cluster(m, inter, k):
    """One tile, the most that are split and one more, K that does not divide among the splits."""
    o, gen = ops(), torch.Generator().manual_seed(inter + k)
    a = torch.randn(m, k, generator=gen).to(torch.bfloat16).cuda()
    gate, up = ((torch.randn(inter, k, generator=gen) / math.sqrt(k)).to(torch.bfloat16).cuda() for _ in range(2))
    for epilogue, options in (("swiglu", {}), ("clipped_swiglu", {"limit": 1.0, "slope": 1.7})):
        out = torch.full((m, inter), float("nan"), dtype=torch.bfloat16, device="cuda")
        o.gemm_tcgen05(a, o.interleave_gate_up(gate, up), out, epilogue=epilogue, **options)
        assert o.gemm_status() == 0
        g, u = a.double() @ gate.double().T, a.double() @ up.double().T
        if epilogue == "swiglu":
            want = torch.nn.functional.silu(g) * u
        else:
            g, u = g.clamp(max=1.0), u.clamp(-1.0, 1.0)
            want = g * torch.sigmoid(1.7 * g) * (u + 1)
        # gate, up, activation and product each round to bfloat16 where the value is below 8
        assert ((out.double() - want).abs() <= 4 * 2.0 ** -8 * (want.abs() + u.abs() + 0.1)).all()
