"""Kernels of whole steps at the edges of their tiles, groups, segments and splits, against float64."""

import functools
import math

import pytest
import torch

from test_gpu_kernels import ops, paged_setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gated, interleaved", [(True, True), (True, False), (False, False)])
@pytest.mark.parametrize("hidden, inter", [(8, 64), (40, 128), (264, 192), (2048, 64)])
def test_expert_products_on_few_rows(gated, interleaved, hidden, inter):
    """Groups of 0, 1, 7, 8, 9 and 17 places beside 40 idle experts (the tiles are counted 32 experts at a time); channels that
    end within a step of 32, features past the last warp's 16."""
    o, gen = ops(), torch.Generator().manual_seed(hidden + inter)
    groups = [0, 1, 7, 8, 9, 17] + [0] * 40 + [2]
    experts, pairs = len(groups), sum(groups)
    h = torch.randn(pairs, hidden, generator=gen).to(torch.bfloat16).cuda()       # top 1: a pair is a token
    rows = 2 * inter if gated else inter
    w = (torch.randn(experts, rows, hidden, generator=gen) / math.sqrt(hidden)).to(torch.bfloat16).cuda()
    down = (torch.randn(experts, hidden, inter, generator=gen) / math.sqrt(inter)).to(torch.bfloat16).cuda()
    scores = torch.rand(pairs, generator=gen).cuda() if gated else None
    order = torch.randperm(pairs, generator=gen).to(torch.int32).cuda()
    offsets = torch.tensor([sum(groups[:e]) for e in range(experts + 1)], dtype=torch.int32, device="cuda")
    stacked = torch.stack([o.interleave_gate_up(x[:inter], x[inter:]) for x in w]) if interleaved else w
    act = torch.full((pairs, inter), float("nan"), dtype=torch.bfloat16, device="cuda")
    o.moe_expert_up(h, order, offsets, scores, stacked, act, 1, "silu" if gated else "relu2", interleaved, gated)
    y = torch.full((pairs, hidden), float("nan"), device="cuda")
    o.moe_expert_down(act, order, offsets, down, y)
    expert_of = [e for e, n in enumerate(groups) for _ in range(n)]
    for place, e in enumerate(expert_of):
        pair = int(order[place])
        z = w[e].double() @ h[pair].double()
        if gated:
            g, u = float(scores[pair]) * z[:inter], float(scores[pair]) * z[inter:]
            want = torch.nn.functional.silu(g) * u
        else:
            want = torch.relu(z) ** 2
        # sums of `hidden` terms of about 1 / sqrt(hidden), 32-bit: far below the rounding to bfloat16
        assert ((act[place].double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-4).all()
        want = down[e].double() @ act[place].double()
        bound = inter * 2.0 ** -23 * (down[e].double().abs() @ act[place].double().abs())
        assert ((y[pair].double() - want).abs() <= bound + 1e-30).all()


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


@pytest.mark.parametrize("m", [1, 8, 9, 16, 17, 32, 33, 64, 65, 128])
def test_few_token_gated_product_of_whole_tiles(m):
    """Columns that the two halves of a tile compute for one another: none, one, all of a half. SwiGLU: the bits of product and activation."""
    o, gen, inter, k = ops(), torch.Generator().manual_seed(m), 3 * 64, 200
    a = torch.randn(m, k, generator=gen).to(torch.bfloat16).cuda()
    w = (2 * torch.randn(2 * inter, k, generator=gen) / math.sqrt(k)).to(torch.bfloat16).cuda()      # interleaved already
    rows, room = torch.empty(m, 2 * inter, dtype=torch.bfloat16, device="cuda"), torch.full((m + 128, inter), float("nan"), dtype=torch.bfloat16, device="cuda")
    out = room[:m]                              # columns are padded to 16, 32, 64 or 128 tokens: none of the padding is stored
    want = torch.empty_like(out)
    o.gemm_tcgen05(a, w, out, epilogue="swiglu")
    o.gemm_tcgen05(a, w, rows, max_splits=1)
    o.swiglu(rows, want, block=o.SWIGLU_BLOCK)
    assert o.gemm_status() == 0 and torch.equal(out, want) and torch.isnan(room[m:]).all()
    if m <= 16:
        o.gemm_tcgen05(a, w, out.fill_(float("nan")), epilogue="clipped_swiglu", limit=1.0, slope=1.7)
        g, u = (a.double() @ part.double().T for part in w.view(-1, 2, o.SWIGLU_BLOCK, k).transpose(0, 1).reshape(2, inter, k))
        g, u = g.clamp(max=1.0), u.clamp(-1.0, 1.0)
        clipped = g * torch.sigmoid(1.7 * g) * (u + 1)
        # gate, up, activation and product each round to bfloat16 at most, as in the split product's test above
        assert o.gemm_status() == 0
        assert ((out.double() - clipped).abs() <= 4 * 2.0 ** -8 * (clipped.abs() + u.abs() + 0.1)).all()
        assert torch.isnan(room[m:]).all()


@pytest.mark.parametrize("q_heads, kv_heads", [(4, 2), (32, 8)])
@pytest.mark.parametrize("window", [0, 200])
def test_prompt_attention_with_keys_dealt_to_several_blocks(q_heads, kv_heads, window):
    """Fewer key tiles than blocks, whole ranges under the mask, rows that end within a tile."""
    o, dim, page = ops(), 128, 16
    lengths, q_lens = [5, 129, 700, 1300, 513], [5, 129, 130, 1, 512]
    k_pool, v_pool, table, ks, vs = paged_setup(torch.bfloat16, lengths, kv_heads, dim, page, 3)
    pool = torch.stack((k_pool, v_pool))[None].contiguous()
    q = torch.randn(sum(q_lens), q_heads * dim, generator=torch.Generator().manual_seed(4)).to(torch.bfloat16).cuda()
    ints = lambda values: torch.tensor(values, dtype=torch.int32, device="cuda")
    starts = [sum(q_lens[:s]) for s in range(len(q_lens) + 1)]
    tiles = [(s, q0) for s, n in enumerate(q_lens) for q0 in range(0, n, 128)]
    outs = []
    for splits in (1, 2, 3, 8, 32):
        out = torch.full_like(q, float("nan"))
        o.attention_tcgen05_prefill(q, pool, 0, out, table, ints(starts), ints(lengths), ints([t[0] for t in tiles]), ints([t[1] for t in tiles]),
                                    len(tiles), q_heads, kv_heads, dim, page, dim ** -0.5, window, splits)
        assert o.attention_tcgen05_status() == 0
        outs.append(out)
    for s, (length, n) in enumerate(zip(lengths, q_lens)):
        i, j = torch.arange(length - n, length)[:, None], torch.arange(length)[None]
        seen = (j <= i) & ((i - j < window) if window else (j >= 0))
        for h in range(q_heads):
            g = h // (q_heads // kv_heads)
            rows = q[starts[s]: starts[s + 1]].view(n, q_heads, dim)[:, h].double().cpu()
            scores = (rows @ ks[s][:, g].double().T * dim ** -0.5).masked_fill(~seen, -math.inf)
            p = torch.softmax(scores, -1)
            want, spread = p @ vs[s][:, g].double(), p @ vs[s][:, g].double().abs()
            for out in outs:
                got = out[starts[s]: starts[s + 1]].view(n, q_heads, dim)[:, h].double().cpu()
                # weights and output round to bfloat16 (2^-9 of their own each)
                assert ((got - want).abs() <= 2.0 ** -8 * (spread + want.abs()) + 1e-6).all()


@pytest.mark.parametrize("heads, dim, vdim, decay", [(2, 33, 7, [0.9, 0.0]), (1, 64, 130, [1.0]), (3, 128, 128, [0.999, 0.5, 0.97]), (2, 36, 4, [0.3, 0.99])])
@pytest.mark.parametrize("lengths, segment", [([1], 128), ([127, 128, 129], 128), ([300, 2, 256], 128), ([70], 64), ([300, 65, 128], 64), ([513, 100], 256)])
def test_segments_as_matrix_products(heads, dim, vdim, decay, lengths, segment):
    """Segments that end at, before and after blocks of 64 tokens, several sequences, heads whose rows allow four channels at a
    time or not, states that are carried in and out."""
    o, gen = ops(), torch.Generator().manual_seed(dim + sum(lengths))
    tokens, n_seqs = sum(lengths), len(lengths)
    qk, vv = heads * dim, heads * vdim
    proj = torch.randn(tokens, 2 * qk + vv, generator=gen).cuda()
    state = torch.randn(n_seqs + 1, heads, dim, vdim, generator=gen).cuda()
    before, slots = state.double().clone(), list(range(n_seqs, 0, -1))
    starts = [sum(lengths[:s]) for s in range(n_seqs + 1)]
    ints = lambda values: torch.tensor(values, dtype=torch.int32, device="cuda")
    lam = torch.tensor(decay, device="cuda")
    segments = sum(max(1, -(-n // segment)) for n in lengths)
    scratch = torch.full((segments, heads, dim, vdim), float("nan"), device="cuda")
    out = torch.full((tokens, vv), float("nan"), device="cuda")
    o.decay_scan(proj, 0, qk, 2 * qk, out, state, ints(starts), ints(slots), lam, n_seqs, heads, dim, vdim, None, segment, scratch)
    assert torch.equal(state[0].double(), before[0])             # a slot of nobody's
    x = proj.double()
    q, k, v = x[:, :qk].view(-1, heads, dim), x[:, qk: 2 * qk].view(-1, heads, dim), x[:, 2 * qk:].view(-1, heads, vdim)
    for s in range(n_seqs):
        at, largest = before[slots[s]], before[slots[s]].abs()
        for t in range(starts[s], starts[s + 1]):
            at = lam.double()[:, None, None] * at + k[t][:, :, None] * v[t][:, None, :]
            largest = lam.double()[:, None, None] * largest + (k[t][:, :, None] * v[t][:, None, :]).abs()
            want = (q[t][:, :, None] * at).sum(1)
            # every partial sum is below the sum of absolute values; a few hundred roundings of 2^-24, powers of the decay to 2^-21
            bound = 2.0 ** -18 * (q[t].abs()[:, :, None] * largest).sum(1)
            assert ((out[t].view(heads, vdim).double() - want).abs() <= bound + 1e-30).all()
        assert ((state[slots[s]].double() - at).abs() <= 2.0 ** -18 * largest + 1e-30).all()


@pytest.mark.parametrize("flags", [{}, {"neighbours": True}, {"whole_norm": True, "norms": True}, {"norms": True, "blend": 2}, {"values_from_keys": True}])
def test_heads_of_a_projection_row_four_channels_at_a_time(flags):
    """Rows on 16-byte boundaries (four channels a thread) give the bits that rows off them (one a thread) give."""
    o, gen = ops(), torch.Generator().manual_seed(9)
    tokens, q_heads, kv_heads, dim, page, room = 5, 6, 2, 24, 16, 32
    vdim = dim if flags.get("values_from_keys") else 20
    width = q_heads * dim + kv_heads * dim + (0 if flags.get("values_from_keys") else kv_heads * vdim)
    values = torch.randn(tokens, width, generator=gen).cuda()
    bias = {n: torch.randn(s, generator=gen).cuda() for n, s in (("q", q_heads * dim), ("k", kv_heads * dim), ("v", kv_heads * vdim))}
    size = q_heads * dim, kv_heads * dim
    norms = [1 + 0.1 * torch.randn(n if flags.get("whole_norm") else dim, generator=gen).cuda() for n in size] if flags.get("norms") else [None, None]
    table = torch.randn(tokens, 2, 8, generator=gen).cuda()
    slots = torch.tensor([0, 17, 5, 40, 31], dtype=torch.int32, device="cuda")
    kept, lam = torch.randn(tokens, kv_heads * vdim, generator=gen).cuda(), torch.tensor([0.3], device="cuda")
    results = []
    for shift in (0, 1):
        wide = torch.zeros(tokens, width + 4, device="cuda")
        wide[:, shift: shift + width] = values
        proj = wide[:, shift: shift + width]
        q = torch.full((tokens, q_heads * room), float("nan"), dtype=torch.bfloat16, device="cuda")
        k_pool, v_pool = (torch.full((3, kv_heads, page, room), 7.0, dtype=torch.bfloat16, device="cuda") for _ in range(2))
        o.heads_bias_rope_kv(proj, q, k_pool, v_pool, bias["q"], bias["k"], None if flags.get("values_from_keys") else bias["v"], table, slots,
                             kept.clone(), flags.get("blend", 0), lam if flags.get("blend") else None, q_heads, kv_heads, dim, vdim, page, norms[0],
                             norms[1], 1e-6, neighbours=flags.get("neighbours", False), values_from_keys=flags.get("values_from_keys", False),
                             whole_norm=flags.get("whole_norm", False))
        results.append((q, k_pool, v_pool))
    for a, b in zip(*results):
        assert not torch.isnan(a).any() and torch.equal(a, b)


@pytest.mark.parametrize("q_heads, kv_heads", [(2, 1), (12, 2)])
@pytest.mark.parametrize("window", [0, 200, -96, -128, -1000])
@pytest.mark.parametrize("extras", [False, True])
def test_prompt_attention_with_exact_weights(q_heads, kv_heads, window, extras):
    """Windows and chunks (negative) that begin inside, at and beyond a tile of 128 keys; sinks, gates, a factor and output rows
    that are part of wider ones."""
    o, dim, page = ops(), 128, 16
    lengths, q_lens = [5, 129, 700, 1300, 513], [5, 129, 130, 1, 512]
    k_pool, v_pool, table, ks, vs = paged_setup(torch.bfloat16, lengths, kv_heads, dim, page, 3)
    pool = torch.stack((k_pool, v_pool))[None].contiguous()
    gen, tokens = torch.Generator().manual_seed(4), sum(q_lens)
    q = torch.randn(tokens, q_heads * dim, generator=gen).to(torch.bfloat16).cuda()
    sinks = (2 * torch.randn(q_heads, generator=gen)).cuda() if extras else None
    gates = torch.rand(tokens, q_heads, generator=gen).cuda() if extras else None
    factor = 0.7 if extras else 1.0
    ints = lambda values: torch.tensor(values, dtype=torch.int32, device="cuda")
    starts = [sum(q_lens[:s]) for s in range(len(q_lens) + 1)]
    tiles = [(s, q0) for s, n in enumerate(q_lens) for q0 in range(0, n, 128)]
    wide = torch.full((tokens, q_heads * dim + (8 if extras else 0)), float("nan"), dtype=torch.bfloat16, device="cuda")
    out = wide[:, : q_heads * dim]
    o.attention_tcgen05_prefill(q, pool, 0, out, table, ints(starts), ints(lengths), ints([t[0] for t in tiles]), ints([t[1] for t in tiles]),
                                len(tiles), q_heads, kv_heads, dim, page, dim ** -0.5, window, 1, True, sinks, gates, factor)
    assert o.attention_tcgen05_status() == 0 and torch.isnan(wide[:, q_heads * dim:]).all()
    for s, (length, n) in enumerate(zip(lengths, q_lens)):
        i, j = torch.arange(length - n, length)[:, None], torch.arange(length)[None]
        seen = (j <= i) & ((i - j < window) if window > 0 else (i // -window == j // -window) if window else (j >= 0))
        for h in range(q_heads):
            g = h // (q_heads // kv_heads)
            rows = q[starts[s]: starts[s + 1]].view(n, q_heads, dim)[:, h].double().cpu()
            scores = (rows @ ks[s][:, g].double().T * dim ** -0.5).masked_fill(~seen, -math.inf)
            if extras:
                scores = torch.cat((scores, sinks[h].double().cpu().expand(n, 1)), 1)
            p = torch.softmax(scores, -1)[:, :length]
            scale = factor * (gates[starts[s]: starts[s + 1], h, None].double().cpu() if extras else 1.0)
            want, spread = p @ vs[s][:, g].double() * scale, p @ vs[s][:, g].double().abs() * scale
            got = out[starts[s]: starts[s + 1]].view(n, q_heads, dim)[:, h].double().cpu()
            # the output rounds to bfloat16 (2^-9), the weights keep 16 bits (2^-17) and their exponentials' 2^-22
            assert ((got - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -14 * spread + 1e-6).all()


@pytest.mark.parametrize("group, page, splits, stages", [(1, 8, 1, 3), (4, 16, 4, 2), (8, 24, 3, 3), (7, 64, 8, 3), (2, 16, 1, 2)])
@pytest.mark.parametrize("window, keep, extras", [(0, 0, False), (100, 0, False), (70, 30, True), (-96, 0, True)])
@pytest.mark.parametrize("factor", [0.3, 4.0])
def test_decode_attention_with_a_warps_own_keys(group, page, splits, stages, window, keep, extras, factor):
    """Contexts that end at, before and after a warp's 16 keys and a tile's 64; scores that stay within a base and that outgrow it."""
    o, dim, kv_heads = ops(), 128, 2
    lengths = [1, 15, 16, 17, 64, 65, 200, 529, 1281]
    k_pool, v_pool, table, ks, vs = paged_setup(torch.bfloat16, lengths, kv_heads, dim, page, 5)
    gen, n, q_heads = torch.Generator().manual_seed(6), len(lengths), group * kv_heads
    q = (factor * torch.randn(n, q_heads * dim, generator=gen)).to(torch.bfloat16).cuda()
    sinks = torch.randn(q_heads, generator=gen).cuda() if extras else None
    gates = torch.rand(n, q_heads, generator=gen).cuda() if extras else None
    out = torch.full((n, q_heads * dim), float("nan"), dtype=torch.bfloat16, device="cuda")
    ints = lambda values: torch.tensor(values, dtype=torch.int32, device="cuda")
    o.attention_decode_bf16(q, k_pool, v_pool, out, table, ints(list(range(n + 1))), ints(lengths), None, n, q_heads, kv_heads, dim, page,
                            dim ** -0.5, window, splits, stages, sinks=sinks, gates=gates, keep_first=keep)
    for s, length in enumerate(lengths):
        j, i = torch.arange(length), length - 1
        seen = (i - j < window) | (j < keep) if window > 0 else (i // -window == j // -window) if window else (j >= 0)
        for h in range(q_heads):
            g = h // group
            scores = (ks[s][:, g].double() @ q[s].view(q_heads, dim)[h].double().cpu() * dim ** -0.5).masked_fill(~seen, -math.inf)
            if extras:
                scores = torch.cat((scores, sinks[h, None].double().cpu()))
            p = torch.softmax(scores, -1)[:length] * (gates[s, h].double().cpu() if extras else 1.0)
            want, spread = p @ vs[s][:, g].double(), p @ vs[s][:, g].double().abs()
            got = out[s].view(q_heads, dim)[h].double().cpu()
            # the output rounds to bfloat16 (2^-9), a weight to bfloat16 (2^-9) or to 16 bits (2^-17, exponentials 2^-22); scores of
            # up to 60 in 32-bit are off by 2^-18
            assert ((got - want).abs() <= 2.0 ** -8 * want.abs() + (2.0 ** -14 if extras else 2.0 ** -8) * spread + 1e-6).all()


@pytest.mark.parametrize("dim", [24, 64])
@pytest.mark.parametrize("products", [False, True])
@pytest.mark.parametrize("lengths", [[0], [130, 0, 70], [0, 300, 0]])
def test_segments_of_a_sequence_without_tokens_leave_its_state(dim, products, lengths):
    """A decay of 0 to the power 0 is 1: the state of a request that brings no tokens keeps its bits."""
    o, heads, vdim, segment = ops(), 2, 20, 64
    gen, tokens, n_seqs = torch.Generator().manual_seed(dim), sum(lengths), len(lengths)
    proj = torch.randn(tokens, heads * (2 * dim + vdim), generator=gen).cuda()
    state = torch.randn(n_seqs, heads, dim, vdim, generator=gen).cuda()
    before = state.clone()
    ints = lambda values: torch.tensor(values, dtype=torch.int32, device="cuda")
    scratch = torch.full((sum(max(1, -(-n // segment)) for n in lengths), heads, dim, vdim), float("nan"), device="cuda")
    out = torch.full((tokens, heads * vdim), float("nan"), device="cuda")
    o.decay_scan(proj, 0, heads * dim, 2 * heads * dim, out, state, ints([sum(lengths[:s]) for s in range(n_seqs + 1)]), ints(list(range(n_seqs))),
                 torch.tensor([0.0, 0.9], device="cuda"), n_seqs, heads, dim, vdim, None, segment, scratch, products)
    assert not torch.isnan(out).any() and not torch.isnan(state).any()
    for s, n in enumerate(lengths):
        assert torch.equal(state[s], before[s]) == (n == 0)


@pytest.mark.parametrize("dim", [24, 128])
@pytest.mark.parametrize("products", [False, True])
@pytest.mark.parametrize("what", ["k", "v"])
@pytest.mark.parametrize("value", [math.inf, -math.inf, math.nan])
def test_segments_keep_a_value_that_is_not_finite_from_earlier_tokens(dim, products, what, value):
    """The outputs of the tokens before it keep their bits, wherever it stands in a block of 64 tokens; its own is not finite."""
    o, heads, vdim, tokens = ops(), 2, 128, 200
    gen = torch.Generator().manual_seed(dim)
    clean = torch.randn(tokens, heads * (2 * dim + vdim), generator=gen).cuda()
    ints = lambda values: torch.tensor(values, dtype=torch.int32, device="cuda")
    lam = torch.tensor([0.9, 0.99], device="cuda")

    def run(proj):
        state, out = torch.zeros(1, heads, dim, vdim, device="cuda"), torch.empty(tokens, heads * vdim, device="cuda")
        scratch = torch.empty(2, heads, dim, vdim, device="cuda")
        o.decay_scan(proj, 0, heads * dim, 2 * heads * dim, out, state, ints([0, tokens]), ints([0]), lam, 1, heads, dim, vdim, None, 128, scratch, products)
        return out.view(tokens, heads, vdim)

    want, column = run(clean), heads * dim + 5 if what == "k" else 2 * heads * dim + 5
    for at in (1, 2, 30, 63, 64, 66, 127, 128, 131, 199):
        proj = clean.clone()
        proj[at, column] = value
        got = run(proj)
        assert torch.equal(got[:at], want[:at]) and torch.equal(got[:, 1], want[:, 1])
        assert not torch.isfinite(got[at, 0]).all()


def test_segments_with_scratch_that_begins_anywhere():
    """Scratch four bytes off a 16-byte boundary gives the bits that aligned scratch gives."""
    o, heads, dim, vdim, tokens = ops(), 2, 64, 64, 150
    proj = torch.randn(tokens, heads * (2 * dim + vdim), generator=torch.Generator().manual_seed(1)).cuda()
    ints = lambda values: torch.tensor(values, dtype=torch.int32, device="cuda")
    lam, floats, results = torch.tensor([0.9, 0.99], device="cuda"), 3 * heads * dim * vdim, []
    for shift in (0, 1):
        scratch = torch.empty(floats + 1, device="cuda")[shift: shift + floats].view(3, heads, dim, vdim)
        state, out = torch.ones(1, heads, dim, vdim, device="cuda"), torch.empty(tokens, heads * vdim, device="cuda")
        o.decay_scan(proj, 0, heads * dim, 2 * heads * dim, out, state, ints([0, tokens]), ints([0]), lam, 1, heads, dim, vdim, None, 64, scratch, True)
        results.append((out, state))
    assert all(torch.equal(a, b) for a, b in zip(*results))


@pytest.mark.parametrize("products", [False, True])
@pytest.mark.parametrize("heads, dim, vdim, decay", [(2, 33, 7, [0.9, 0.0]), (1, 64, 130, [1.0]), (3, 128, 128, [0.999, 0.5, 0.97]), (2, 5, 4, [0.3, 0.99])])
@pytest.mark.parametrize("lengths, segment", [([1], 128), ([127, 128, 129], 128), ([300, 65, 128], 64), ([513, 100], 256)])
def test_segments_in_both_forms(monkeypatch, products, heads, dim, vdim, decay, lengths, segment):
    """The form asked for, whatever the plan would take: walked token by token or as matrix products."""
    o = ops()
    monkeypatch.setattr(o, "decay_scan", functools.partial(o.decay_scan, products=products))
    test_segments_as_matrix_products(heads, dim, vdim, decay, lengths, segment)


def test_segments_as_products_refuse_heads_that_a_block_does_not_hold():
    o = ops()
    proj, state, out = torch.zeros(300, 3 * 192, device="cuda"), torch.zeros(1, 1, 192, 192, device="cuda"), torch.zeros(300, 192, device="cuda")
    ints = lambda values: torch.tensor(values, dtype=torch.int32, device="cuda")
    scratch = torch.zeros(5, 1, 192, 192, device="cuda")
    with pytest.raises(ValueError):
        o.decay_scan(proj, 0, 192, 384, out, state, ints([0, 300]), ints([0]), torch.ones(1, device="cuda"), 1, 1, 192, 192, None, 64, scratch, True)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("experts, shared", [(7, True), (8, False), (8, True), (15, True), (16, True), (31, True), (32, True), (40, False)])
@pytest.mark.parametrize("hidden", [512, 4096, 1001])
def test_router_gives_a_token_the_same_bits_in_every_batch(dtype, experts, shared, hidden):
    """One, two and four rows of the router a warp: on both sides of where each is taken."""
    o, gen = ops(), torch.Generator().manual_seed(experts + hidden)
    h = torch.randn(70, hidden, generator=gen).to(dtype).cuda()
    router = torch.randn(experts, hidden, generator=gen).cuda() / math.sqrt(hidden)
    gate = torch.randn(hidden, generator=gen).cuda() / math.sqrt(hidden) if shared else None
    results = []
    for tokens in (70, 64, 1):
        ids, scores = torch.empty(tokens, 3, dtype=torch.int32, device="cuda"), torch.empty(tokens, 3, device="cuda")
        factor = torch.empty(tokens, device="cuda") if shared else None
        o.moe_route(h[:tokens], router, 3, ids, scores, gate, factor)
        results.append((ids, scores) + ((factor,) if shared else ()))
    for got in results[1:]:
        assert all(torch.equal(a[: b.shape[0]], b) for a, b in zip(results[0], got))
    chosen = torch.gather(h.double() @ router.double().T, 1, results[0][0].long())
    # a lane's chain of at most hidden / 32 + 8 products and five sums, each off by 2^-24 of the terms' absolute sum; a sigmoid's slope is 1/4
    bound = (hidden / 32 + 13) * 2.0 ** -26 * torch.gather(h.double().abs() @ router.double().abs().T, 1, results[0][0].long()) + 2.0 ** -22
    assert ((results[0][1].double() - torch.sigmoid(chosen)).abs() <= bound).all()


@pytest.mark.parametrize("q_heads, kv_heads", [(4, 2), (3, 1)])
def test_plain_prompt_attention_takes_a_negative_window_as_none(q_heads, kv_heads):
    """A chunked mask is the exact variant's; without it a window that is not positive masks nothing."""
    o, dim, page, lengths, q_lens = ops(), 128, 16, [40, 300], [40, 130]
    k_pool, v_pool, table, _, _ = paged_setup(torch.bfloat16, lengths, kv_heads, dim, page, 3)
    pool = torch.stack((k_pool, v_pool))[None].contiguous()
    q = torch.randn(170, q_heads * dim, generator=torch.Generator().manual_seed(4)).to(torch.bfloat16).cuda()
    ints = lambda values: torch.tensor(values, dtype=torch.int32, device="cuda")
    outs = []
    for window in (0, -64):
        outs.append(torch.full_like(q, float("nan")))
        o.attention_tcgen05_prefill(q, pool, 0, outs[-1], table, ints([0, 40, 170]), ints(lengths), ints([0, 1, 1]), ints([0, 0, 128]), 3,
                                    q_heads, kv_heads, dim, page, dim ** -0.5, window)
    assert not torch.isnan(outs[0]).any() and torch.equal(*outs)


@pytest.mark.parametrize("products", [False, True])
@pytest.mark.parametrize("heads, dim, vdim, decay", [(2, 33, 7, [0.9, 0.0]), (3, 128, 128, [0.999, 0.5, 0.97])])
@pytest.mark.parametrize("lengths, segment", [([512], 64), ([513], 64), ([1024, 70], 64), ([1500], 64), ([1025, 1153], 128)])
def test_segments_that_are_joined_in_several_trips(monkeypatch, products, heads, dim, vdim, decay, lengths, segment):
    """The joining takes eight segments a trip: 8, 9, 10, 16 and 24 of a sequence, a head's size that allows 16 bytes a load and one that
    does not, in both forms (a first segment from the slot, all from zero)."""
    o = ops()
    monkeypatch.setattr(o, "decay_scan", functools.partial(o.decay_scan, products=products))
    test_segments_as_matrix_products(heads, dim, vdim, decay, lengths, segment)


@pytest.mark.parametrize("products", [False, True])
@pytest.mark.parametrize("what", ["scratch", "state"])
def test_joining_of_many_segments_gives_the_same_bits_from_anywhere(products, what):
    """Scratch or states four bytes off a 16-byte boundary, 8, 9 and 17 segments a sequence."""
    o, heads, dim, vdim, lengths, segment = ops(), 2, 64, 64, [512, 1088, 513], 64
    tokens, n_seqs = sum(lengths), len(lengths)
    gen = torch.Generator().manual_seed(2)
    proj, start = torch.randn(tokens, heads * (2 * dim + vdim), generator=gen).cuda(), torch.randn(n_seqs, heads, dim, vdim, generator=gen).cuda()
    ints = lambda values: torch.tensor(values, dtype=torch.int32, device="cuda")
    lam, segments, results = torch.tensor([0.9, 0.999], device="cuda"), sum(-(-n // segment) for n in lengths), []
    room = lambda count, shift: torch.full((count * heads * dim * vdim + 1,), float("nan"), device="cuda")[shift: shift + count * heads * dim * vdim] \
        .view(count, heads, dim, vdim)
    for shift in (0, 1):
        scratch, state = room(segments, shift if what == "scratch" else 0), room(n_seqs, shift if what == "state" else 0).copy_(start)
        out = torch.full((tokens, heads * vdim), float("nan"), device="cuda")
        o.decay_scan(proj, 0, heads * dim, 2 * heads * dim, out, state, ints([sum(lengths[:s]) for s in range(n_seqs + 1)]), ints([2, 0, 1]), lam, n_seqs,
                     heads, dim, vdim, None, segment, scratch, products)
        results.append((out, state))
    assert not any(torch.isnan(x).any() for x in results[0]) and all(torch.equal(a, b) for a, b in zip(*results))
