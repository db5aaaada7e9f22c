"""The 32-bit path's products and attention at the edges of their tiles, ranges, groups and splits.

Both promise the same bits for a row however the work is cut; the values are checked against float64."""

import math

import pytest
import torch

from test_gpu_kernels import ops, paged_setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, k", [(1, 4), (31, 32), (33, 36), (64, 1024), (65, 1028), (257, 2560), (100, 4100), (70, 9728), (33, 8200), (5, 37)])
def test_f32_product_has_the_same_bits_in_every_batch(n, k):
    """Up to 2, 4, 8 and 16 tokens, tiles of 32 and of 64, every group of ranges a block of its own, K that TMA takes or not (37)."""
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


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("q_heads, kv_heads, dim, vdim", [(4, 1, 16, 16), (4, 2, 128, 128), (6, 2, 64, 132), (9, 1, 28, 256), (5, 1, 300, 260)])
@pytest.mark.parametrize("mask", [{}, {"window": 100}, {"window": 40, "keep_first": 5}, {"chunk": 96}])
def test_f32_attention_split_over_blocks_has_the_bits_of_one_block(dtype, q_heads, kv_heads, dim, vdim, mask):
    """Contexts at the edges of a tile of 32 and a chunk of 128 keys; decoded tokens alone, and beside portions."""
    o, page = ops(), 16
    for lengths, q_lens in (([1, 127, 128, 129, 700], [1] * 5), ([31, 300, 260, 513], [31, 1, 40, 2])):
        k_pool, _, table, ks, _ = paged_setup(dtype, lengths, kv_heads, dim, page, 5)
        _, v_pool, _, _, vs = paged_setup(dtype, lengths, kv_heads, vdim, page, 5)      # the same pages, from the same seed
        tokens = sum(q_lens)
        gen = torch.Generator().manual_seed(6)
        q = torch.randn(tokens, q_heads * dim, generator=gen).to(dtype).cuda()
        starts = [sum(q_lens[:s]) for s in range(len(q_lens) + 1)]
        bq = o.attention_simt_block_queries()
        tiles = [(s, q0) for s, n in enumerate(q_lens) for q0 in range(0, n, bq)]
        ints = lambda values: torch.tensor(values, dtype=torch.int32, device="cuda")
        tile_seq, tile_q0 = ints([t[0] for t in tiles]), ints([t[1] for t in tiles])
        outs = []
        for hints in ({}, {"max_q_len": max(q_lens)}, {"max_q_len": max(q_lens), "max_ctx": max(lengths)}, {"max_ctx": 200}):
            out = torch.full((tokens, q_heads * vdim), float("nan"), dtype=dtype, device="cuda")
            o.attention_simt(q, k_pool, v_pool, out, table, ints(starts), ints(lengths), tile_seq, tile_q0, len(tiles), q_heads, kv_heads,
                             dim, page, dim ** -0.5, vdim=vdim, **mask, **hints)
            outs.append(out)
        assert all(torch.equal(outs[0], other) for other in outs[1:])
        for s, (length, n) in enumerate(zip(lengths, q_lens)):
            i, j = torch.arange(length - n, length)[:, None], torch.arange(length)[None]
            seen = j <= i
            if "window" in mask:
                seen &= (i - j < mask["window"]) | (j < mask.get("keep_first", 0))
            if "chunk" in mask:
                seen &= i // mask["chunk"] == j // mask["chunk"]
            for h in range(q_heads):
                g = h // (q_heads // kv_heads)
                rows = q[starts[s]: starts[s + 1]].view(n, q_heads, dim)[:, h].double().cpu()
                scores = (rows @ ks[s][:, g].double().T * dim ** -0.5).masked_fill(~seen, -math.inf)
                expected = torch.softmax(scores, -1) @ vs[s][:, g].double()
                got = outs[0][starts[s]: starts[s + 1]].view(n, q_heads, vdim)[:, h].double().cpu()
                # scores of dim / 4 + 4 sums of terms below 12 in all, weights and their sums within as much, values below 6
                tolerance = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -24 * (dim / 4 + 16) * 12
                assert ((got - expected).abs() <= 6 * tolerance).all()


@pytest.mark.parametrize("tokens", [1, 4, 16, 40])
def test_f32_product_of_weights_that_the_kernel_before_wrote(tokens):
    """Without `early_weights` the weights may be another kernel's output, in the same stream and a moment ago."""
    o, n, k = ops(), 256, 2048
    gen = torch.Generator().manual_seed(tokens)
    a, first, second = torch.randn(tokens, k, generator=gen).cuda(), *(torch.randn(n, k, generator=gen).cuda() for _ in range(2))
    wants = []
    for w in (first, second):
        wants.append(torch.empty(tokens, n, device="cuda"))
        o.gemm_simt(a, w, wants[-1])
    w, outs = torch.empty_like(first), [torch.empty(tokens, n, device="cuda") for _ in range(40)]
    torch.cuda.synchronize()
    for i, out in enumerate(outs):
        o.lower_rows((first, second)[i % 2], w)
        o.gemm_simt(a, w, out)
    assert all(torch.equal(out, wants[i % 2]) for i, out in enumerate(outs))


@pytest.mark.parametrize("tokens", [1, 2, 3, 4, 5, 16])
@pytest.mark.parametrize("n, k", [(1, 1), (15, 31), (17, 33), (33, 129), (40, 1028), (100, 4100), (16, 8200), (2600, 64), (2049, 512)])
def test_f32_product_of_a_few_tokens_has_the_same_bits_with_and_without_tma(tokens, n, k):
    """Rows that TMA takes and rows that begin one float further; K on both sides of where the streaming kernel takes over."""
    gen = torch.Generator().manual_seed(n * 10007 + k)
    wide_a, wide_w = torch.zeros(40, -(-k // 4) * 4 + 4, device="cuda"), torch.zeros(n, -(-k // 4) * 4 + 4, device="cuda")
    a, w, outs = torch.randn(40, k, generator=gen).cuda(), torch.randn(n, k, generator=gen).cuda(), []
    for shift in (0, 1):
        x, y = wide_a[:, shift: shift + k], wide_w[:, shift: shift + k]
        x.copy_(a); y.copy_(w)
        for rows in (tokens, 40):              # 40: the tiles of many tokens
            outs.append(torch.empty(rows, n, device="cuda"))
            ops().gemm_simt(x[:rows], y, outs[-1])
    assert all(torch.equal(outs[0], out[:tokens]) for out in outs[1:])
    bound = (k / 4 + 44) * 2.0 ** -24 * (a[:tokens].abs().double() @ w.abs().double().T)      # as above
    assert ((outs[0].double() - a[:tokens].double() @ w.double().T).abs() <= bound).all()


@pytest.mark.parametrize("m, n, k", [(1, 70, 9728), (16, 33, 2560), (40, 100, 4100), (600, 2400, 2500), (130, 2560, 9728), (520, 9728, 2500), (513, 19456, 1100)])
def test_f32_product_says_how_much_scratch_its_form_takes(m, n, k):
    """Groups of ranges dealt out one, several or all to a block: the bits of row slices; scratch, and a second launch, only
    where the form that runs has one."""
    o, gen = ops(), torch.Generator().manual_seed(m + n)
    launches = lambda x, out: (lambda before: (o.gemm_simt(x, w, out), o.LAUNCHES - before)[1])(o.LAUNCHES)
    a, w = torch.randn(m, k, generator=gen).cuda(), torch.randn(n, k, generator=gen).cuda()
    full, part, few = torch.empty(m, n, device="cuda"), torch.empty(17, n, device="cuda"), torch.empty(3, n, device="cuda")
    plan = lambda rows, shift=0: o._FUNCTIONS["lb_gemm_simt_scratch"](a.data_ptr() + 4 * shift, w.data_ptr(), rows, n, k, k, k, 148)
    assert launches(a, full) == (2 if plan(m) else 1) and plan(m, 1) == 0
    assert plan(m) <= 64 << 20 and (m > 16 or plan(m) == 0)
    if m >= 17:
        o.gemm_simt(a[m - 17:], w, part)
        assert torch.equal(part, full[m - 17:])
    if m >= 3:
        o.gemm_simt(a[:3], w, few)
        assert torch.equal(few, full[:3])
    rows = slice(0, min(m, 20))
    bound = (k / 4 + 44) * 2.0 ** -24 * (a[rows].abs().double() @ w.abs().double().T)
    assert ((full[rows].double() - a[rows].double() @ w.double().T).abs() <= bound).all()


@pytest.mark.parametrize("m", [1, 7, 16])
def test_f32_product_sums_through_scratch_where_clusters_are_off(m):
    """The form without clusters, asked for through the exported function with scratch of its size: the same bits."""
    import ctypes

    o, n, k = ops(), 100, 9728
    gen = torch.Generator().manual_seed(m)
    a, w = torch.randn(m, k, generator=gen).cuda(), torch.randn(n, k, generator=gen).cuda()
    want, got = torch.empty(m, n, device="cuda"), torch.full((m, n), float("nan"), device="cuda")
    o.gemm_simt(a, w, want)
    scratch = torch.full((8 * m * n,), float("nan"), device="cuda")
    code = o._FUNCTIONS["lb_gemm_simt"](0, 0, a.data_ptr(), w.data_ptr(), got.data_ptr(), m, n, k, k, k, n, scratch.data_ptr(), 148, 0,
                                        torch.cuda.current_stream().cuda_stream)
    assert code == 0 and torch.equal(got, want)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("dim", [16, 128, 300])
def test_f32_attention_of_queries_that_begin_anywhere(dtype, dim):
    """Queries one element off an aligned address give the bits of aligned ones; keys or values there are refused."""
    o, page, q_heads, kv_heads, lengths, q_lens = ops(), 16, 4, 2, [1, 40, 200], [1, 5, 17]
    k_pool, v_pool, table, _, _ = paged_setup(dtype, lengths, kv_heads, dim, page, 5)
    tokens, ints = sum(q_lens), lambda values: torch.tensor(values, dtype=torch.int32, device="cuda")
    q = torch.randn(tokens * q_heads * dim, generator=torch.Generator().manual_seed(2)).to(dtype).cuda()
    tiles = [(s, q0) for s, n in enumerate(q_lens) for q0 in range(0, n, 16)]
    outs = []

    def run(x, k, v):
        out = torch.full((tokens, q_heads * dim), float("nan"), dtype=dtype, device="cuda")
        o.attention_simt(x, k, v, out, table, ints([0, 1, 6, 23]), ints(lengths), ints([t[0] for t in tiles]), ints([t[1] for t in tiles]),
                         len(tiles), q_heads, kv_heads, dim, page, dim ** -0.5)
        return out

    def shifted(t):
        wide = torch.empty(t.numel() + 1, dtype=dtype, device="cuda")[1:]
        return wide.copy_(t.reshape(-1)).view(t.shape)

    q = q.view(tokens, q_heads * dim)
    assert torch.equal(run(q, k_pool, v_pool), run(shifted(q), k_pool, v_pool))
    for k, v in ((shifted(k_pool), v_pool), (k_pool, shifted(v_pool))):
        with pytest.raises(ValueError, match="alignment"):
            run(q, k, v)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("q_heads, kv_heads, dim, vdim", [(40, 2, 16, 16), (32, 1, 128, 128), (12, 1, 64, 200), (12, 1, 300, 512)])
def test_f32_attention_has_the_same_bits_however_many_rows_share_a_warp(monkeypatch, dtype, q_heads, kv_heads, dim, vdim):
    o, page, lengths, q_lens = ops(), 16, [1, 40, 300, 520], [1, 5, 1, 18]
    k_pool, _, table, _, _ = paged_setup(dtype, lengths, kv_heads, dim, page, 5)
    _, v_pool, _, _, _ = paged_setup(dtype, lengths, kv_heads, vdim, page, 5)
    tokens, ints = sum(q_lens), lambda values: torch.tensor(values, dtype=torch.int32, device="cuda")
    q = torch.randn(tokens, q_heads * dim, generator=torch.Generator().manual_seed(2)).to(dtype).cuda()
    tiles = [(s, q0) for s, n in enumerate(q_lens) for q0 in range(0, n, 16)]
    rows_seen, outs, plan = set(), [], o._simt_plan
    for sms in (0, 1 << 20):          # a device with no room and one with room for everything
        def planned(*args):
            splits, room, _, _ = plan(*args)
            rows = o.c_int(0)
            blocks = o._FUNCTIONS["lb_attention_simt_plan"](len(tiles), q_heads, kv_heads, dim, vdim, 18, 5, sms, o.ctypes.addressof(rows))
            rows_seen.add(rows.value)
            return splits, room, blocks, rows.value
        monkeypatch.setattr(o, "_simt_plan", planned)
        for max_ctx in (0, 520):
            out = torch.full((tokens, q_heads * vdim), float("nan"), dtype=dtype, device="cuda")
            o.attention_simt(q, k_pool, v_pool, out, table, ints([0, 1, 6, 7, 25]), ints(lengths), ints([t[0] for t in tiles]),
                             ints([t[1] for t in tiles]), len(tiles), q_heads, kv_heads, dim, page, dim ** -0.5, vdim=vdim, max_q_len=18, max_ctx=max_ctx)
            outs.append(out)
    assert len(rows_seen) == 2 and not torch.isnan(outs[0]).any() and all(torch.equal(outs[0], out) for out in outs[1:])
