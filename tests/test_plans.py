"""Launch plans that are plain functions of sizes (no device needed)."""

import pytest
import torch

from layover_b200 import ops
from layover_b200.cache import CacheManager
from layover_b200.engine.batch import BatchBuilder, BatchCapacity, StepEntry
from layover_b200.parts.base import PagedKVNeed

SMS = 148


def test_decode_plan_for_equal_lengths_keeps_the_measured_choices():
    plan = lambda seqs, ctx: ops.decode_plan(seqs, 32, 8, 128, ctx, SMS)
    assert plan(1, 3072) == (16, 3)            # one sequence: a cluster of 16, every block on an SM of its own
    assert plan(2, 3072) == (8, 3)
    assert plan(8, 3072) == (4, 3)
    assert plan(16, 3072) == (2, 3)
    assert plan(32, 3072) == (1, 3)
    assert plan(64, 3072) == (4, 2)            # more blocks than two an SM hold: three slower ones an SM
    assert plan(1, 32768)[0] > 16              # a long lone sequence: more splits, merged through scratch memory
    assert ops.decode_plan(8, 32, 8, 64, 3072, SMS)[1] == 3      # other head sizes have the three-stage kernel only


def test_decode_plan_cuts_further_when_the_longest_sequence_stands_out():
    plan = lambda seqs, ctx, mean: ops.decode_plan(seqs, 32, 8, 128, ctx, SMS, mean)
    # a mean close to the longest changes nothing
    assert plan(32, 8192, 7000) == ops.decode_plan(32, 32, 8, 128, 8192, SMS)
    assert plan(8, 8192, 4096) == (8, 2)
    assert plan(8, 3072, 1500) == (4, 3)       # at least 12 tiles a block, and two blocks an SM still hold them
    assert plan(16, 3072, 1500) == (4, 2)
    assert plan(16, 8192, 4096) == (8, 2)
    assert plan(32, 8192, 4096) == (4, 2)
    assert plan(32, 3072, 1500) == (4, 2)
    # few blocks (one round anyway) and very many (already cut for three blocks an SM) keep their plans
    assert plan(2, 8192, 3000) == ops.decode_plan(2, 32, 8, 128, 8192, SMS)
    assert plan(128, 8192, 3000) == ops.decode_plan(128, 32, 8, 128, 8192, SMS)
    # groups of more than 8 heads have no two-stage variant
    assert ops.decode_plan(16, 64, 4, 128, 8192, SMS, 3000) == ops.decode_plan(16, 64, 4, 128, 8192, SMS)
    for seqs in range(1, 200, 7):
        for ctx in (130, 1000, 5000, 70000):
            splits, stages = plan(seqs, ctx, ctx // 3)
            assert splits >= 1 and stages in (2, 3)


def test_decode_plan_for_unequal_lengths_cuts_at_least_as_far_as_for_equal_ones():
    for seqs in range(5, 16):
        for ctx in range(256, 3072, 128):
            equal = ops.decode_plan(seqs, 32, 8, 128, ctx, SMS)
            assert ops.decode_plan(seqs, 32, 8, 128, ctx, SMS, ctx // 2)[0] >= equal[0]
    assert ops.decode_plan(8, 32, 8, 128, 2400, SMS, 1300) == (4, 3)


def test_tensors_of_another_device_are_refused_before_the_device_is_asked_about():
    a, w, out = torch.zeros(4, 64), torch.zeros(32, 64), torch.zeros(4, 32)
    with pytest.raises(ops.KernelError):
        ops.gemm_simt(a, w, out)
    ints = lambda *values: torch.tensor(values, dtype=torch.int32)
    q, pool, out = torch.zeros(1, 128), torch.zeros(4, 1, 16, 64), torch.zeros(1, 128)
    with pytest.raises(ops.KernelError):
        ops.attention_simt(q, pool, pool, out, ints(0, 1, 2)[None], ints(0, 1), ints(40), ints(0), ints(0), 1, 2, 1, 64, 16, 0.125, max_ctx=40)


class _Recorder:
    """`ops.attention_bf16` for a step of (tokens before, new tokens) requests on the CPU: which kernels it would launch, and how."""

    def __init__(self, monkeypatch, q_heads=32, kv_heads=8):
        self.heads, self.calls = (q_heads, kv_heads), []
        monkeypatch.setattr(ops, "gemm_scratch", lambda device: (None, None, SMS))
        monkeypatch.setattr(ops, "sm_count", lambda device: SMS)
        monkeypatch.setattr(ops, "attention_mma_block_queries", lambda: 64)
        names = ("q", "pool", "layer", "out", "table", "cu_q", "ctx_len", "tile_seq", "tile_q0", "n_tiles", "q_heads", "kv_heads", "dim", "page",
                 "scale", "window", "splits", "exact_weights")
        monkeypatch.setattr(ops, "attention_tcgen05_prefill", lambda *a: self.calls.append(("tcgen05", dict(zip(names, a)))))
        monkeypatch.setattr(ops, "attention_prefill_bf16", lambda *a, **k: self.calls.append(("mma", k)))
        monkeypatch.setattr(ops, "attention_decode_bf16", lambda *a, **k: self.calls.append(("decode", k)))

    def run(self, requests, capacity=None, **options):
        q_heads, kv_heads = self.heads
        cache = CacheManager([(0, PagedKVNeed(kv_heads, 128, None), None)], 4096, 16, torch.bfloat16, "meta", 64)
        entries = []
        for i, (held, new) in enumerate(requests):
            seq = cache.open(str(i))
            cache.grow(seq, held + new)
            cache.commit(seq, held)
            entries.append(StepEntry(seq, [0] * new, []))
        batch = BatchBuilder(cache, torch.device("cpu"), (64, 128)).build(entries, capacity)
        q = torch.empty(batch.n_tokens, q_heads * 128, dtype=torch.bfloat16)
        self.calls.clear()
        ops.attention_bf16(q, cache.view(0), torch.empty_like(q), batch.groups[0].block_table, batch, q_heads, kv_heads, 128, 16, 128 ** -0.5,
                           options.pop("window", 0), **options)
        return self.calls


def test_a_portions_split_is_planned_from_the_portions_own_contexts(monkeypatch):
    """What other requests of the step hold changes nothing: not the launches of a portion, and not its rounding."""
    step = _Recorder(monkeypatch)
    split = lambda requests: next(call["splits"] for name, call in step.run(requests) if name == "tcgen05")
    for portion in ((0, 64), (0, 256), (0, 512), (1000, 128), (8209, 512)):
        alone = split([portion])
        for decoding in ((200, 1), (4000, 1), (8192, 1)):
            assert split([portion, decoding]) == alone and split([decoding, portion, decoding]) == alone
    assert split([(0, 64), (8192, 1)]) == 1 and split([(8209, 512)]) > 1
    assert split([(0, 64), (3000, 64), (8192, 1)]) == split([(3000, 64), (0, 64)])     # the longest of the portions counts


def test_scan_plan_takes_products_where_their_tiles_are_full():
    plan = lambda q_lens, heads=32, dim=128, vdim=128, dtype=torch.bfloat16: ops.scan_plan(q_lens, heads, dim, vdim, dtype)
    assert plan([1500]) == (64, 24, True) and plan([300]) == (64, 5, True)
    assert plan([255]) == (0, 0, False) and plan([1] * 64) == (0, 0, False)
    assert plan([1500], vdim=64) == (128, 12, False) and plan([1500], dim=64, vdim=64) == (128, 12, False)
    assert plan([1500], vdim=96) == (128, 12, False) and plan([1500], dim=96)[2] and plan([1500], dim=256) == (128, 12, False)
    assert plan([600], heads=4) == (128, 5, False) and plan([4000], heads=4)[2]             # few chains: the walk is not waited for
    assert plan([1500] + [1] * 4)[2] and not plan([1500] + [1] * 16)[2]                     # segments of one token
    f32 = torch.float32
    assert plan([1500], dtype=f32)[2] and not plan([1500] + [1] * 4, dtype=f32)[2]
    assert not plan([4000], dtype=f32)[2]                                                   # the states leave the L2
    assert plan([256] * 300, heads=64, vdim=1024)[0] > 64                                   # scratch of 1 GiB at most


def test_scan_form_of_a_call_is_that_of_its_plan():
    for heads, dim, vdim in ((32, 128, 128), (4, 128, 128), (16, 96, 160), (8, 64, 64), (2, 128, 512)):
        for dtype in (torch.float32, torch.bfloat16):
            for q_lens in ([256], [300], [1500], [4000], [300] + [1] * 9, [700, 900], [600] * 4, [20, 260, 7]):
                tokens, segments, products = ops.scan_plan(q_lens, heads, dim, vdim, dtype)
                if products:
                    assert ops.scan_as_products(sum(q_lens), segments, tokens, heads, dim, vdim, dtype)


def test_exact_weights_stay_on_mma_sync_for_short_portions(monkeypatch):
    step = _Recorder(monkeypatch, 16, 4)
    kernel = lambda requests, **options: step.run(requests, exact_weights=True, **options)[-1][0]
    assert kernel([(0, 20)]) == kernel([(0, 261)]) == kernel([(500, 40)]) == "mma"
    assert kernel([(0, 611), (0, 611)]) == kernel([(0, 1500)]) == kernel([(3000, 64)]) == "tcgen05"
    assert kernel([(0, 64), (8000, 1)]) == "mma"                     # what a decoding request holds is nothing to the portion
    assert kernel([(0, 128)] * 16) == "tcgen05"                      # many short prompts fill the SMs
    assert kernel([(0, 1500)], window=1024) == "tcgen05" and kernel([(2000, 100)], window=128) == "mma"
    assert kernel([(0, 1500)], chunk=1024) == "tcgen05" and kernel([(8000, 8)], chunk=4096) == "tcgen05"


def test_captured_portion_with_exact_weights_is_planned_for_its_class(monkeypatch):
    step = _Recorder(monkeypatch, 16, 4)
    run = lambda tokens, width: step.run([], BatchCapacity(1, width, tokens), exact_weights=True)[-1][0]
    assert run(512, 64) == run(64, 256) == "tcgen05" and run(16, 8) == "mma"


def test_portion_splits_weigh_what_a_split_takes():
    plan = lambda *lens, heads=(32, 8), window=0: ops.portion_splits(lens, *heads, window, SMS)
    assert plan((512, 8721)) == 2 and plan((512, 8512), heads=(16, 4)) == 4            # one round of blocks
    assert plan((512, 512)) == plan((1280, 2280)) == plan((2048, 4096)) == 1           # partial results that cost more than they bring
    assert plan((1280, 16280)) in (3, 4) and plan((512, 1512)) == 1
    assert plan((512, 30512), heads=(64, 8)) == 1 and plan((1024, 30000), heads=(64, 8)) == 1
    assert plan((8, 8008)) == 8 and plan((1, 100)) == 1
    assert plan((64, 16000), heads=(12, 4)) == 1                                       # an odd number of heads a group
    assert plan((64, 16000), window=256) == 1 and plan((64, 16000), window=8192) > 1   # the keys that are seen count
    for new in (1, 40, 128, 300, 700, 1500):
        for ctx in (new, new + 900, new + 20000, new + 120000):
            for heads in ((2, 1), (32, 8), (64, 8)):
                for count in (1, 3, 9):
                    splits = plan(*[(new, ctx)] * count, heads=heads)
                    tiles = count * -(-new // 128)
                    assert 1 <= splits <= 8 and (splits == 1 or tiles * heads[0] * splits * 128 * 130 <= 32 << 20)


@pytest.mark.parametrize("new, context, splits", [(128, 768, 1), (128, 897, 1), (128, 1024, 1), (256, 1400, 1), (256, 2600, 3), (512, 2100, 1),
                                                  (512, 2200, 2), (777, 12100, 1), (5, 827, 3), (2, 749, 3)])
def test_a_portion_keeps_its_number_of_blocks(new, context, splits):
    """How many blocks share a row's keys decides how its outputs are rounded."""
    assert ops.portion_splits(((new, context),), 32, 8, 0, SMS) == splits


@pytest.mark.parametrize("window", [0, 1024, -1024])
@pytest.mark.parametrize("heads", [16, 32])
def test_prompts_with_exact_weights_keep_their_kernel(window, heads):
    """The two kernels add a row's keys in tiles of different sizes and round differently."""
    kernel = lambda new: ops.exact_on_tcgen05(((new, new),), heads, window, SMS)
    assert not any(kernel(new) for new in (65, 97, 261, 320, 396, 404, 435)) and all(kernel(new) for new in (321, 371, 384, 512, 611, 1500))
