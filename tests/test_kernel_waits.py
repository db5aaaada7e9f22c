"""What a kernel does when one of its bounded waits runs out, read from the sources: nothing here lets a GPU wait for what never comes."""

import re

from layover_b200.csrc.build import HERE


def _prompt_attention_of_pairs():
    source = (HERE / "attention_tcgen05.cu").read_text()
    return source[source.index("attention_tcgen05_pair_kernel(const"): source.index("attention_merge_kernel(const")]


def test_prompt_attention_tells_which_wait_ran_out():
    kernel = _prompt_attention_of_pairs()
    codes = [int(code) for code in re.findall(r"g_attn_error, 0, (\d+)|ran_out\((\d+)\)|flag, (\d+), lane", kernel) for code in code if code]
    assert set(codes) == set(range(21, 30))


def test_prompt_attention_announces_nothing_of_a_tile_whose_wait_ran_out():
    # the waits before stand in an inner loop, whose break leaves only that one
    announced = re.findall(r"if \((.*?)\) mbar_arrive\(&p_full\[u\]\)", _prompt_attention_of_pairs())
    assert announced == ["ok && lane == 0"]


def test_persistent_product_issues_no_tile_after_another_warps_wait_ran_out():
    source = (HERE / "gemm_tcgen05.cu").read_text()
    kernel = source[source.index("gemm_tcgen05_kernel(const"): source.index("// ---------------- teardown", source.index("gemm_tcgen05_kernel(const"))]
    loops = re.findall(r"for \(int j = 0; j < n_segments(.*?)const Segment seg", kernel, re.S)
    assert len(loops) == 4 and all("flag[0]" in loop for loop in loops[:3])        # two forms of the producer, the issuing warp; the epilogue is last
