"""Which tile family a problem gets, through dg_best_config (no GPU: the choice is host code).  The lines are measured ones; the
figures stand beside the rule in csrc/dg_api.cu."""
import pytest

import deepgemm_rust_b200 as dg

NORMAL, CONTIGUOUS, MASKED = dg.GemmType.Normal, dg.GemmType.MGroupedContiguous, dg.GemmType.MGroupedMasked
E4M3, F32, FP8_OUT = {}, {"cd_dtype": 1}, {"cd_dtype": 2}
PER_32 = [{"a_bits": 8, "b_bits": 4, "gran_b": 32}, {"a_bits": 4, "b_bits": 4, "gran_a": 32, "gran_b": 32}, {"gran_a": 32}, {"gran_b": 32}]


def choice(*sizes, **kw):
    return dg.best_config(dg.Sm100Desc(*sizes, **kw))


@pytest.mark.parametrize("operands", PER_32)
@pytest.mark.parametrize("out", [E4M3, F32])
@pytest.mark.parametrize("sizes", [
    (MASKED, 256, 4096, 7168, 32, 128), (MASKED, 128, 7168, 2048, 32, 32),          # decode steps of a layer of 32 experts
    (CONTIGUOUS, 65536, 4096, 7168, 256), (CONTIGUOUS, 8192, 5824, 6144, 22),       # small expert groups
    (NORMAL, 2, 11992, 10752), (NORMAL, 32, 18936, 4096),                           # few dense rows
])
def test_operands_with_per_32_scales_keep_the_first_family(sizes, out, operands):
    assert choice(*sizes).swap_ab                     # with per-128 scales
    assert not choice(*sizes, **operands, **out).swap_ab


@pytest.mark.parametrize("sizes,kw,tile", [
    ((dg.GemmType.Batched, 420, 1792, 512, 10), F32, (256, 192, 256, 1)),
    ((dg.GemmType.Batched, 24, 3200, 512, 12), FP8_OUT, (128, 128, 128, 1)),
    ((dg.GemmType.Batched, 876, 3072, 2048, 6), E4M3, (256, 224, 256, 1)),
    ((NORMAL, 972, 8704, 1024), {"gran_a": 32, "gran_b": 32, **F32}, (256, 160, 256, 1)),
])
def test_problems_outside_the_fit_of_the_dense_costs_keep_their_tiles(sizes, kw, tile):
    # the cost constants of dense problems were fitted to unbatched ones, e4m3 with per-128 scales or e2m1; these measured 5-28 %
    # slower with the tiles the fitted constants gave them
    c = choice(*sizes, **kw)
    assert (c.block_m, c.block_n, c.block_k, c.num_splits) == tile


@pytest.mark.parametrize("layout", [CONTIGUOUS, MASKED])
def test_shared_memory_of_a_choice_counts_the_group_table(layout, monkeypatch):
    # 16 bytes per group beside what the stages take, as many as fit; none for single CTAs, whose kernels have no table
    monkeypatch.setenv("DG_STAGES", "6")

    def smem(groups):
        c = choice(layout, 256 * (groups if layout == CONTIGUOUS else 1), 4096, 7168, groups, 128)
        assert c.swap_ab
        return c.smem_size
    assert smem(200) - smem(100) == 16 * 100
    assert smem(1 << 14) == dg.SM100_SMEM_CAPACITY // 16 * 16
    monkeypatch.setenv("DG_CTAS", "1")
    assert smem(200) == smem(100)


@pytest.mark.parametrize("slot,height", [(64, 64), (76, 96), (128, 128), (250, 128), (516, 160), (924, 256), (4096, 256)])
@pytest.mark.parametrize("expected", [1, 16])
def test_a_weak_hint_does_not_shorten_the_tiles_of_a_masked_problem(slot, height, expected):
    # expected_m is a hint about the mean of the groups; a group may fill its slot whatever it says
    c = choice(MASKED, slot, 4096, 7168, 32, expected, **FP8_OUT)
    assert c.swap_ab and c.block_m == height


@pytest.mark.parametrize("sizes,kw,swapped", [
    # decode steps of 32 experts: e4m3 output, then bf16 with short K
    ((MASKED, 256, 4096, 7168, 32, 128), FP8_OUT, True), ((MASKED, 128, 7168, 2048, 32, 32), E4M3, True),
    # masked: half a wave of pair tiles (37 of 74), 28 slabs of K, 4096 columns
    ((MASKED, 128, 256, 7168, 37, 32), E4M3, True), ((MASKED, 128, 256, 7168, 36, 32), FP8_OUT, False),
    ((MASKED, 128, 2048, 3584, 32, 32), E4M3, True), ((MASKED, 128, 2048, 3456, 32, 32), E4M3, False),
    ((MASKED, 128, 2048, 2048, 32, 32), FP8_OUT, True), ((MASKED, 128, 2048, 1920, 32, 32), FP8_OUT, False),
    ((MASKED, 128, 4096, 2048, 10, 32), E4M3, True), ((MASKED, 128, 4096, 2048, 9, 32), E4M3, False), ((MASKED, 128, 3968, 2048, 64, 32), F32, False),
    ((MASKED, 1024, 4096, 7168, 32, 450), E4M3, True), ((MASKED, 1024, 4096, 7168, 32, 451), E4M3, False),
    # prefill of 256 experts, about 256 rows each and 64 of padding
    ((CONTIGUOUS, 98304, 4096, 7168, 256), E4M3, True), ((CONTIGUOUS, 98304, 7168, 2048, 256), E4M3, True),
    # contiguous: a wave of pair tiles, 2048 columns, groups that fit one tile where K is short
    ((CONTIGUOUS, 10 * 256, 2048, 3584, 10), E4M3, True), ((CONTIGUOUS, 9 * 256, 2048, 3584, 9), E4M3, False),
    ((CONTIGUOUS, 64 * 256, 2040, 7168, 64), E4M3, False), ((CONTIGUOUS, 64 * 256, 2048, 3456, 64), E4M3, True),
    ((CONTIGUOUS, 64 * 128, 2048, 3456, 64), E4M3, False), ((CONTIGUOUS, 64 * 512, 2048, 3456, 64), E4M3, False),
    ((CONTIGUOUS, 64 * 512, 2048, 3584, 64), E4M3, True), ((CONTIGUOUS, 64 * 520, 2048, 3584, 64), E4M3, False),
    ((CONTIGUOUS, 20 * 128, 1792, 2048, 20), E4M3, False), ((CONTIGUOUS, 6 * 128, 264, 2176, 6), E4M3, False),
])
def test_family_of_a_grouped_problem(sizes, kw, swapped):
    assert choice(*sizes, **kw).swap_ab == swapped


@pytest.mark.parametrize("sizes,kw", [
    ((2894, 6144, 1024), E4M3), ((4801, 3704, 1024), E4M3), ((7467, 3448, 2560), F32), ((1096, 14696, 2560), F32), ((7706, 7800, 512), F32),
    ((1862, 9152, 512), {**PER_32[0], **F32}), ((1727, 9504, 1536), PER_32[0]), ((7620, 7272, 512), {**PER_32[1], **F32}), ((1539, 8384, 1024), {**PER_32[1], **F32}),
])
def test_dense_problems_of_several_waves_store_beside_the_next_tile(sizes, kw):
    # with one accumulator every wave's epilogue is exposed: 256-column tiles measured 1.18 to 1.36 times as long here as narrower
    # ones with two accumulators
    c = choice(NORMAL, *sizes, **kw)
    assert c.num_accum_stages == 2 and not c.swap_ab
