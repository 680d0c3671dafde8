"""Wide tiles (two accumulators of up to 224 columns per CTA pair) against the other tiles of the same family, bit for bit: both add
up the same products in the same order, so that nothing may differ, whatever the shape, the formats and the output."""
import pytest
import torch

import deepgemm_rust_b200 as dg

@pytest.fixture(scope="module")
def ctx():
    c = dg.DgContext(0)
    yield c
    c.sync()
    c.close()


def operand(ctx, rows, k, bits, seed, groups=1, gran=128, rows_per_group=None):
    """Quantised with K rounded up to what the quantiser takes, of which the operand is the first k columns (their scale words come first)."""
    ld = -(-k // 512) * 512
    x = torch.randn((rows, ld), generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda", dtype=torch.bfloat16)
    if bits == 4:
        data, sf = dg.cast_bf16_to_fp4_packed_sf_dev(ctx, x, ld, rows, ld, groups, dg.SF_RULE_RANGE_FIT)
        return dg.LpOperand(data, sf, rows_per_group or rows, k, ld, 4, 32)
    data, sf = dg.cast_bf16_to_fp8_sf_dev(ctx, x, ld, rows, ld, gran, groups)
    return dg.LpOperand(data, sf, rows_per_group or rows, k, ld, 8, gran)


def each(monkeypatch, run):
    """run() with the wide tiles and with 224-column tiles of a CTA pair."""
    monkeypatch.setenv("DG_WIDE_TILE", "1")
    for rows in (1, 4096):
        assert dg.kernel_name(dg.Sm100Desc(dg.GemmType.Normal, rows, 392, 128)) == "dg_gemm_wide_kernel"
    wide = run()
    monkeypatch.setenv("DG_WIDE_TILE", "0")
    monkeypatch.setenv("DG_SWAP", "0")
    monkeypatch.setenv("DG_BLOCK_N", "224")
    monkeypatch.setenv("DG_CTAS", "2")
    monkeypatch.setenv("DG_SPLITS", "1")
    return wide, run()


def both(ctx, monkeypatch, run):
    """Both leave the same."""
    def done():
        d = run()
        ctx.sync()
        return d
    assert torch.equal(*each(monkeypatch, done))


# units of work: fewer than pairs of CTAs; whole tiles, then at most one half each, then at most two; an odd number of halves across, and a last
# half of 8 columns; K of one stage, of a part of a stage, and of an odd number of them
SIZES = [(1, 392, 128), (300, 456, 1152), (257, 680, 640), (2100, 4296, 384), (4352, 1800, 256), (4000, 4488, 128), (2560, 8288, 640)]


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", SIZES)
@pytest.mark.parametrize("a_bits,b_bits", [(8, 8), (8, 4), (4, 8), (4, 4)])
def test_dense(ctx, monkeypatch, m, n, k, a_bits, b_bits):
    a, b = operand(ctx, m, k, a_bits, 1), operand(ctx, n, k, b_bits, 2)

    def run():
        d = torch.full((m, n), 7.0, dtype=torch.bfloat16, device="cuda")
        dg.fp8_fp4_gemm_dev(ctx, a, b, dg.Sm100Out.Bf16(d, n))
        return d
    both(ctx, monkeypatch, run)


@pytest.mark.gpu
@pytest.mark.parametrize("epilogue", [dict(alpha=-0.5), dict(accumulate=True), dict(tc_util=60)])
@pytest.mark.parametrize("f32", [True, False])
@pytest.mark.parametrize("gran_a,gran_b", [(128, 128), (32, 128), (32, 32)])
def test_outputs_and_scales(ctx, monkeypatch, epilogue, f32, gran_a, gran_b):
    m, n, k = 700, 904, 1280
    a, b = operand(ctx, m, k, 8, 3, gran=gran_a), operand(ctx, n, k, 8, 4, gran=gran_b)

    def run():
        d = torch.full((m, n), 3.0, dtype=torch.float32 if f32 else torch.bfloat16, device="cuda")
        dg.fp8_fp4_gemm_dev(ctx, a, b, dg.Sm100Out.F32(d, n) if f32 else dg.Sm100Out.Bf16(d, n), dg.Sm100Epilogue(**epilogue))
        return d
    both(ctx, monkeypatch, run)


@pytest.mark.gpu
def test_duty_cycle_paces_them_like_the_other_tiles(ctx, monkeypatch):
    # 37 x 896: one wide tile per pair of CTAs, or two of 224 columns: the same columns and slabs of K, so the same pauses, four times what the
    # tensor cores take for bf16 operands and eight times for these, in which the tiles' own differences drown
    m, n, k = 37 * 256, 896, 4096
    a, b = operand(ctx, m, k, 8, 8), operand(ctx, n, k, 8, 9)
    d = torch.zeros((m, n), dtype=torch.bfloat16, device="cuda")

    def run():
        times = []
        for _ in range(5):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            dg.fp8_fp4_gemm_dev(ctx, a, b, dg.Sm100Out.Bf16(d, n), dg.Sm100Epilogue(tc_util=20))
            e1.record()
            ctx.sync()
            times.append(e0.elapsed_time(e1))
        return sorted(times)[2]
    wide, narrow = each(monkeypatch, run)
    assert 0.85 * narrow < wide < 1.15 * narrow


@pytest.mark.gpu
@pytest.mark.parametrize("alignment", [16, 128])
# 24 and 36 tiles, all as single halves; 72 whole ones; 74 whole ones and 10 as halves, some of which have no columns
@pytest.mark.parametrize("n", [456, 1096, 2600, 2704])
@pytest.mark.parametrize("f32", [True, False])
def test_grouped(ctx, monkeypatch, alignment, n, f32):
    # groups of nothing, of one row, of just a tile, of a tile and a row: boxes that cross a group's end, tiles that run into the next group
    sizes, k = [0, 1, 256, 257, 100, 700, 0, 31, 520], 640
    m_indices, rows = [], 0
    for g, size in enumerate(sizes):
        m_indices += [g] * size + [-1] * (-size % alignment)
    rows, groups = len(m_indices), len(sizes)
    m_indices = torch.tensor(m_indices, dtype=torch.int32, device="cuda")
    a, b = operand(ctx, rows, k, 8, 5), operand(ctx, groups * n, k, 8, 6, groups=groups)
    dtype, kind = (torch.float32, dg.Sm100Out.F32) if f32 else (torch.bfloat16, dg.Sm100Out.Bf16)

    def contiguous():
        d = torch.full((rows, n), 5.0, dtype=dtype, device="cuda")
        dg.m_grouped_fp8_fp4_gemm_contiguous_dev(ctx, a, m_indices, b, kind(d, n), groups)
        return d

    slot = 704
    am = operand(ctx, groups * slot, k, 8, 7, groups=groups, rows_per_group=slot)
    masked_m = torch.tensor(sizes, dtype=torch.int32, device="cuda")

    def masked():
        d = torch.full((groups * slot, n), 5.0, dtype=dtype, device="cuda")
        dg.m_grouped_fp8_fp4_gemm_masked_dev(ctx, am, masked_m, b, kind(d, n), groups, 600)
        return d
    dg.set_mk_alignment_for_contiguous_layout(alignment)
    try:
        with monkeypatch.context() as patch:
            both(ctx, patch, contiguous)
        with monkeypatch.context() as patch:
            both(ctx, patch, masked)
    finally:
        dg.set_mk_alignment_for_contiguous_layout(128)


CONTIGUOUS = dg.GemmType.MGroupedContiguous
E2M1 = dict(a_bits=4, b_bits=4, gran_a=32, gran_b=32)
MIXED = dict(b_bits=4, gran_b=32)


@pytest.mark.parametrize("sizes,kw,wide", [
    ((dg.GemmType.Normal, 4096, 7168, 16384), {}, True), ((dg.GemmType.Normal, 4096, 7168, 7168), dict(a_bits=4, b_bits=4, gran_a=32, gran_b=32), True),
    ((dg.GemmType.Normal, 4096, 7168, 16384), dict(gran_a=32), False), ((dg.GemmType.Normal, 4096, 7168, 16384), dict(cd_dtype=2), False),
    ((dg.GemmType.Normal, 1024, 4096, 7168), {}, False),                                       # one wave
    ((dg.GemmType.Normal, 4096, 7168, 7168), dict(**E2M1, cd_dtype=1), False),
    # K of 32 slabs with many halves per pair, of 16 and 24 with two e2m1 operands; few and even numbers of halves; more columns
    ((dg.GemmType.Normal, 8192, 8192, 4096), {}, True), ((dg.GemmType.Normal, 8192, 8192, 3968), {}, False), ((dg.GemmType.Normal, 5604, 3400, 8192), {}, True),
    ((dg.GemmType.Normal, 5604, 3400, 6016), {}, False), ((dg.GemmType.Normal, 6516, 4616, 9216), {}, False), ((dg.GemmType.Normal, 2607, 6624, 10240), MIXED, False),
    ((dg.GemmType.Normal, 4096, 7168, 4096), E2M1, True), ((dg.GemmType.Normal, 4096, 7168, 3840), E2M1, False),
    ((dg.GemmType.Normal, 7300, 4216, 6144), E2M1, True), ((dg.GemmType.Normal, 7300, 4216, 4096), E2M1, False),
    ((CONTIGUOUS, 32 * 2112, 4096, 7168, 32), {}, True), ((CONTIGUOUS, 32 * 520, 4096, 7168, 32), {}, True), ((CONTIGUOUS, 32 * 512, 4096, 7168, 32), {}, False),
    # groups whose first 256 rows make 1.3 waves of tiles, whatever the arena holds, with K below 20 slabs three and a half; no more columns than the other tiles have
    ((CONTIGUOUS, 10 * 2048, 4096, 2560, 10), {}, True), ((CONTIGUOUS, 9 * 2048, 4096, 7168, 9), {}, False), ((CONTIGUOUS, 13696, 1600, 7168, 8), {}, False),
    ((CONTIGUOUS, 26 * 2048, 4096, 2048, 26), {}, True), ((CONTIGUOUS, 25 * 2048, 4096, 2048, 25), {}, False), ((CONTIGUOUS, 25 * 2048, 4096, 2560, 25), {}, True),
    ((CONTIGUOUS, 32 * 2112, 4096, 1920, 32), {}, False), ((CONTIGUOUS, 32 * 2112, 5568, 7168, 32), {}, True),
    ((CONTIGUOUS, 32 * 2112, 5568, 3072, 32), {}, True), ((CONTIGUOUS, 32 * 2112, 5568, 2944, 32), {}, False), ((CONTIGUOUS, 17 * 1414, 3840, 5120, 17), {}, True),
    ((CONTIGUOUS, 17 * 1414, 3840, 4992, 17), {}, False),
    ((dg.GemmType.MGroupedMasked, 2048, 4096, 7168, 32, 2048), {}, False), ((dg.GemmType.Batched, 2048, 4096, 7168, 16), {}, False),
])
def test_which_problems_get_them(sizes, kw, wide):
    assert (dg.kernel_name(dg.Sm100Desc(*sizes, **kw)) == "dg_gemm_wide_kernel") == wide
