"""The dense kernel for a handful of activation rows, against a f64 product of the dequantised operands."""
import pytest
import torch

import deepgemm_rust_b200 as dg


@pytest.fixture(scope="module")
def ctx():
    c = dg.DgContext(0)
    yield c
    c.sync()
    c.close()


def operand(rows, k, ld, seed, exponents=(118, 136)):
    """Any e4m3 code but NaN and any scale of a range, in the packed layout: (operand, its values in f64)."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    data = torch.randint(0, 256, (rows, ld), generator=gen, device="cuda", dtype=torch.uint8)
    data[(data & 0x7F) == 0x7F] = 0
    stride, cols = dg.sf_aligned_rows(rows), dg.sf_packed_cols(k, 128)
    e = torch.randint(*exponents, (4 * cols, stride), generator=gen, device="cuda", dtype=torch.int32)
    sf = (e.view(cols, 4, stride) << torch.tensor([0, 8, 16, 24], device="cuda", dtype=torch.int32).view(1, 4, 1)).sum(1, dtype=torch.int32)
    scale = torch.exp2(e[:k // 128, :rows].double() - 127).T.repeat_interleave(128, 1)
    return dg.LpOperand(data, sf.view(-1), rows, k, ld, 8, 128), data[:, :k].view(torch.float8_e4m3fn).double() * scale


def is_skinny(m, n, k):
    return dg.kernel_name(dg.Sm100Desc(dg.GemmType.Normal, m, n, k)) == "dg_gemm_skinny_kernel"


@pytest.mark.parametrize("m,n,k,skinny", [
    (8, 2112, 7168, True), (1, 4096, 15616, True), (8, 4096, 15744, False), (8, 9344, 5248, True), (8, 9352, 5248, False), (16, 5856, 4096, True),
    (16, 5864, 4096, False), (9, 1016, 12288, True), (9, 1016, 12416, False), (9, 2376, 7168, True), (9, 2376, 7296, False), (32, 1952, 4096, True),
    (17, 1960, 4096, False), (17, 512, 4224, False), (33, 512, 1024, False),
    # K that few blocks share among 16 warps; blocks in one, two and more waves; more of them than those of a few warps are worth
    (8, 1184, 16384, True), (8, 1184, 16512, False), (8, 1192, 24576, True), (8, 2368, 24704, False), (8, 2376, 16512, False),
    (9, 496, 10240, True), (9, 496, 10368, False), (9, 504, 12288, True), (9, 504, 12416, False), (8, 33152, 128, True), (8, 33160, 128, False), (8, 343744, 128, False),
    (16, 9472, 2432, True), (16, 9480, 1024, True), (16, 9480, 1152, False), (16, 18944, 896, True), (16, 18952, 896, False),
    (16, 18952, 1024, True), (16, 23440, 1024, False), (16, 33152, 512, True),
    (16, 33160, 128, False), (17, 4736, 1664, True), (17, 4744, 1024, True), (17, 4744, 1152, False), (17, 9472, 768, True), (17, 9480, 512, True),
    (17, 9480, 640, False), (17, 16576, 256, True), (17, 16584, 128, False),
    (8, 2112, 7200, False),
])
def test_which_problems_get_it(m, n, k, skinny):
    assert is_skinny(m, n, k) == skinny


@pytest.mark.parametrize("m,n,k,stages,smem", [(8, 2112, 7168, 2, 16 * 8 * 17 * 4), (16, 4736, 4096, 2, 8 * 16 * 17 * 4), (17, 4744, 896, 1, 4 * 32 * 17 * 4)])
def test_tile_choice_describes_it(m, n, k, stages, smem, monkeypatch):
    # 16, 8 and 4 warps: what the query reports is what a call launches
    c = dg.best_config(dg.Sm100Desc(dg.GemmType.Normal, m, n, k))
    assert (c.swap_ab, c.block_m, c.block_n, c.block_k, c.cluster_m, c.cluster_n) == (False, -(-m // 8) * 8 if m <= 16 else 32, 16, 128, 1, 1)
    assert (c.num_stages, c.num_accum_stages, c.smem_size, c.num_tiles, c.num_splits) == (stages, 1, smem, -(-n // 16), 1)
    monkeypatch.setenv("DG_SKINNY", "0")
    assert dg.best_config(dg.Sm100Desc(dg.GemmType.Normal, m, n, k)).block_n > 16


@pytest.mark.gpu
def test_a_duty_cycle_goes_to_the_tiles_that_have_one(ctx):
    # the order of the sums tells the kernels apart
    m, n, k = 8, 2112, 7168
    (a, _), (b, _) = operand(m, k, k, 8), operand(n, k, k, 9)
    d = [torch.zeros((m, n), dtype=torch.float32, device="cuda") for _ in range(3)]
    dg.fp8_fp4_gemm_dev(ctx, a, b, dg.Sm100Out.F32(d[0], n), dg.Sm100Epilogue(tc_util=99))
    with pytest.MonkeyPatch.context() as patch:
        patch.setenv("DG_SKINNY", "0")
        dg.fp8_fp4_gemm_dev(ctx, a, b, dg.Sm100Out.F32(d[1], n))
    dg.fp8_fp4_gemm_dev(ctx, a, b, dg.Sm100Out.F32(d[2], n))
    ctx.sync()
    assert torch.equal(d[0], d[1]) and not torch.equal(d[0], d[2])


@pytest.mark.gpu
@pytest.mark.parametrize("m", [1, 7, 8, 9, 16, 17, 32])
@pytest.mark.parametrize("n,k", [
    (8, 128), (16, 256), (24, 2048),              # one block, a block and a part; fewer K blocks than warps, and as many
    (2368, 2176), (2376, 384), (4736, 640), (4744, 896),      # either side of the lines between 16, 8 and 4 warps; odd numbers of K blocks per warp
])
@pytest.mark.parametrize("f32", [True, False])
def test_product(ctx, m, n, k, f32):
    check_product(ctx, m, n, k, f32)


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [
    (8, 2112, 7168), (8, 1280, 24576), (1, 4096, 15616), (8, 9344, 5248),      # the longest K of 16, 8 and 4 warps
    (9, 1024, 12288), (16, 3344, 7168), (16, 9472, 2432), (32, 1920, 4096), (17, 9472, 768),
])
@pytest.mark.parametrize("f32", [True, False])
def test_product_of_the_longest_k(ctx, m, n, k, f32):
    check_product(ctx, m, n, k, f32)


def check_product(ctx, m, n, k, f32):
    assert is_skinny(m, n, k)
    (a, fa), (b, fb) = operand(m, k, k + 16, 1), operand(n, k, k + 32, 2)
    ld = n + 8
    d = torch.full((m, ld), 7.0, dtype=torch.float32 if f32 else torch.bfloat16, device="cuda")
    dg.fp8_fp4_gemm_dev(ctx, a, b, dg.Sm100Out.F32(d, ld) if f32 else dg.Sm100Out.Bf16(d, ld))
    ctx.sync()
    want, size = fa @ fb.T, fa.abs() @ fb.abs().T
    # f32 sums: fewer than 128 roundings of 2^-24 of the terms' magnitudes (four instructions and a sum for each of a warp's K blocks, 16 at most, then the
    # warps', 16 at most); a bf16 result is rounded once more, 8 significant bits
    bound = 128 * 2.0 ** -24 * size + (0.0 if f32 else 2.0 ** -8) * want.abs()
    assert bool(((d[:, :n].double() - want).abs() <= bound).all())
    assert bool((d[:, n:] == 7.0).all())


@pytest.mark.gpu
@pytest.mark.parametrize("f32", [True, False])
@pytest.mark.parametrize("m", [3, 12])
def test_epilogue(ctx, m, f32):
    n, k = 536, 1280
    (a, fa), (b, fb) = operand(m, k, k, 3), operand(n, k, k, 4)
    dtype, kind = (torch.float32, dg.Sm100Out.F32) if f32 else (torch.bfloat16, dg.Sm100Out.Bf16)
    want, size = fa @ fb.T, fa.abs() @ fb.abs().T
    unit = 2.0 ** -23 if f32 else 2.0 ** -8
    d = torch.zeros((m, n), dtype=dtype, device="cuda")
    dg.fp8_fp4_gemm_dev(ctx, a, b, kind(d, n), dg.Sm100Epilogue(alpha=-0.375))
    ctx.sync()
    assert bool(((d.double() + 0.375 * want).abs() <= 128 * 2.0 ** -24 * size + unit * want.abs()).all())
    old = (torch.randn((m, n), generator=torch.Generator(device="cuda").manual_seed(5), device="cuda") * size.mean().sqrt()).to(dtype)
    d = old.clone()
    dg.fp8_fp4_gemm_dev(ctx, a, b, kind(d, n), dg.Sm100Epilogue(accumulate=True))
    ctx.sync()
    # the product and the sum are each rounded to the output type
    assert bool(((d.double() - old.double() - want).abs() <= 128 * 2.0 ** -24 * size + unit * (2 * want.abs() + old.double().abs())).all())


@pytest.mark.gpu
@pytest.mark.parametrize("f32", [True, False])
def test_calls_on_two_streams_add_into_one_output(f32):
    # the first column of both operands is 1, the rest 0: every call adds 1, exact in bf16 up to 256
    m, n, k, calls = 8, 2112, 1024, 100
    assert is_skinny(m, n, k)
    ops = []
    for rows in (m, n):
        data = torch.zeros((rows, k), dtype=torch.uint8, device="cuda")
        data[:, 0] = 0x38
        words = dg.sf_packed_cols(k, 128) * dg.sf_aligned_rows(rows)
        ops.append(dg.LpOperand(data, torch.full((words,), 0x7F7F7F7F, dtype=torch.int32, device="cuda"), rows, k, k, 8, 128))
    d = torch.zeros((m, n), dtype=torch.float32 if f32 else torch.bfloat16, device="cuda")
    out = dg.Sm100Out.F32(d, n) if f32 else dg.Sm100Out.Bf16(d, n)
    torch.cuda.synchronize()
    contexts = [dg.DgContext(0, own_stream=True) for _ in range(2)]
    for _ in range(calls):
        for c in contexts:
            dg.fp8_fp4_gemm_dev(c, *ops, out, dg.Sm100Epilogue(accumulate=True))
    for c in contexts:
        c.sync()
    assert bool((d == 2 * calls).all())
    for c in contexts:
        c.close()


@pytest.mark.gpu
def test_scales_and_codes_at_the_ends_of_their_range(ctx, monkeypatch):
    # exponents far apart whose product is ordinary, scales of 2^-127, NaN scales and NaN codes: as the block-scaled tensor core has them
    m, n, k = 5, 64, 512
    a, fa = operand(m, k, k, 6, (230, 234))
    b, fb = operand(n, k, k, 7, (20, 24))
    words = b.sf.view(1, n)
    words[0, 3] = 0                                   # 2^-127
    words[0, 9] = words[0, 9] | 0xFF                  # NaN in the first K block of one column
    a.data[2, 300] = 0x7F                             # NaN in a row
    out = []
    for skinny in ("1", "0"):
        monkeypatch.setenv("DG_SKINNY", skinny)
        d = torch.zeros((m, n), dtype=torch.float32, device="cuda")
        dg.fp8_fp4_gemm_dev(ctx, a, b, dg.Sm100Out.F32(d, n))
        ctx.sync()
        out.append(d)
    assert torch.equal(out[0].isnan(), out[1].isnan())
    assert bool(out[0][2].isnan().all()) and bool(out[0][:, 9].isnan().all()) and int(out[0].isnan().sum()) == n + m - 1
    size = (fa.abs() @ fb.abs().T)
    ok = ~out[0].isnan()
    ok[:, 3] = False
    assert bool(((out[0].double() - out[1].double()).abs() <= 2 * 128 * 2.0 ** -24 * size)[ok].all())
    assert bool(torch.isclose(out[0][:2, 3], out[1][:2, 3], rtol=1e-4, atol=0).all())
