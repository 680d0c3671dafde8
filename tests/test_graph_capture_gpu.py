"""Stream capture: calls that need the context's scratch, first in a graph, and graphs replayed after the scratch has grown."""
import pytest
import torch

import deepgemm_rust_b200 as dg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def stream():
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        yield s
    torch.cuda.synchronize()


def operand(ctx, rows, k, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    data, sf = dg.cast_bf16_to_fp8_sf_dev(ctx, torch.randn((rows, k), generator=gen, device="cuda").bfloat16(), k, rows, k, 128)
    return dg.LpOperand(data, sf, rows, k, k)


def f32scale(ctx, m, n, k):
    gen = torch.Generator(device="cuda").manual_seed(m + n + k)
    a, b = (dg.Fp8Tensor(torch.randn((r, k), generator=gen, device="cuda").to(torch.float8_e4m3fn).view(torch.uint8), r, k, k) for r in (m, n))
    sfa_t = dg.transform_sf_dev(ctx, torch.rand((m, k // 128), generator=gen, device="cuda"), m, k // 128)
    sfb = torch.rand(((n + 127) // 128, k // 128), generator=gen, device="cuda")
    return lambda c, out: dg.fp8_gemm_nt_dev(c, a, sfa_t, b, sfb, out, n)


def dense(ctx, m, n, k):
    a, b = operand(ctx, m, k, m), operand(ctx, n, k, n)
    return lambda c, out: dg.fp8_fp4_gemm_dev(c, a, b, dg.Sm100Out.Bf16(out, n))


def contiguous(ctx, m, n, k):
    groups = m // 128
    a, b = operand(ctx, m, k, m), operand(ctx, groups * n, k, n)
    index = torch.arange(groups, dtype=torch.int32, device="cuda").repeat_interleave(128)
    return lambda c, out: dg.m_grouped_fp8_fp4_gemm_contiguous_dev(c, a, index, b, dg.Sm100Out.Bf16(out, n), groups)


# (call, sizes, larger sizes for the same scratch, tile choice pinned by environment variables)
CASES = {
    "f32 scales, K ranges": (f32scale, (64, 1024, 2048), (64, 4096, 7168), {}),
    "f32 scales by their exponents": (f32scale, (64, 1024, 2048), (64, 4096, 7168), {"DG_F32_SCALES": "exponent"}),
    "dense, K ranges": (dense, (8, 2112, 7168), (128, 7168, 16384), {"DG_SKINNY": "0"}),
    "dense, swapped family, K ranges": (dense, (8, 1024, 4096), (128, 2048, 8192), {"DG_SWAP": "1", "DG_SPLITS": "3"}),
    "contiguous groups": (contiguous, (512, 256, 512), (8 * 128, 256, 512), {}),
}


@pytest.mark.parametrize("case", list(CASES))
def test_scratch_of_a_captured_call(case, stream, monkeypatch):
    make, small, large, env = CASES[case]
    for name, value in env.items():
        monkeypatch.setenv(name, value)
    if make is dense:
        for size in (small, large):
            choice = dg.best_config(dg.Sm100Desc(dg.GemmType.Normal, *size))
            assert choice.num_splits > 1 and choice.swap_ab == ("DG_SWAP" in env)
    warm = dg.DgContext(0)
    call, big_call = make(warm, *small), make(warm, *large)
    outs = [torch.zeros(size[:2], dtype=torch.bfloat16, device="cuda") for size in (small, small, small, large, large)]
    eager, graphed, after, big_eager, big_after = outs
    call(warm, eager)
    big_call(warm, big_eager)
    warm.sync()
    ctx = dg.DgContext(0)         # has no scratch yet
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        call(ctx, graphed)
    call(ctx, after)              # outside the graph, on scratch that came into being while capturing
    ctx.sync()
    assert torch.equal(after, eager)
    graph.replay()
    ctx.sync()
    assert torch.equal(graphed, eager)
    big_call(ctx, big_after)      # the scratch grows; the graph keeps what it holds
    ctx.sync()
    assert torch.equal(big_after, big_eager)
    graphed.zero_()
    graph.replay()
    ctx.sync()
    assert torch.equal(graphed, eager)
    del graph
    ctx.close()
    warm.close()
