"""The older f32-scale API (deepgemm/src/ops.rs:328,422,535,635), checked against the literal CPU references
(reference.rs:85-208) in the style of the reference's own end-to-end tests (deepgemm/tests/e2e.rs:47-249): LCG inputs
quantised with f32_to_e4m3, constant scales, the same shapes and the same masked_m fixture.

Two routes serve these calls.  The default applies every f32 scale exactly, K block by K block (dg_gemm_f32scale_kernel): it
is run with the reference's own scale values 0.01 / 0.02, with per-block amax / 448 scales (the CPU-runnable benchmark case as
the contract words it, against a committed fixture), and with powers of two.  DG_F32_SCALES=exponent is what the reference
itself does on Blackwell -- only the exponent of each scale reaches the block-scaled kernel (cuda/sm100_cast.rs:214) -- and
is exact for powers of two only, so it is run with 2^-6 / 2^-5."""
import numpy as np
import pytest
import torch

import deepgemm_rust_b200 as dg
from oracle import oracle as O
from tests.helpers import dev, to_f32

pytestmark = pytest.mark.gpu
import os
import subprocess
import sys

# (route, activation scale, weight scale)
ROUTES = [("exact", 0.01, 0.02), ("exact", 2.0 ** -6, 2.0 ** -5), ("exponent", 2.0 ** -6, 2.0 ** -5)]
routes = pytest.mark.parametrize("route,SFA,SFB", ROUTES)


def pin_route(monkeypatch, route):
    if route == "exponent":
        monkeypatch.setenv("DG_F32_SCALES", "exponent")
    else:
        monkeypatch.delenv("DG_F32_SCALES", raising=False)


@pytest.fixture(scope="module")
def ctx():
    c = dg.DgContext(0)
    yield c
    c.sync()
    c.close()


def lcg_e4m3(seed, rows, k):
    v = O.lcg_values(seed, rows * k, 2.0).reshape(rows, k)
    return np.vectorize(O.f32_to_e4m3_fast, otypes=[np.uint8])(v)


def reference_tolerance(got, want):
    # e2e.rs: |g - w| / max(|w|, 1) < 0.05
    assert np.max(np.abs(got - want) / np.maximum(np.abs(want), 1.0)) < 0.05
    assert O.calc_diff(got, want) <= 2e-5


@routes
def test_fp8_gemm_nt(ctx, route, SFA, SFB, monkeypatch):
    pin_route(monkeypatch, route)
    m, n, k = 256, 512, 768                                  # e2e.rs:47
    a, b = lcg_e4m3(1, m, k), lcg_e4m3(2, n, k)
    sfa = np.full((m, k // 128), SFA, np.float32)
    sfb = np.full((n // 128, k // 128), SFB, np.float32)
    a_sf_t = dg.transform_sf_dev(ctx, dev(sfa), m, k // 128, 1)
    out = torch.zeros((m, n), dtype=torch.bfloat16, device="cuda")
    dg.fp8_gemm_nt_dev(ctx, dg.Fp8Tensor(dev(a), m, k, k), a_sf_t, dg.Fp8Tensor(dev(b), n, k, k), dev(sfb), out, n)
    ctx.sync()
    reference_tolerance(to_f32(out), O.ref_fp8_gemm_nt(a, sfa, b, sfb, threads=8))


@routes
def test_m_grouped_contiguous(ctx, route, SFA, SFB, monkeypatch):
    pin_route(monkeypatch, route)
    groups, gm, n, k = 4, 128, 256, 512                      # e2e.rs:88
    m = groups * gm
    a, b = lcg_e4m3(3, m, k), lcg_e4m3(4, groups * n, k)
    sfa = np.full((m, k // 128), SFA, np.float32)
    sfb = np.full((groups * n // 128, k // 128), SFB, np.float32)
    m_idx = np.repeat(np.arange(groups, dtype=np.int32), gm)
    a_sf_t = dg.transform_sf_dev(ctx, dev(sfa), m, k // 128, 1)
    out = torch.zeros((m, n), dtype=torch.bfloat16, device="cuda")
    dg.m_grouped_fp8_gemm_nt_contiguous_dev(ctx, dg.Fp8Tensor(dev(a), m, k, k), a_sf_t, dg.Fp8Tensor(dev(b), groups * n, k, k), dev(sfb), out, n,
                                            dev(m_idx), groups)
    ctx.sync()
    want = O.ref_m_grouped_contiguous(a, sfa, m_idx, b, sfb[:n // 128].reshape(-1), n, threads=8)   # the reference indexes one shared scale block
    reference_tolerance(to_f32(out), want)


@routes
def test_m_grouped_masked_and_bmm(ctx, route, SFA, SFB, monkeypatch):
    pin_route(monkeypatch, route)
    masked = np.array([37, 128, 1, 64, 15, 100, 128, 3], np.int32)   # e2e.rs:131
    groups, m_max, n, k = len(masked), 128, 256, 512
    a, b = lcg_e4m3(5, groups * m_max, k), lcg_e4m3(6, groups * n, k)
    sfa = np.full((groups * m_max, k // 128), SFA, np.float32)
    sfb = np.full((groups * n // 128, k // 128), SFB, np.float32)
    a_sf_t = dg.transform_sf_dev(ctx, dev(sfa), m_max, k // 128, groups)
    out = torch.zeros((groups * m_max, n), dtype=torch.bfloat16, device="cuda")
    A, B = dg.Fp8Tensor(dev(a), groups * m_max, k, k), dg.Fp8Tensor(dev(b), groups * n, k, k)
    dg.m_grouped_fp8_gemm_nt_masked_dev(ctx, A, a_sf_t, B, dev(sfb), out, n, dev(masked), groups, m_max, 64)
    ctx.sync()
    want = O.ref_m_grouped_masked(a, sfa, masked, m_max, b, sfb[:n // 128].reshape(-1), n, threads=8)
    got = to_f32(out)
    valid = np.concatenate([np.arange(g * m_max, g * m_max + masked[g]) for g in range(groups)])
    reference_tolerance(got[valid], want[valid])
    # batched: every row of every group
    out2 = torch.zeros((groups * m_max, n), dtype=torch.bfloat16, device="cuda")
    dg.fp8_bmm_nt_dev(ctx, A, a_sf_t, B, dev(sfb), out2, n, groups, m_max, n)
    ctx.sync()
    want2 = O.ref_m_grouped_masked(a, sfa, np.full(groups, m_max, np.int32), m_max, b, sfb[:n // 128].reshape(-1), n, threads=8)
    reference_tolerance(to_f32(out2), want2)


def test_shape_errors(ctx):
    a = torch.zeros((128, 256), dtype=torch.uint8, device="cuda")
    sf = torch.ones((2, 128), dtype=torch.float32, device="cuda")
    out = torch.zeros((128, 128), dtype=torch.bfloat16, device="cuda")
    with pytest.raises(dg.DgError) as e:                      # ops.rs:308 k % 128
        dg.fp8_gemm_nt_dev(ctx, dg.Fp8Tensor(a, 128, 192, 256), sf, dg.Fp8Tensor(a, 128, 192, 256), sf, out, 128)
    assert e.value.kind == "Shape"
    with pytest.raises(dg.DgError):                           # ops.rs:313 n % 8
        dg.fp8_gemm_nt_dev(ctx, dg.Fp8Tensor(a, 128, 256, 256), sf, dg.Fp8Tensor(a, 100, 256, 256), sf, out, 128)


def test_cpu_runnable_case_with_amax_over_448_scales(ctx):
    # the benchmark contract's first configuration as it is worded: M=128, N=256, K=512, e4m3 with f32 scales amax / 448 (A per
    # 1x128, B per 128x128), f32 accumulation, bf16 output -- committed fixture: inputs, scales and ref_fp8_gemm_nt's output
    z = np.load(os.path.join(os.path.dirname(__file__), "golden", "fp8_gemm_f32scale_128x256x512.npz"))
    a, b, sfa, sfb, want = z["a"], z["b"], z["sfa"], z["sfb"], z["out"]
    m, n, k = 128, 256, 512
    a_sf_t = dg.transform_sf_dev(ctx, dev(sfa), m, k // 128, 1)
    out = torch.zeros((m, n), dtype=torch.bfloat16, device="cuda")
    dg.fp8_gemm_nt_dev(ctx, dg.Fp8Tensor(dev(a), m, k, k), a_sf_t, dg.Fp8Tensor(dev(b), n, k, k), dev(sfb), out, n)
    ctx.sync()
    assert O.calc_diff(to_f32(out), want) <= 2e-5             # contract: 1e-3; only the bf16 rounding of the output separates the two


def test_exact_route_ragged_shapes_and_varying_scales(ctx):
    # scales that differ per row, per tile and per K block (mantissas included), M and N off the tile grid, several tiles and
    # k-blocks per CTA; contiguous groups of uneven size with alignment padding
    rng = np.random.default_rng(5)
    m, n, k = 333, 392, 1664
    a, b = lcg_e4m3(11, m, k), lcg_e4m3(12, n, k)
    sfa = rng.uniform(0.004, 0.03, (m, k // 128)).astype(np.float32)
    sfb = rng.uniform(0.004, 0.03, ((n + 127) // 128, k // 128)).astype(np.float32)
    a_sf_t = dg.transform_sf_dev(ctx, dev(sfa), m, k // 128, 1)
    out = torch.zeros((m, n), dtype=torch.bfloat16, device="cuda")
    dg.fp8_gemm_nt_dev(ctx, dg.Fp8Tensor(dev(a), m, k, k), a_sf_t, dg.Fp8Tensor(dev(b), n, k, k), dev(sfb), out, n)
    ctx.sync()
    reference_tolerance(to_f32(out), O.ref_fp8_gemm_nt(a, sfa, b, sfb, threads=8))
    sizes, gn = [200, 0, 37, 129], 256
    m_idx = np.concatenate([np.concatenate([np.full(s, g, np.int32), np.full((-s) % 128, -1, np.int32)]) for g, s in enumerate(sizes)])
    mt, groups = len(m_idx), len(sizes)
    a, b = lcg_e4m3(13, mt, k), lcg_e4m3(14, groups * gn, k)
    sfa = rng.uniform(0.004, 0.03, (mt, k // 128)).astype(np.float32)
    sfb = rng.uniform(0.004, 0.03, (groups * gn // 128, k // 128)).astype(np.float32)
    a_sf_t = dg.transform_sf_dev(ctx, dev(sfa), mt, k // 128, 1)
    out = torch.full((mt, gn), float("nan"), dtype=torch.bfloat16, device="cuda")
    dg.m_grouped_fp8_gemm_nt_contiguous_dev(ctx, dg.Fp8Tensor(dev(a), mt, k, k), a_sf_t, dg.Fp8Tensor(dev(b), groups * gn, k, k), dev(sfb), out, gn,
                                            dev(m_idx), groups)
    ctx.sync()
    want = O.ref_m_grouped_contiguous(a, sfa, m_idx, b, sfb.reshape(-1), gn, per_group_sfb=True, threads=8)
    valid = np.nonzero(m_idx >= 0)[0]
    got = to_f32(out)
    assert not np.isnan(got[valid]).any()
    reference_tolerance(got[valid], want[valid])


@pytest.mark.parametrize("m,n,k", [
    (1500, 4104, 256),      # 256 x 256 tiles of CTA pairs: one full wave, ragged rows and columns, two K blocks
    (3000, 3976, 384),      # several tiles per pair, an odd number of K blocks (the accumulator buffers swap over between tiles)
    (130, 520, 6272),       # K ranges with an uneven last one, partial planes of ragged rows and columns
    (64, 4096, 2048),       # K ranges of four K blocks
    (1, 8, 128),            # one row, one K block
])
def test_exact_route_tile_variants(ctx, m, n, k):
    # every element against a float64 sum over the K blocks of exact block products; bf16 rounding (2^-8 of a value at most) is
    # what separates the two, so the squared difference stays below 2^-16 of the squared sum: calc_diff <= 2^-17
    gen = torch.Generator(device="cuda").manual_seed(m + n + k)
    kb, nb = k // 128, (n + 127) // 128
    a8 = torch.randn((m, k), generator=gen, device="cuda").to(torch.float8_e4m3fn)
    b8 = torch.randn((n, k), generator=gen, device="cuda").to(torch.float8_e4m3fn)
    sfa = torch.rand((m, kb), generator=gen, device="cuda") * 0.03 + 0.004
    sfb = torch.rand((nb, kb), generator=gen, device="cuda") * 0.03 + 0.004
    if m % 2 == 0:
        sfa[0, 0], sfb[0, 0] = 1e-24, 1e-24      # a product outside the range of one factor
        sfa[1, :], sfb[0, -1] = 1e-21, 1e18
    a64 = a8.double().view(m, kb, 128) * sfa.double().unsqueeze(-1)
    b64 = b8.double().view(n, kb, 128) * sfb.double().repeat_interleave(128, 0)[:n].unsqueeze(-1)
    want = a64.view(m, k) @ b64.view(n, k).t()
    out = torch.full((m, n), float("nan"), dtype=torch.bfloat16, device="cuda")
    a_sf_t = dg.transform_sf_dev(ctx, sfa, m, kb, 1)
    dg.fp8_gemm_nt_dev(ctx, dg.Fp8Tensor(a8.view(torch.uint8), m, k, k), a_sf_t, dg.Fp8Tensor(b8.view(torch.uint8), n, k, k), sfb, out, n)
    ctx.sync()
    got = out.double()
    assert not torch.isnan(got).any()
    for rows in ([0], [min(1, m - 1)], range(m)):       # the rows with extreme scales on their own, then everything
        x, y = got[list(rows)], want[list(rows)]
        # scaled so that squares of tiny rows do not underflow
        s = y.abs().max().clamp_min(1e-300)
        x, y = x / s, y / s
        assert float(1 - 2 * (x * y).sum() / (x * x + y * y).sum()) <= 2.0 ** -17


def test_one_context_on_two_streams(ctx):
    # calls on different streams run beside each other; each stream's K ranges have their partial planes to themselves
    gen = torch.Generator(device="cuda").manual_seed(77)
    m, n, k = 64, 2048, 7168
    b = dg.Fp8Tensor(torch.randn((n, k), generator=gen, device="cuda").to(torch.float8_e4m3fn).view(torch.uint8), n, k, k)
    sfb = torch.rand((n // 128, k // 128), generator=gen, device="cuda")
    acts = [dg.Fp8Tensor(torch.randn((m, k), generator=gen, device="cuda").to(torch.float8_e4m3fn).view(torch.uint8), m, k, k) for _ in range(2)]
    sfas = [dg.transform_sf_dev(ctx, torch.rand((m, k // 128), generator=gen, device="cuda"), m, k // 128) for _ in range(2)]
    want = [torch.zeros((m, n), dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    for a, sfa, out in zip(acts, sfas, want):
        dg.fp8_gemm_nt_dev(ctx, a, sfa, b, sfb, out, n)
    ctx.sync()
    torch.cuda.synchronize()
    c = dg.DgContext(0, own_stream=True)      # its own stream goes with the first switch
    streams = [torch.cuda.Stream() for _ in range(2)]
    got = [[torch.zeros((m, n), dtype=torch.bfloat16, device="cuda") for _ in range(20)] for _ in range(2)]
    torch.cuda.synchronize()
    dg.fp8_gemm_nt_dev(c, acts[0], sfas[0], b, sfb, got[0][0], n)
    for i in range(20):
        for s in range(2):
            c.set_stream(streams[s].cuda_stream)
            dg.fp8_gemm_nt_dev(c, acts[s], sfas[s], b, sfb, got[s][i], n)
    torch.cuda.synchronize()
    for s in range(2):
        for out in got[s]:
            assert torch.equal(out, want[s])
    c.set_stream(streams[0].cuda_stream)      # the same stream again
    c.sync()
    c.close()


def test_small_contiguous_groups_get_small_tiles():
    # arenas of 128 rows per group: a group fits one tile of 128 rows and all tiles one wave of the SMs; the arena's padding must not
    # be taken for rows that make a second wave of them.  16 groups of at most 512: pairs are faster by a little if the arena is full and slower
    # by up to 1.7 if it is not, which only the device knows.
    code = """
import torch, deepgemm_rust_b200 as dg
ctx = dg.DgContext(0)
for groups, rows, n, k in ((12, 128, 1152, 3456), (18, 128, 1024, 512), (16, 512, 1152, 2816)):
    m = groups * rows
    a, b = (dg.Fp8Tensor(torch.zeros((r, k), dtype=torch.uint8, device="cuda"), r, k, k) for r in (m, groups * n))
    sfa_t = dg.transform_sf_dev(ctx, torch.ones((m, k // 128), device="cuda"), m, k // 128)
    out = torch.empty((m, n), dtype=torch.bfloat16, device="cuda")
    index = torch.arange(groups, dtype=torch.int32, device="cuda").repeat_interleave(rows)
    dg.m_grouped_fp8_gemm_nt_contiguous_dev(ctx, a, sfa_t, b, torch.ones((groups * n // 128, k // 128), device="cuda"), out, n, index, groups)
ctx.sync()
"""
    run = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300, cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                         env={**os.environ, "DG_PRINT_CONFIGS": "1"})
    assert run.returncode == 0, run.stderr
    lines = [line for line in run.stderr.splitlines() if "f32 scales" in line]
    assert len(lines) == 3 and all("block=128x128 ctas=1" in line for line in lines), lines


@pytest.mark.parametrize("k_blocks", [1, 2, 3, 6])
def test_pair_tiles_of_few_k_blocks(ctx, k_blocks):
    # 48 tiles of 256 x 256 (the choice for this many rows): their K blocks go two a turn, so odd and even counts, one and two among them;
    # rows and columns off the tile grid, and scales whose product leaves the range in which one factor stands for both
    rng = np.random.default_rng(k_blocks)
    m, n, k = 2040, 1400, 128 * k_blocks
    a, b = lcg_e4m3(31, m, k), lcg_e4m3(32, n, k)
    sfa = (rng.random((m, k_blocks)) * 0.03 + 0.001).astype(np.float32)
    sfb = (rng.random((-(-n // 128), k_blocks)) * 0.03 + 0.001).astype(np.float32)
    sfa[300:400] *= 1e-15
    sfb[2:4] *= 1e-15
    a_sf_t = dg.transform_sf_dev(ctx, dev(sfa), m, k_blocks, 1)
    out = torch.zeros((m, n), dtype=torch.bfloat16, device="cuda")
    dg.fp8_gemm_nt_dev(ctx, dg.Fp8Tensor(dev(a), m, k, k), a_sf_t, dg.Fp8Tensor(dev(b), n, k, k), dev(sfb), out, n)
    ctx.sync()
    fa = dev(a).view(torch.float8_e4m3fn).double() * dev(sfa).double().repeat_interleave(128, 1)
    fb = dev(b).view(torch.float8_e4m3fn).double() * dev(sfb).double().repeat_interleave(128, 0)[:n].repeat_interleave(128, 1)
    want, size = fa @ fb.T, fa.abs() @ fb.abs().T
    # one bf16 rounding (8 significant bits: 2^-8 of the value at most), and f32 sums: fewer than 32 roundings of 2^-24 of the terms' magnitudes
    assert bool(((out.double() - want).abs() <= 2.0 ** -8 * want.abs() + 32 * 2.0 ** -24 * size).all())
