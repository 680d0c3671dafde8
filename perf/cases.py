"""Workloads of the library's public entry points: what a serving or training program runs on one GPU.

A case is a dict of plain values; its "path" names the call sequence it takes:

  linear    bf16 activations -> e4m3 quantiser -> dense block-scaled GEMM (a decode-time projection)
  dense     dense block-scaled GEMM on operands that are already quantised (e4m3, packed e2m1, or one of each)
  f32scale  f32 activation scales -> transposed layout -> FP8 GEMM with exact f32 scales
  grouped   contiguous m-grouped GEMM over a routed arena, from its m_indices
  masked    masked m-grouped GEMM with e4m3 output and per-32-column scales
  moe       a whole MoE layer on one rank: quantise, dispatch, gate/up, silu * up + quantise, down, combine
  quantise  bf16 -> e4m3 or packed e2m1 with packed UE8M0 scales
"""
import math

import torch

import deepgemm_rust_b200 as dg
from deepgemm_rust_b200.moe_ep import PeerExpertParallel

ALIGNMENT = 128     # rows every group of the contiguous layout starts at a multiple of (the library's default)


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # one decode step of a few sequences through a small projection: launches and host time
        {"name": "linear_decode_8", "path": "linear", "m": 8, "n": 2112, "k": 7168},
        # decode batch of 128 on the largest projection: weights are read once
        {"name": "dense_decode_128", "path": "dense", "m": 128, "n": 7168, "k": 16384, "a_bits": 8, "b_bits": 8, "out": "bf16", "alpha": False},
        # a prompt of odd length, f32 scores scaled by alpha
        {"name": "dense_ragged_f32", "path": "dense", "m": 777, "n": 4096, "k": 7168, "a_bits": 8, "b_bits": 8, "out": "f32", "alpha": True},
        # prefill of 4096 tokens through the largest projection
        {"name": "dense_prefill_4096", "path": "dense", "m": 4096, "n": 7168, "k": 16384, "a_bits": 8, "b_bits": 8, "out": "bf16", "alpha": False},
        # prefill with both operands in MXFP4
        {"name": "dense_mxfp4_4096", "path": "dense", "m": 4096, "n": 7168, "k": 7168, "a_bits": 4, "b_bits": 4, "out": "bf16", "alpha": False},
        # FP8 activations on FP4 weights, a medium batch
        {"name": "dense_fp8xfp4_256", "path": "dense", "m": 256, "n": 7168, "k": 7168, "a_bits": 8, "b_bits": 4, "out": "bf16", "alpha": False},
        # the older f32-scale interface at prefill size
        {"name": "f32scale_4096", "path": "f32scale", "m": 4096, "n": 7168, "k": 7168},
        # gate/up GEMM of one rank of eight: 32 local experts, 65 536 routed rows
        {"name": "grouped_32_experts", "path": "grouped", "experts": 32, "tokens": 8192, "topk": 8, "n": 4096, "k": 7168},
        # masked decode GEMM, 32 local experts of at most 256 rows each
        {"name": "masked_decode_32", "path": "masked", "experts": 32, "slot": 256, "n": 4096, "k": 7168},
        # a decode step of an MoE layer: 128 tokens, 32 experts in fixed slots
        {"name": "moe_decode_128", "path": "moe", "experts": 32, "topk": 8, "tokens": 128, "hidden": 7168, "inter": 2048, "slot": 128},
        # prefill of an MoE layer whose 256 experts all live on this GPU
        {"name": "moe_prefill_8192", "path": "moe", "experts": 256, "topk": 8, "tokens": 8192, "hidden": 7168, "inter": 2048, "slot": 0},
        # activation quantiser at prefill size
        {"name": "quantise_4096", "path": "quantise", "rows": 4096, "k": 7168, "bits": 8, "gran": 128},
    ]


def _spread(rng, lo, hi, step=1):
    """A multiple of `step` from [lo, hi], even over the logarithm."""
    x = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(hi // step, max(-(-lo // step), round(x / step))) * step


def draw(rng):
    path = rng.choice(["linear", "linear", "dense", "dense", "dense", "f32scale", "grouped", "masked", "moe", "moe", "quantise"])
    if path == "linear":
        return {"path": path, "m": _spread(rng, 1, 64), "n": _spread(rng, 512, 24576, 8), "k": _spread(rng, 1024, 16384, 512)}
    if path == "dense":
        a_bits, b_bits = rng.choice([(8, 8), (8, 8), (8, 8), (4, 4), (8, 4)])
        out, alpha = rng.choice([("bf16", False), ("bf16", False), ("f32", True)])
        return {"path": path, "m": _spread(rng, 16, 8192), "n": _spread(rng, 512, 16384, 8), "k": _spread(rng, 1024, 16384, 512),
                "a_bits": a_bits, "b_bits": b_bits, "out": out, "alpha": alpha}
    if path == "f32scale":
        return {"path": path, "m": _spread(rng, 64, 8192), "n": _spread(rng, 512, 8192, 8), "k": _spread(rng, 1024, 8192, 128)}
    if path == "grouped":
        return {"path": path, "experts": _spread(rng, 8, 64), "tokens": _spread(rng, 256, 8192), "topk": 8,
                "n": _spread(rng, 1024, 7168, 64), "k": _spread(rng, 1024, 7168, 512)}
    if path == "masked":
        return {"path": path, "experts": _spread(rng, 4, 64), "slot": _spread(rng, 64, 512, 4), "n": _spread(rng, 1024, 7168, 128),
                "k": _spread(rng, 1024, 7168, 512)}
    if path == "moe":
        experts, hidden, inter = _spread(rng, 16, 128), _spread(rng, 2048, 7168, 512), _spread(rng, 1024, 2048, 512)
        if rng.random() < 0.5:
            return {"path": path, "experts": experts, "topk": 8, "tokens": _spread(rng, 16, 256), "hidden": hidden, "inter": inter, "slot": 256}
        return {"path": path, "experts": experts, "topk": 8, "tokens": _spread(rng, 256, 8192), "hidden": hidden, "inter": inter, "slot": 0}
    bits, gran = rng.choice([(8, 128), (8, 128), (8, 32), (4, 32)])
    return {"path": path, "rows": _spread(rng, 16, 16384), "k": _spread(rng, 1024, 16384, 512), "bits": bits, "gran": gran}


# --------------------------------------------------------------------------------------- inputs in hand before a call
_context = None


def _ctx():
    """One context for the process, as a program has."""
    global _context
    if _context is None:
        _context = dg.DgContext(0)
    return _context


def _bf16(gen, rows, k, scale=1.0):
    x = torch.randn((rows, k), generator=gen, device="cuda", dtype=torch.bfloat16)
    return x if scale == 1.0 else x.mul_(scale)


def _operand(ctx, x, rows_per_group, bits, gran=128, groups=1):
    """x quantised by the library: a batch of `groups` equal groups, declared with `rows_per_group` rows."""
    rows, k = x.shape
    if bits == 4:
        data, sf = dg.cast_bf16_to_fp4_packed_sf_dev(ctx, x, k, rows, k, groups, dg.SF_RULE_RANGE_FIT)
        return dg.LpOperand(data, sf, rows_per_group, k, k, 4, 32)
    data, sf = dg.cast_bf16_to_fp8_sf_dev(ctx, x, k, rows, k, gran, groups)
    return dg.LpOperand(data, sf, rows_per_group, k, k, 8, gran)


def _route(gen, tokens, experts, topk):
    """Top-k experts and their weights for every token, from N(0, 1) router logits."""
    logits = torch.randn((tokens, experts), generator=gen, device="cuda")
    weights, idx = torch.softmax(logits, -1).topk(topk, dim=-1)
    return weights.contiguous(), idx.to(torch.int32).contiguous()


class _Exchange(PeerExpertParallel):
    """The exchange buffers of a layer, given back with the state that holds them."""

    def __del__(self):
        if getattr(self, "_base", None) is not None:
            self.close()


def prepare(case, seed):
    ctx = _ctx()
    gen = torch.Generator(device="cuda").manual_seed(seed)
    path = case["path"]
    s = {"case": case, "ctx": ctx}
    if path == "linear":
        m, n, k = case["m"], case["n"], case["k"]
        s["x"] = _bf16(gen, m, k)
        s["w"] = _operand(ctx, _bf16(gen, n, k, k ** -0.5), n, 8)
        s["d"] = torch.zeros((m, n), dtype=torch.bfloat16, device="cuda")
        s["out"] = dg.Sm100Out.Bf16(s["d"], n)
    elif path == "dense":
        m, n, k = case["m"], case["n"], case["k"]
        f32 = case["out"] == "f32"
        s["a"] = _operand(ctx, _bf16(gen, m, k), m, case["a_bits"])
        s["w"] = _operand(ctx, _bf16(gen, n, k, k ** -0.5), n, case["b_bits"])
        s["d"] = torch.zeros((m, n), dtype=torch.float32 if f32 else torch.bfloat16, device="cuda")
        s["out"] = dg.Sm100Out.F32(s["d"], n) if f32 else dg.Sm100Out.Bf16(s["d"], n)
        s["epilogue"] = dg.Sm100Epilogue(alpha=0.125) if case["alpha"] else None
    elif path == "f32scale":
        m, n, k = case["m"], case["n"], case["k"]
        x, w = _bf16(gen, m, k).float(), _bf16(gen, n, k, k ** -0.5).float()
        sfa = x.view(m, k // 128, 128).abs().amax(-1).clamp_min_(1e-10) / 448.0
        xq = (x.view(m, k // 128, 128) / sfa.unsqueeze(-1)).to(torch.float8_e4m3fn).view(torch.uint8).view(m, k)
        tiles = -(-n // 128)
        padded = torch.zeros((tiles * 128, k), device="cuda")
        padded[:n] = w
        padded = padded.view(tiles, 128, k // 128, 128)
        sfb = padded.abs().amax((1, 3)).clamp_min_(1e-10) / 448.0
        wq = (padded / sfb[:, None, :, None]).to(torch.float8_e4m3fn).view(torch.uint8).view(tiles * 128, k)[:n].contiguous()
        s["sfa"], s["sfb"] = sfa.contiguous(), sfb.contiguous()
        s["a"], s["b"] = dg.Fp8Tensor(xq, m, k, k), dg.Fp8Tensor(wq, n, k, k)
        s["d"] = torch.zeros((m, n), dtype=torch.bfloat16, device="cuda")
    elif path == "grouped":
        experts, n, k = case["experts"], case["n"], case["k"]
        _, idx = _route(gen, case["tokens"], experts, case["topk"])
        sizes = torch.bincount(idx.view(-1).long(), minlength=experts).tolist()
        starts, total = [], 0
        for size in sizes:
            starts.append(total)
            total += -(-size // ALIGNMENT) * ALIGNMENT
        total = case["tokens"] * case["topk"] + experts * ALIGNMENT     # the arena is sized for any routing of these tokens
        m_indices = torch.full((total,), -1, dtype=torch.int32)
        for e, (start, size) in enumerate(zip(starts, sizes)):
            m_indices[start:start + size] = e
        s["m_indices"] = m_indices.cuda()
        s["a"] = _operand(ctx, _bf16(gen, total, k), total, 8)
        s["w"] = _operand(ctx, _bf16(gen, experts * n, k, k ** -0.5), experts * n, 8, groups=experts)
        s["d"] = torch.zeros((total, n), dtype=torch.bfloat16, device="cuda")
        s["out"] = dg.Sm100Out.Bf16(s["d"], n)
    elif path == "masked":
        experts, slot, n, k = case["experts"], case["slot"], case["n"], case["k"]
        s["masked_m"] = torch.randint(0, slot + 1, (experts,), generator=gen, device="cuda", dtype=torch.int32)
        s["a"] = _operand(ctx, _bf16(gen, experts * slot, k), slot, 8, groups=experts)
        s["w"] = _operand(ctx, _bf16(gen, experts * n, k, k ** -0.5), experts * n, 8, groups=experts)
        s["d"] = torch.zeros((experts * slot, n), dtype=torch.uint8, device="cuda")
        s["sfd"] = torch.zeros(n // 128 * experts * dg.sf_aligned_rows(slot), dtype=torch.int32, device="cuda")
        s["out"] = dg.Sm100Out.Fp8(s["d"], n, s["sfd"])
    elif path == "moe":
        experts, hidden, inter, tokens, slot = case["experts"], case["hidden"], case["inter"], case["tokens"], case["slot"]
        s["x"] = _bf16(gen, tokens, hidden)
        s["topw"], s["topi"] = _route(gen, tokens, experts, case["topk"])
        s["gate_up"] = _operand(ctx, _bf16(gen, experts * 2 * inter, hidden, hidden ** -0.5), experts * 2 * inter, 8, groups=experts)
        s["down"] = _operand(ctx, _bf16(gen, experts * hidden, inter, inter ** -0.5), experts * hidden, 8, groups=experts)
        ex = s["exchange"] = _Exchange(ctx, experts, case["topk"], tokens, hidden, hidden, alignment=ALIGNMENT, slot_rows=slot)
        rows = experts * slot if slot else ex.capacity
        groups = experts if slot else 1
        h = torch.zeros((rows, 2 * inter), dtype=torch.bfloat16, device="cuda")
        act, act_sf = torch.zeros((rows, inter), dtype=torch.uint8, device="cuda"), dg.alloc_sf(ctx, rows, inter, 128, groups)
        s["h"], s["act"], s["rows"], s["groups"] = h, (act, act_sf), rows, groups
        s["h_out"] = dg.Sm100Out.Bf16(h, 2 * inter)
        s["act_op"] = dg.LpOperand(act, act_sf, slot or rows, inter, inter, 8, 128)
        s["y_out"] = dg.Sm100Out.Bf16(ex.result, hidden)
    else:
        s["x"] = _bf16(gen, case["rows"], case["k"])
    return s


# ---------------------------------------------------------------------------------------------------- one pass
def run(s):
    case, ctx = s["case"], s["ctx"]
    path = case["path"]
    if path == "linear":
        m, k = case["m"], case["k"]
        xq, xsf = dg.cast_bf16_to_fp8_sf_dev(ctx, s["x"], k, m, k, 128)
        dg.fp8_fp4_gemm_dev(ctx, dg.LpOperand(xq, xsf, m, k, k), s["w"], s["out"])
        return s["d"]
    if path == "dense":
        dg.fp8_fp4_gemm_dev(ctx, s["a"], s["w"], s["out"], s["epilogue"])
        return s["d"]
    if path == "f32scale":
        sfa_t = dg.transform_sf_dev(ctx, s["sfa"], case["m"], case["k"] // 128)
        dg.fp8_gemm_nt_dev(ctx, s["a"], sfa_t, s["b"], s["sfb"], s["d"], case["n"])
        return s["d"]
    if path == "grouped":
        dg.m_grouped_fp8_fp4_gemm_contiguous_dev(ctx, s["a"], s["m_indices"], s["w"], s["out"], case["experts"])
        return s["d"]
    if path == "masked":
        dg.m_grouped_fp8_fp4_gemm_masked_dev(ctx, s["a"], s["masked_m"], s["w"], s["out"], case["experts"], case["slot"] // 2)
        return s["d"], s["sfd"]
    if path == "moe":
        return _moe_layer(s)
    rows, k = case["rows"], case["k"]
    if case["bits"] == 4:
        return dg.cast_bf16_to_fp4_packed_sf_dev(ctx, s["x"], k, rows, k, 1, dg.SF_RULE_RANGE_FIT)
    return dg.cast_bf16_to_fp8_sf_dev(ctx, s["x"], k, rows, k, case["gran"])


def _moe_layer(s):
    case, ctx, ex = s["case"], s["ctx"], s["exchange"]
    experts, hidden, inter, tokens = case["experts"], case["hidden"], case["inter"], case["tokens"]
    xq, xsf = dg.cast_bf16_to_fp8_sf_dev(ctx, s["x"], hidden, tokens, hidden, 128)
    a, groups = ex.dispatch(s["topi"], xq, xsf)
    if case["slot"]:
        expected = max(1, tokens * case["topk"] // experts)
        dg.m_grouped_fp8_fp4_gemm_masked_dev(ctx, a, groups, s["gate_up"], s["h_out"], experts, expected)
        dg.silu_mul_cast_fp8_sf_dev(ctx, s["h"], 2 * inter, s["rows"], inter, 128, s["groups"], out=s["act"])
        dg.m_grouped_fp8_fp4_gemm_masked_dev(ctx, s["act_op"], groups, s["down"], s["y_out"], experts, expected)
    else:
        dg.m_grouped_fp8_fp4_gemm_contiguous_ends_dev(ctx, a, groups, s["gate_up"], s["h_out"], experts)
        dg.silu_mul_cast_fp8_sf_dev(ctx, s["h"], 2 * inter, s["rows"], inter, 128, s["groups"], live_rows=ex.totals, out=s["act"])
        dg.m_grouped_fp8_fp4_gemm_contiguous_ends_dev(ctx, s["act_op"], groups, s["down"], s["y_out"], experts)
    return ex.combine(s["topw"])


# ----------------------------------------------------------------------------- what a pass cannot do without
def _operand_bytes(rows, k, bits, gran=128):
    gran = 32 if bits == 4 else gran
    return rows * (k * bits / 8 + 4 * -(-k // (4 * gran)))


def work(case):
    path = case["path"]
    if path == "linear":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 2 * m * k + _operand_bytes(n, k, 8) + 2 * m * n, "flops": 2 * m * n * k}
    if path == "dense":
        m, n, k = case["m"], case["n"], case["k"]
        out = m * n * (4 if case["out"] == "f32" else 2)
        return {"bytes": _operand_bytes(m, k, case["a_bits"]) + _operand_bytes(n, k, case["b_bits"]) + out, "flops": 2 * m * n * k}
    if path == "f32scale":
        m, n, k = case["m"], case["n"], case["k"]
        scales = 4 * (m + -(-n // 128)) * (k // 128)
        return {"bytes": (m + n) * k + scales + 2 * m * n, "flops": 2 * m * n * k}
    if path == "grouped":
        rows, n, k = case["tokens"] * case["topk"], case["n"], case["k"]
        return {"bytes": _operand_bytes(rows, k, 8) + _operand_bytes(case["experts"] * n, k, 8) + 2 * rows * n + 4 * rows, "flops": 2 * rows * n * k}
    if path == "masked":
        rows, n, k = case["experts"] * case["slot"] / 2, case["n"], case["k"]     # expected valid rows
        return {"bytes": _operand_bytes(rows, k, 8) + _operand_bytes(case["experts"] * n, k, 8) + _operand_bytes(rows, n, 8, 32), "flops": 2 * rows * n * k}
    if path == "moe":
        experts, tokens, hidden, inter = case["experts"], case["tokens"], case["hidden"], case["inter"]
        rows = tokens * case["topk"]
        touched = experts * (1 - (1 - case["topk"] / experts) ** tokens)          # experts that get a row
        weights = touched * (_operand_bytes(2 * inter, hidden, 8) + _operand_bytes(hidden, inter, 8))
        return {"bytes": 4 * tokens * hidden + weights + 8 * rows, "flops": 6 * rows * inter * hidden}
    rows, k = case["rows"], case["k"]
    return {"bytes": 2 * rows * k + _operand_bytes(rows, k, case["bits"], case["gran"]), "flops": 0}


def tolerance(case):
    """Products of e4m3 / e2m1 values and power-of-two scales are exact in f32; what may differ between two correct
    implementations is the order of the f32 sums and the rounding to the output type that follows."""
    path = case["path"]
    if path == "quantise":
        return "exact"
    if path == "dense" and case["out"] == "f32":
        return {"rel": 1e-5, "max": 1e-3}
    if path == "masked":
        return {"differ": 1e-3}      # e4m3 codes and scale exponents that sit on a rounding tie of the sum
    if path == "moe":
        return {"rel": 1e-2, "max": 0.1}        # an e4m3 rounding of the activation that falls the other way is 2^-4 of that element
    return {"rel": 4e-3, "max": 2e-2}            # one bf16 rounding is at most 2^-8 of the value
