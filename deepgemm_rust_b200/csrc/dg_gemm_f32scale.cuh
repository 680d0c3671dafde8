// FP8 GEMM with f32 scale factors applied exactly (the reference's older "1d2d" contract):
//
//   D[g][m, n] = sum over 128-wide K blocks kb of ( sum_{k in kb} A[m, k] B[n, k] ) * sfa[m, kb] * sfb[n / 128, kb]
//
// which is what deepgemm/src/reference.rs:85-114 (and :133-208 for the grouped layouts) computes.  The tensor core's block
// scaling only takes power-of-two (UE8M0) scales, so an f32 scale with a mantissa cannot ride the UMMA: here every K block
// is multiplied on its own (tcgen05.mma kind::f8f6f4 into one of two TMEM buffers, starting from zero) and the epilogue
// warps fold it into f32 accumulators they keep in registers: acc = fma(block, sfa * sfb, acc).
//
// What bounds it: every K block's partial tile has to leave TMEM (128 lanes x 4 bytes per cycle) and go through one FMA per
// element (128 per cycle and SM), each 256 cycles for 128 x 256 elements, beside 512 cycles of tensor time; a K block takes ~950
// cycles all told.  The two TMEM buffers are what couples the two sides: a buffer is filled (512), seen to be full, read and folded (~470),
// and seen to be empty, ~850 cycles of hand-over in it, once per two K blocks.  The operands of a 128 x 128 tile
// (32 KB for 256 tensor cycles) also arrive slower than the tensor core takes them.  So a CTA pair computes 256 x 256
// (kCtas = 2, kBlockN = 256): 32 KB per CTA for 512 tensor cycles, both TMEM buffers 256 columns wide, and 128 x 256 f32
// accumulators in the registers of eight epilogue warps (the other four give registers back for that).  Problems with too few
// such tiles use 128 x 128 tiles of single CTAs, and cut K into ranges (f32 partial planes summed by dg_splitk_reduce_kernel)
// when even those do not fill the SMs.  4096 x 7168 x 7168: 348 us with 128 x 128 tiles and three rounded operations per
// element, 313 with one FMA, 260 with the pair, 237 with the pair's shorter loop; sixteen epilogue warps of 64 columns (96 registers) spilled
// and took 350.  Four buffers of 128 columns (a half of the pair's tile each, N = 128) were no faster than two; loads of 32 columns, scalar FMAs and
// asking early whether the next block is complete (which holds up the release of the present one) were slower.
// Roles of the 384-thread CTA: warp 0 loads A / B k-blocks with TMA, warp 1 issues the UMMAs, warps 4-11 are the epilogue: each
// owns 32 rows (TMEM quadrant warp % 4) x half of the tile's columns.
#pragma once
#include "dg_gemm_kernel.cuh"

namespace dg {

constexpr uint32_t kF32Threads = 384;     // TMA producer, UMMA issuer, two idle warps, eight epilogue warps

struct F32ScaleParams {
    GemmParams g;              // shape, layout, scheduler inputs (block_n = tile_n = kBlockN, block_k_elems = 128)
    const float* sfa_t;        // activation scales, transposed: [(group * k_blocks + kb) * sfa_stride + row]
    const float* sfb;          // weight scales: [(group * n_blocks128 + n / 128) * k_blocks + kb]
    uint32_t sfa_stride;       // align4(rows per group)
    uint32_t k_blocks, n_blocks128;
};

// kind::f8f6f4 instruction descriptor, e4m3 operands, f32 accumulate, both K-major:
//   [4,6) D format (1 = f32), [7,10) A format (0 = e4m3), [10,13) B format, [17,23) N >> 3, [24,29) M >> 4.
DG_DEVICE uint32_t make_idesc_f8(uint32_t m, uint32_t n) { return (1u << 4) | ((n >> 3) << 17) | ((m >> 4) << 24); }

template <uint32_t kCtas>
DG_DEVICE void umma_f8(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    if constexpr (kCtas == 1)
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
            "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
            : "memory");
    else
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
            "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
            : "memory");
}

// kPartial: the tile is one K range of a split problem and goes to its f32 plane (tmap_d: f32) instead of the bf16 output.
template <uint32_t kCtas, uint32_t kBlockN, bool kPartial>
__global__ void __launch_bounds__(kF32Threads, 1)
dg_gemm_f32scale_kernel(const __grid_constant__ F32ScaleParams q, const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                        const __grid_constant__ CUtensorMap tmap_d) {
    const GemmParams& p = q.g;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t lane = threadIdx.x % 32;
    const uint32_t warp = kCtas == 2 ? __shfl_sync(0xFFFFFFFFu, threadIdx.x / 32, 0) : threadIdx.x / 32;      // pair: known to be the same in every lane
    const uint32_t cta_rank = kCtas == 2 ? cluster_cta_rank() : 0u;
    constexpr uint32_t kLoadN = kBlockN / kCtas;              // weight rows this CTA loads
    constexpr uint32_t kTileA = kBlockM * kBlockKBytes, kTileB = kLoadN * kBlockKBytes;
    constexpr uint32_t kEpiBuf = kPartial ? 4096 : 2048;      // 32 rows x 32 columns
    constexpr uint32_t kEpiWarps = 8, kWarpCols = kBlockN / 2;     // accumulator columns of an epilogue warp
    const uint32_t num_stages = p.num_stages;

    uint8_t* smem_a = smem;
    uint8_t* smem_b = smem_a + num_stages * kTileA;
    uint8_t* smem_epi = smem_b + num_stages * kTileB;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem_epi + kEpiWarps * kEpiBuf);
    uint64_t* bar_full = bars;                               // a k-block's operands landed (pair: both CTAs', on rank 0)
    uint64_t* bar_empty = bars + kMaxStages;
    uint64_t* bar_tmem_full = bars + 2 * kMaxStages;         // a K block's partial tile is complete in TMEM buffer e
    uint64_t* bar_tmem_empty = bar_tmem_full + 2;            // the epilogue warps (of both CTAs) have read buffer e
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar_tmem_empty + 2);
    volatile uint32_t* abort_flag = tmem_slot + 1;

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < num_stages; ++s) {
            mbar_init(bar_full + s, 1);
            mbar_init(bar_empty + s, 1);
        }
        for (uint32_t e = 0; e < 2; ++e) {
            mbar_init(bar_tmem_full + e, 1);
            mbar_init(bar_tmem_empty + e, kEpiWarps * kCtas);
        }
        *abort_flag = 0;
        fence_mbar_init();
        tma_prefetch_desc(&tmap_a);
        tma_prefetch_desc(&tmap_b);
        tma_prefetch_desc(&tmap_d);
    }
    if (warp == 1) {
        tmem_alloc<kCtas>(tmem_slot, 2 * kBlockN);
        tmem_relinquish<kCtas>();
    }
    tc_fence_before();
    if constexpr (kCtas == 2) cluster_sync(); else __syncthreads();
    tc_fence_after();
    griddep_wait();
    griddep_launch_dependents();
    const uint32_t tmem_base = kCtas == 2 ? __shfl_sync(0xFFFFFFFFu, *tmem_slot, 0) : *tmem_slot;

    // 384 threads x 168 registers at launch = 128 x 72 + 256 x 216
    constexpr bool kMoveRegs = kBlockN == 256;
    if (warp < 4) {
        if constexpr (kMoveRegs) setmaxnreg_dec<72>();
        if (warp == 0) {
            // ------------------------------------------------------------ TMA producer
            Scheduler sched(p, kCtas);
            Tile t;
            uint32_t stage = 0, phase = 0;
            bool ok = true;
            const uint32_t full_addr = kCtas == 2 ? mapa_u32(smem_u32(bar_full), 0) : 0u;
            while (ok && sched.next(t)) {
                const int32_t row_a = static_cast<int32_t>(t.m0 + cta_rank * kBlockM), row_b = static_cast<int32_t>(t.n0 + cta_rank * kLoadN);
                for (uint32_t kb = t.kb0; kb < t.kb1; ++kb) {
                    if (!mbar_wait_warp(bar_empty + stage, phase ^ 1, abort_flag, p.status, 0x100 + stage)) { ok = false; break; }
                    if (elect_one()) {
                        const int32_t kx = static_cast<int32_t>(kb * kBlockKBytes);
                        if constexpr (kCtas == 1) {
                            mbar_arrive_expect_tx(bar_full + stage, kTileA + kTileB);
                            tma_load_3d(smem_a + stage * kTileA, &tmap_a, bar_full + stage, kx, row_a, static_cast<int32_t>(t.ga));
                            tma_load_3d(smem_b + stage * kTileB, &tmap_b, bar_full + stage, kx, row_b, static_cast<int32_t>(t.gb));
                        } else {
                            if (cta_rank == 0) mbar_arrive_expect_tx(bar_full + stage, 2 * (kTileA + kTileB));
                            tma_load_3d_2cta(smem_a + stage * kTileA, &tmap_a, full_addr + stage * 8, kx, row_a, static_cast<int32_t>(t.ga));
                            tma_load_3d_2cta(smem_b + stage * kTileB, &tmap_b, full_addr + stage * 8, kx, row_b, static_cast<int32_t>(t.gb));
                        }
                    }
                    __syncwarp();
                    if (++stage == num_stages) { stage = 0; phase ^= 1; }
                }
            }
        } else if (warp == 1 && cta_rank == 0) {
            // ------------------------------------------------------------- UMMA issuer
            Scheduler sched(p, kCtas);
            Tile t;
            uint32_t stage = 0, phase = 0, block = 0;
            constexpr uint32_t kM = kBlockM * kCtas;
            const uint32_t idesc = make_idesc_f8(kM, kBlockN);
            const bool leader_lane = elect_one();
            bool ok = true;
            while (ok && sched.next(t)) {
                for (uint32_t kb = t.kb0; kb < t.kb1; ++kb, ++block) {
                    const uint32_t e = block & 1, buf_phase = (block >> 1) & 1;
                    if (!mbar_wait_warp(bar_tmem_empty + e, buf_phase ^ 1, abort_flag, p.status, 0x200 + e)) { ok = false; break; }
                    if (!mbar_wait_warp(bar_full + stage, phase, abort_flag, p.status, 0x300 + stage)) { ok = false; break; }
                    tc_fence_after();
                    const uint64_t a_desc = make_smem_desc(smem_u32(smem_a + stage * kTileA), 0, 1024, 2);
                    const uint64_t b_desc = make_smem_desc(smem_u32(smem_b + stage * kTileB), 0, 1024, 2);
                    if (leader_lane) {
                        #pragma unroll
                        for (uint32_t k = 0; k < kBlockKBytes / kUmmaKBytes; ++k)
                            umma_f8<kCtas>(tmem_base + e * kBlockN, a_desc + k * (kUmmaKBytes >> 4), b_desc + k * (kUmmaKBytes >> 4), idesc, k != 0 ? 1u : 0u);
                        if constexpr (kCtas == 1) {
                            umma_commit(bar_empty + stage);
                            umma_commit(bar_tmem_full + e);
                        } else {
                            umma_commit_2cta(bar_tmem_full + e, static_cast<uint16_t>(3));
                            umma_commit_2cta(bar_empty + stage, static_cast<uint16_t>(3));
                        }
                    }
                    __syncwarp();
                    if (++stage == num_stages) { stage = 0; phase ^= 1; }
                }
            }
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------------ epilogue
        if constexpr (kMoveRegs) setmaxnreg_inc<216>();
        const uint32_t ew = warp % 4, col_part = (warp - 4) / 4;       // TMEM lane quadrant; which half of the tile's columns
        uint8_t* const buf = smem_epi + (warp - 4) * kEpiBuf;
        const bool leader = elect_one();
        const uint32_t tmem_mine = tmem_base + ((ew * 32) << 16) + col_part * kWarpCols;
        const uint32_t empty_addr = kCtas == 2 ? mapa_u32(smem_u32(bar_tmem_empty), 0) : smem_u32(bar_tmem_empty);
        Scheduler sched(p, kCtas);
        Tile t;
        uint32_t e = 0, phase = 0;
        bool ok = true;
        while (ok && sched.next(t)) {
            const uint32_t row0 = t.m0 + cta_rank * kBlockM + ew * 32, row = row0 + lane, n0 = t.n0 + col_part * kWarpCols;
            // the activation scale of this thread's row for K block kb, and the weight scale of the warp's columns
            const uint32_t nb = n0 / 128 < q.n_blocks128 ? n0 / 128 : q.n_blocks128 - 1;
            const float* next_a = q.sfa_t + (static_cast<size_t>(t.ga) * q.k_blocks + t.kb0) * q.sfa_stride + row;
            const float* next_b = q.sfb + (static_cast<size_t>(t.gb) * q.n_blocks128 + nb) * q.k_blocks + t.kb0;
            const uint32_t stride = q.sfa_stride;
            const bool row_ok = row < t.m_end;
            auto load_scales = [&](float& sa, float& sb) {
                sa = 0.0f;
                if (row_ok) sa = ld_ro(next_a);
                sb = ld_ro(next_b);
                next_a += stride;
                ++next_b;
            };
            float acc[kWarpCols];
            #pragma unroll
            for (uint32_t i = 0; i < kWarpCols; ++i) acc[i] = 0.0f;
            uint32_t left = t.kb1 - t.kb0, va[16], vb[16];
            // One factor for both scales: one rounding fewer than scaling twice.  Where their product leaves the range that keeps full
            // precision (never with scales of quantised data) the block is multiplied by the activation scale first, in place in TMEM:
            // a second path over the accumulators would cost every K block register moves.
            auto in_range = [](float s) { return fabsf(s) >= 1e-30f && fabsf(s) <= 1e30f; };
            auto rescale = [&](uint32_t taddr, float sa) {
                #pragma unroll 1
                for (uint32_t c = 0; c < kWarpCols; c += 16) {
                    tmem_ld_32x32b_x16(taddr + c, va);
                    tmem_ld_wait_x16(va);
                    #pragma unroll
                    for (uint32_t i = 0; i < 16; ++i) va[i] = __float_as_uint(__uint_as_float(va[i]) * sa);
                    tmem_st_32x32b_x16(taddr + c, va);
                }
                tmem_st_wait();
            };
            auto block_done = [&]() { return mbar_wait(bar_tmem_full + e, phase, abort_flag, p.status, 0x600 + e); };
            // the K block in buffer e, whose first 16 columns are already on their way to va
            auto fold_block = [&](uint32_t taddr, float s) {
                // two elements per instruction (packed f32x2: the same IEEE operations, half the issue slots)
                auto fold = [&](uint32_t (&v)[16], uint32_t c) {
                    #pragma unroll
                    for (uint32_t i = 0; i < 16; i += 2) {
                        const float2 r = __ffma2_rn(make_float2(__uint_as_float(v[i]), __uint_as_float(v[i + 1])), make_float2(s, s),
                                                    make_float2(acc[c * 16 + i], acc[c * 16 + i + 1]));
                        acc[c * 16 + i] = r.x;
                        acc[c * 16 + i + 1] = r.y;
                    }
                };
                // the TMEM load of the next 16 columns is in flight while the current ones are folded in
                #pragma unroll
                for (uint32_t c = 0; c < kWarpCols / 16; c += 2) {
                    tmem_ld_wait_x16(va);
                    tmem_ld_32x32b_x16(taddr + (c + 1) * 16, vb);
                    fold(va, c);
                    tmem_ld_wait_x16(vb);
                    if (c + 2 < kWarpCols / 16) {
                        tmem_ld_32x32b_x16(taddr + (c + 2) * 16, va);
                    } else {
                        // the buffer is in registers: hand it back to the UMMA warp
                        tc_fence_before();
                        __syncwarp();
                        if constexpr (kCtas == 1) {
                            if (lane == 0) mbar_arrive(bar_tmem_empty + e);
                        } else if (leader) {
                            mbar_arrive_cluster(empty_addr + e * 8);
                        }
                    }
                    fold(vb, c + 1);
                }
                phase ^= e;
                e ^= 1;
                --left;
            };
            float sa = 0.0f, sb = 0.0f, sa1 = 0.0f, sb1 = 0.0f;      // the scales are fetched two K blocks ahead of their use
            load_scales(sa, sb);
            if (left > 1) load_scales(sa1, sb1);
            if constexpr (kCtas == 2) {
                // With 128 accumulators in registers every instruction beside the 64 FMAs and 8 loads of a K block shows: two K blocks a turn,
                // each with scale registers of its own that are loaded again as soon as they have been used (handed from one name to the
                // next they had to arrive within the turn they were asked for in), addresses in uniform registers, the factor worked out
                // beside the first load.  210 -> 140 instructions per warp and K block.
                auto k_block = [&](float& a, float& b) {
                    if (!block_done()) return false;
                    tc_fence_after();
                    const uint32_t taddr = tmem_mine + e * kBlockN;
                    tmem_ld_32x32b_x16(taddr, va);
                    float s = a * b;
                    if (!__all_sync(0xFFFFFFFFu, in_range(s)) && !__all_sync(0xFFFFFFFFu, in_range(s) || a == 0.0f || b == 0.0f)) {
                        tmem_ld_wait_x16(va);
                        rescale(taddr, a);
                        s = b;
                        tmem_ld_32x32b_x16(taddr, va);
                    }
                    if (left > 2) load_scales(a, b);
                    fold_block(taddr, s);
                    return true;
                };
                while (ok && left != 0) {
                    ok = k_block(sa, sb);
                    if (ok && left != 0) ok = k_block(sa1, sb1);
                }
            } else {
                // 64 accumulators: registers to spare, and the shorter code starts sooner (150 x 1000 x 1152: 8.7 us, 8.9 with the other loop)
                while (left != 0) {
                    float sa2 = 0.0f, sb2 = 0.0f;
                    if (left > 2) load_scales(sa2, sb2);
                    const float both = sa * sb;
                    const bool one_factor = __all_sync(0xFFFFFFFFu, in_range(both) || sa == 0.0f || sb == 0.0f);
                    if (!block_done()) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t taddr = tmem_mine + e * kBlockN;
                    if (!one_factor) rescale(taddr, sa);
                    tmem_ld_32x32b_x16(taddr, va);
                    fold_block(taddr, one_factor ? both : sb);
                    sa = sa1; sb = sb1; sa1 = sa2; sb1 = sb2;
                }
            }
            if (!ok) break;
            // 32 columns at a time through swizzled staging, one TMA store each (rows past the group's end are cut off by the store's
            // 32-row granularity exactly as in the block-scaled kernel)
            #pragma unroll
            for (uint32_t c = 0; c < kWarpCols / 32; ++c) {
                if (lane == 0) tma_store_wait_read<0>();
                __syncwarp();
                if constexpr (kPartial) {
                    const uint32_t row_addr = smem_u32(buf) + lane * 128;
                    #pragma unroll
                    for (uint32_t j = 0; j < 8; ++j)
                        st_shared_v4(row_addr + ((j ^ (lane & 7)) << 4), __float_as_uint(acc[c * 32 + 4 * j]), __float_as_uint(acc[c * 32 + 4 * j + 1]),
                                     __float_as_uint(acc[c * 32 + 4 * j + 2]), __float_as_uint(acc[c * 32 + 4 * j + 3]));
                } else {
                    const uint32_t row_addr = smem_u32(buf) + lane * 64;
                    auto bf16x2 = [&](uint32_t i) { return pack_bf16x2(acc[c * 32 + 2 * i], acc[c * 32 + 2 * i + 1]); };
                    #pragma unroll
                    for (uint32_t j = 0; j < 4; ++j)
                        st_shared_v4(row_addr + ((j ^ ((lane >> 1) & 3)) << 4), bf16x2(4 * j), bf16x2(4 * j + 1), bf16x2(4 * j + 2), bf16x2(4 * j + 3));
                }
                fence_proxy_async_smem();
                __syncwarp();
                const uint32_t col0 = n0 + c * 32;
                if (lane == 0) {
                    if (col0 < p.n && row0 < t.m_end) tma_store_3d(&tmap_d, buf, static_cast<int32_t>(col0), static_cast<int32_t>(row0), static_cast<int32_t>(t.gd));
                    tma_store_commit();
                }
            }
        }
        if (lane == 0) tma_store_wait<0>();
        __syncwarp();
    }

    tc_fence_before();
    if constexpr (kCtas == 2) cluster_sync(); else __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc<kCtas>(tmem_base, 2 * kBlockN);
    }
}

inline uint32_t f32scale_smem_bytes(uint32_t ctas, uint32_t block_n, bool partial, uint32_t stages) {
    return 1024 + stages * (kBlockM + block_n / ctas) * kBlockKBytes + 8 * (partial ? 4096 : 2048) + (2 * kMaxStages + 4) * 8 + 16;
}

}  // namespace dg
