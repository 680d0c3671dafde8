// Wide tiles of the first tile family: a CTA pair computes 256 rows x (block_n + block_n2) columns, up to 448, as two UMMAs per
// K step on the same rows of A, each half with an accumulator of its own.
//
// What it is for: large problems, which the power cap bounds.  A 256 x 224 tile takes 30 KB per SM and 128 bytes of K for 448 cycles of
// tensor work: shared memory then has 67 bytes per cycle to take in and 67 to hand to the tensor core (A again for every UMMA), beside a ring
// of three such stages of two slabs that covers the ~1700 cycles of a load only just.  448 columns take 44 KB for 896 cycles, 49 bytes
// per cycle, and four stages last 3584 cycles: the tensor pipe is busy for 93 % of the cycles (5885 x 11232 x 6144), and a flop moves a quarter
// fewer bytes from L2.  There is no second pair of accumulators (2 x 448 columns do not fit TMEM): each half is drained by four warps of
// its own, half 0 while half 1 gets its last UMMAs, and half 1 while the next tile's half 0 gets its first.  bf16 outputs leave TMEM as
// pairs in registers before the first of them is stored (chunk by chunk the next tile waited for the stores: 6861 x 12696 x 3072 240 -> 211 us).
// 4096 x 7168 x 16384 e4m3 395 -> 377 us, 4096 x 7168 x 7168 mxfp4 92.3 -> 84.7, 32 groups of 2048 rows 4096 x 7168 1698 -> 1632.
//
// Roles of the 384-thread CTA (one per SM, persistent, always a pair): warp 0 loads A and its scale words, warp 3 B and its scale words,
// warp 2 re-orders the scale words, warp 1 of rank 0 issues the UMMAs, warps 4-7 store half 0 and warps 8-11 half 1.
// The last wave is made of single halves where that is the shorter one.
#pragma once
#include "dg_gemm_kernel.cuh"

namespace dg {

constexpr uint32_t kWideThreads = 384;
constexpr uint32_t kWideEpiWarps = 8;
constexpr uint32_t kWideMostSubs = 7;     // 32-column chunks of a half

// Walks the tile list of one CTA pair: the first family's order, with the columns of the two halves (0: no second half).  Whole tiles come
// first; what is left for a last wave goes out as single halves where that wave is the shorter for it.
// Grouped layouts: an arena may be sized for far more rows than it holds, and only the device knows how many tiles those make.  Every role counts
// them for itself, a group per lane.  (36 groups of 141 rows, 1216 x 5120, 1.46 waves: 73.9 us with 224-column tiles, 72.7 here.  All tiles of a short launch as
// single halves, with the ring cut into stages of one and the accumulators in turn: 5-25 % slower than whole tiles below two waves.)
struct WideScheduler {
    Scheduler base;
    uint32_t whole_tiles;
    DG_DEVICE explicit WideScheduler(const GemmParams& params) : base(params, 2), whole_tiles(params.whole_tiles) {
        if (params.gemm_type == kGemmNormal) {
            // columns of tiles whose two halves both have something to do
            base.num_n_blocks = (params.n + params.block_n - 1) / params.block_n / 2;
            return;
        }
        uint32_t m_blocks = 0;
        for (base.cur_group = threadIdx.x % 32; base.cur_group < params.num_groups; base.cur_group += 32) {
            base.load_group();
            m_blocks += base.cur_m_blocks;
        }
        const uint32_t tiles = __reduce_add_sync(0xFFFFFFFFu, m_blocks) * base.num_n_blocks, rest = tiles % base.num_workers;
        whole_tiles = 2 * rest <= base.num_workers ? tiles - rest : tiles;
        base.cur_group = 0;
        base.load_group();
    }
    DG_DEVICE uint32_t columns(uint32_t n0, uint32_t most) const {
        // of the tile's part at n0, rounded up to what a UMMA of a pair takes
        const uint32_t left = base.p.n > n0 ? (base.p.n - n0 + 31) / 32 * 32 : 0u;
        return left < most ? left : most;
    }
    DG_DEVICE bool next(Tile& t, uint32_t (&n)[2]) {
        const GemmParams& p = base.p;
        bool whole;
        uint32_t idx, half;
        auto advance = [&]() {
            idx = base.worker + (base.iter++) * base.num_workers;
            whole = idx < whole_tiles;
            half = whole ? 0u : (idx - whole_tiles) & 1;
            if (!whole) idx = whole_tiles + (idx - whole_tiles) / 2;
        };
        if (p.gemm_type != kGemmNormal) {
            do {
                advance();
                if (!base.tile(idx, t)) return false;
                if (half) t.n0 += p.block_n;
                n[0] = columns(t.n0, half ? p.block_n2 : p.block_n);
                n[1] = whole ? columns(t.n0 + p.block_n, p.block_n2) : 0u;
            } while (n[0] == 0);      // the second half of a tile that has none
            return true;
        }
        // (then the halves that have no second one)
        advance();
        const uint32_t paired = base.num_n_blocks, tiles = base.num_m_blocks * paired;
        t.kb0 = 0;
        t.kb1 = (p.k + p.block_k_elems - 1) / p.block_k_elems;
        t.ga = t.gb = t.gd = 0;
        if (idx < tiles) {
            base.dense_tile(idx, t);
            if (half) t.n0 += p.block_n;
        } else {
            const uint32_t mb = (idx - tiles) * 2 + half;
            if (paired * p.tile_n >= p.n || mb >= base.num_m_blocks) return false;
            t.m0 = mb * base.tile_m;
            t.m_end = p.m;
            t.n0 = paired * p.tile_n;
        }
        n[0] = columns(t.n0, p.block_n);
        n[1] = whole ? columns(t.n0 + p.block_n, p.block_n) : 0u;
        return true;
    }
};

template <uint32_t kFmt, uint32_t kOut>
__global__ void __launch_bounds__(kWideThreads, 1)
dg_gemm_wide_kernel(const __grid_constant__ GemmParams p, const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                    const __grid_constant__ CUtensorMap tmap_sfa, const __grid_constant__ CUtensorMap tmap_sfb,
                    const __grid_constant__ CUtensorMap tmap_d) {
    constexpr bool kMXF4 = kFmt == kFmtMxf4;
    constexpr uint32_t kBlockKElems = kMXF4 ? 256 : 128;      // one 128-byte slab of K per stage
    constexpr uint32_t kEpiBufBytes = epilogue_buf_bytes(kOut), kMaxWords = kMXF4 ? 2 : 1;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));

    const uint32_t lane = threadIdx.x % 32, warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x / 32, 0);
    const uint32_t cta_rank = cluster_cta_rank();
    const uint32_t chunks = (p.block_n + 127) / 128;          // 128-row chunks of a half's scale words
    const SfPlan plan_a = sf_plan(p.gran_a, kBlockKElems), plan_b = sf_plan(p.gran_b, kBlockKElems);
    const uint32_t sfa_bytes = 512 * plan_a.words, sfb_bytes = 512 * chunks * plan_b.words, sf_bytes = sfa_bytes + 2 * sfb_bytes;
    constexpr uint32_t a_bytes = kBlockM * kBlockKBytes;
    const uint32_t half_bytes = p.block_n / 2 * kBlockKBytes, b_bytes = 2 * half_bytes;
    const uint32_t num_stages = p.num_stages;

    // shared memory carve-up (every tile base stays 1024-byte aligned)
    uint8_t* smem_a = smem;
    uint8_t* smem_b = smem_a + num_stages * a_bytes;
    uint8_t* smem_epi = smem_b + num_stages * b_bytes;
    uint8_t* smem_sf = smem_epi + kWideEpiWarps * p.epi_bufs * kEpiBufBytes;      // per stage: A's words, half 0's, half 1's
    uint64_t* bar_full = reinterpret_cast<uint64_t*>(smem_sf + num_stages * sf_bytes);
    uint64_t* bar_empty = bar_full + kMaxStages;
    uint64_t* bar_sf_raw = bar_full + 2 * kMaxStages;
    uint64_t* bar_tmem_full = bar_full + 3 * kMaxStages;      // a half's accumulator is complete
    uint64_t* bar_tmem_empty = bar_tmem_full + 2;             // ... and has been read
    uint64_t* bar_tc = bar_tmem_full + 4;                     // the UMMAs of a k-block finished (only with a duty cycle below 100 %)
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar_tmem_full + 5);
    volatile uint32_t* abort_flag = tmem_slot + 1;

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < num_stages; ++s) {
            mbar_init(bar_full + s, 4);       // two producers (their bytes are counted too), and per CTA the scale words or, where none are new, A's producer
            mbar_init(bar_empty + s, 1);
            mbar_init(bar_sf_raw + s, 2);
        }
        for (uint32_t h = 0; h < 2; ++h) {
            mbar_init(bar_tmem_full + h, 1);
            mbar_init(bar_tmem_empty + h, kWideEpiWarps);      // four warps in each CTA
        }
        mbar_init(bar_tc, 1);
        *abort_flag = 0;
        fence_mbar_init();
        tma_prefetch_desc(&tmap_a);
        tma_prefetch_desc(&tmap_b);
        tma_prefetch_desc(&tmap_sfa);
        tma_prefetch_desc(&tmap_sfb);
        tma_prefetch_desc(&tmap_d);
    }
    if (warp == 1) {
        tmem_alloc<2>(tmem_slot, kTmemCols);
        tmem_relinquish<2>();
    }
    tc_fence_before();
    cluster_sync();
    tc_fence_after();
    griddep_wait();
    griddep_launch_dependents();
    const uint32_t tmem_base = __shfl_sync(0xFFFFFFFFu, *tmem_slot, 0);
    const uint32_t tmem_sfa = tmem_base + p.block_n + p.block_n2;
    const uint32_t tmem_sfb = tmem_sfa + 4 * plan_a.words, sfb_half_cols = 4 * chunks * plan_b.words;
    auto new_words = [](const SfPlan& plan, uint32_t kb, const Tile& t) { return (kb & (plan.period - 1)) == 0 || kb == t.kb0; };

    if (warp == 0 || warp == 3) {
        // ------------------------------------------------------------ TMA producers, one warp per operand
        const bool b_side = warp == 3;
        WideScheduler sched(p);
        Tile t;
        uint32_t n[2], stage = 0, phase = 0;
        bool ok = true;
        const uint32_t full_leader = mapa_u32(smem_u32(bar_full), 0);
        const bool leader_lane = elect_one();
        const uint32_t a_tx = a_bytes >> p.tx_shift_a, half_tx = half_bytes >> p.tx_shift_b;
        while (ok && sched.next(t, n)) {
            const int32_t row_a = static_cast<int32_t>(t.m0 + cta_rank * kBlockM);
            // a pair's UMMA takes the first half of its N rows from rank 0
            const int32_t row_b[2] = {static_cast<int32_t>(t.n0 + cta_rank * (n[0] / 2)), static_cast<int32_t>(t.n0 + p.block_n + cta_rank * (n[1] / 2))};
            const uint32_t parts = n[1] ? 2 : 1;
            // a pair's second CTA whose rows all lie past the end of the group loads none: its accumulator rows are never stored
            const bool load_a = static_cast<uint32_t>(row_a) < t.m_end;
            for (uint32_t kb = t.kb0; kb < t.kb1; ++kb) {
                if (!mbar_wait_warp(bar_empty + stage, phase ^ 1, abort_flag, p.status, (b_side ? 0x180 : 0x100) + stage)) { ok = false; break; }
                const bool need_a = new_words(plan_a, kb, t), need_b = new_words(plan_b, kb, t);
                const uint32_t full_addr = full_leader + stage * 8;
                const int32_t kx = static_cast<int32_t>(kb * kBlockKElems);
                uint8_t* sf = smem_sf + stage * sf_bytes;
                if (leader_lane) {
                    if (!b_side) {
                        if (need_a || need_b) {
                            mbar_arrive_expect_tx(bar_sf_raw + stage, need_a ? sfa_bytes : 0u);
                            if (need_a) tma_load_2d(sf, &tmap_sfa, bar_sf_raw + stage, row_a, static_cast<int32_t>(t.ga * p.sf_a_cols + (kb >> plan_a.shift) * plan_a.words));
                        } else {
                            mbar_arrive_cluster(full_addr);      // no new scale words: in place of this CTA's re-ordering warp
                        }
                        if (cta_rank == 0) mbar_arrive_expect_tx(bar_full + stage, (t.m0 + kBlockM < t.m_end ? 2u : 1u) * a_tx);
                        if (load_a) tma_load_3d_2cta(smem_a + stage * a_bytes, &tmap_a, full_addr, kx, row_a, static_cast<int32_t>(t.ga));
                    } else {
                        if (need_a || need_b) {
                            mbar_arrive_expect_tx(bar_sf_raw + stage, need_b ? parts * sfb_bytes : 0u);
                            if (need_b) {
                                const int32_t word = static_cast<int32_t>(t.gb * p.sf_b_cols + (kb >> plan_b.shift) * plan_b.words);
                                for (uint32_t h = 0; h < parts; ++h)
                                    tma_load_2d(sf + sfa_bytes + h * sfb_bytes, &tmap_sfb, bar_sf_raw + stage, static_cast<int32_t>(t.n0 + h * p.block_n), word);
                            }
                        }
                        if (cta_rank == 0) mbar_arrive_expect_tx(bar_full + stage, 2 * parts * half_tx);
                        #pragma unroll
                        for (uint32_t h = 0; h < 2; ++h)
                            if (h < parts)
                                tma_load_3d_2cta(smem_b + stage * b_bytes + h * half_bytes, &tmap_b, full_addr, kx, row_b[h], static_cast<int32_t>(t.gb));
                    }
                }
                __syncwarp();
                if (++stage == num_stages) { stage = 0; phase ^= 1; }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------------------------------------- UMMA issuer
        if (cta_rank == 0) {
            WideScheduler sched(p);
            Tile t;
            uint32_t n[2], stage = 0, phase = 0, tc_phase = 0;
            uint32_t uses[2] = {0, 0};      // tiles that have used each half's accumulator
            bool ok = true;
            const bool leader_lane = elect_one();
            const uint32_t desc_hi = static_cast<uint32_t>(make_smem_desc(0, 0, 1024, 2) >> 32), sf_hi = static_cast<uint32_t>(make_smem_desc(0, 0, 128, 0) >> 32);
            const uint32_t a_lo0 = smem_u32(smem_a) >> 4, b_lo0 = smem_u32(smem_b) >> 4, sf_lo0 = smem_u32(smem_sf) >> 4;
            const bool per128_a = p.gran_a == 128, per128_b = p.gran_b == 128;
            while (ok && sched.next(t, n)) {
                if (!mbar_wait_warp(bar_tmem_empty, (uses[0] & 1) ^ 1, abort_flag, p.status, 0x200)) break;
                ++uses[0];
                uint32_t idesc[2];
                #pragma unroll
                for (uint32_t h = 0; h < 2; ++h) idesc[h] = make_idesc_block_scaled(2 * kBlockM, n[h], kMXF4 ? 1u : p.fmt_a, kMXF4 ? 1u : p.fmt_b);
                for (uint32_t kb = t.kb0; kb < t.kb1; ++kb) {
                    const bool need_a = new_words(plan_a, kb, t), need_b = new_words(plan_b, kb, t), last = kb + 1 == t.kb1;
                    if (!mbar_wait_warp(bar_full + stage, phase, abort_flag, p.status, 0x300 + stage)) { ok = false; break; }
                    tc_fence_after();
                    // operands of both halves, computed by the whole warp ahead of the single-lane regions (warp-uniform values)
                    const uint64_t a_desc = desc64(a_lo0 + stage * (a_bytes >> 4), desc_hi), sf_desc = desc64(sf_lo0 + stage * (sf_bytes >> 4), sf_hi);
                    uint64_t b_desc[2];
                    uint32_t ids[4];
                    #pragma unroll
                    for (uint32_t k = 0; k < 4; ++k) ids[k] = kMXF4 ? idesc_with_sf_ids(0, (k & 1) * 2, (k & 1) * 2) : idesc_with_sf_ids(0, per128_a ? kb & 3 : k, per128_b ? kb & 3 : k);
                    #pragma unroll
                    for (uint32_t h = 0; h < 2; ++h) b_desc[h] = desc64(b_lo0 + stage * (b_bytes >> 4) + h * (half_bytes >> 4), desc_hi);
                    auto issue = [&](uint32_t h) {
                        if (need_b) {
                            #pragma unroll
                            for (uint32_t c = 0; c < 2 * kMaxWords; ++c)
                                if (c < chunks * plan_b.words)
                                    utccp_32x128b_warpx4<2>(tmem_sfb + h * sfb_half_cols + 4 * c, sf_desc + ((sfa_bytes + h * sfb_bytes + c * 512) >> 4));
                        }
                        #pragma unroll
                        for (uint32_t k = 0; k < 4; ++k)
                            umma_block_scaled<2, kMXF4>(tmem_base + h * p.block_n, a_desc + k * (kUmmaKBytes >> 4), b_desc[h] + k * (kUmmaKBytes >> 4), idesc[h] | ids[k],
                                                        tmem_sfa + (kMXF4 ? 4 * (k / 2) : 0u), tmem_sfb + h * sfb_half_cols + (kMXF4 ? 4 * (k / 2) * chunks : 0u),
                                                        kb != t.kb0 || k != 0 ? 1u : 0u);
                    };
                    if (leader_lane) {
                        if (need_a) {
                            #pragma unroll
                            for (uint32_t c = 0; c < kMaxWords; ++c)
                                if (c < plan_a.words) utccp_32x128b_warpx4<2>(tmem_sfa + 4 * c, sf_desc + c * (512 >> 4));
                        }
                        issue(0);
                        if (last) umma_commit_2cta(bar_tmem_full, static_cast<uint16_t>(3));
                    }
                    __syncwarp();
                    if (n[1] != 0) {
                        if (kb == t.kb0) {
                            if (!mbar_wait_warp(bar_tmem_empty + 1, (uses[1] & 1) ^ 1, abort_flag, p.status, 0x280)) { ok = false; break; }
                            ++uses[1];
                            tc_fence_after();
                        }
                        if (leader_lane) {
                            issue(1);
                            if (last) umma_commit_2cta(bar_tmem_full + 1, static_cast<uint16_t>(3));
                        }
                    }
                    if (leader_lane) umma_commit_2cta(bar_empty + stage, static_cast<uint16_t>(3));
                    __syncwarp();
                    if (p.tc_util < 100) {
                        // duty cycle: wait until this k-block's UMMAs are done, then idle for the requested share
                        if (leader_lane) umma_commit_2cta(bar_tc, static_cast<uint16_t>(1));
                        __syncwarp();
                        if (!mbar_wait_warp(bar_tc, tc_phase, abort_flag, p.status, 0x480)) { ok = false; break; }
                        tc_phase ^= 1;
                        duty_cycle_pause(p.tc_util, n[0] + n[1]);
                        __syncwarp();
                    }
                    if (++stage == num_stages) { stage = 0; phase ^= 1; }
                }
            }
        }
        __syncwarp();
    } else if (warp == 2) {
        // -------------------------------------------------- scale words: word r of a 128-word chunk moves to position (r % 32) * 4 + r / 32
        WideScheduler sched(p);
        Tile t;
        uint32_t n[2], stage = 0, phase_bits = 0;
        bool ok = true;
        const uint32_t full_leader = mapa_u32(smem_u32(bar_full), 0);
        while (ok && sched.next(t, n)) {
            const uint32_t chunks_b = chunks * plan_b.words * (n[1] ? 2 : 1);
            for (uint32_t kb = t.kb0; kb < t.kb1; ++kb) {
                const bool need_a = new_words(plan_a, kb, t), need_b = new_words(plan_b, kb, t);
                if (need_a || need_b) {
                    if (!mbar_wait(bar_sf_raw + stage, (phase_bits >> stage) & 1, abort_flag, p.status, 0x500 + stage)) { ok = false; break; }
                    phase_bits ^= 1u << stage;
                    // a batch of chunks at a time, their loads all on the way before the first store
                    constexpr uint32_t kBatch = kMXF4 ? 5 : 6;
                    const uint32_t end = plan_a.words + (need_b ? chunks_b : 0u), base = smem_u32(smem_sf + stage * sf_bytes) + lane * 4;
                    for (uint32_t c0 = need_a ? 0u : plan_a.words; c0 < end; c0 += kBatch) {
                        uint32_t w[kBatch][4];
                        #pragma unroll
                        for (uint32_t i = 0; i < kBatch; ++i) {
                            #pragma unroll
                            for (uint32_t q = 0; q < 4; ++q)
                                if (c0 + i < end) w[i][q] = ld_shared_u32(base + (c0 + i) * 512 + q * 128);
                        }
                        __syncwarp();
                        #pragma unroll
                        for (uint32_t i = 0; i < kBatch; ++i)
                            if (c0 + i < end) st_shared_v4(base + (c0 + i) * 512 + lane * 12, w[i][0], w[i][1], w[i][2], w[i][3]);
                    }
                    fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_cluster(full_leader + stage * 8);
                }
                if (++stage == num_stages) stage = 0;
            }
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------------ epilogue: four warps per half, 32 rows each, 32 columns at a time
        const uint32_t ew = warp % 4, half = (warp - 4) / 4;
        uint8_t* const buf0 = smem_epi + (warp - 4) * p.epi_bufs * kEpiBufBytes;
        const bool leader = elect_one();
        const uint32_t empty_addr = mapa_u32(smem_u32(bar_tmem_empty + half), 0);
        const uint32_t taddr = tmem_base + ((ew * 32) << 16) + half * p.block_n;
        WideScheduler sched(p);
        Tile t;
        uint32_t n[2], phase = 0, buf_idx = 0;
        while (sched.next(t, n)) {
            const uint32_t columns = half ? n[1] : n[0];
            if (columns == 0) continue;
            if (!mbar_wait(bar_tmem_full + half, phase, abort_flag, p.status, 0x600 + half)) break;
            phase ^= 1;
            tc_fence_after();
            const uint32_t row0 = t.m0 + cta_rank * kBlockM + ew * 32, row = row0 + lane, subs = columns / 32, n0 = t.n0 + half * p.block_n;
            auto release = [&]() {
                tc_fence_before();
                __syncwarp();
                if (leader) mbar_arrive_cluster(empty_addr);
            };
            // Stores 32 columns from v: kValues registers of a row, its f32 values or bf16 pairs.
            constexpr uint32_t kValues = kOut == kOutBf16 ? 16 : 32;
            auto store = [&](const uint32_t* v, uint32_t s) {
                const uint32_t col0 = n0 + s * 32;
                if (p.mask_rows && row0 < t.m_end && row0 + 32 > t.m_end) {
                    // this box crosses the end of the group: each lane writes its own row's columns, if the row is valid
                    if (row < t.m_end) {
                        const size_t at = static_cast<size_t>(row) * p.out_ld + col0;
                        #pragma unroll
                        for (uint32_t i = 0; i < 32; ++i) {
                            if (col0 + i >= p.n) break;
                            if constexpr (kOut == kOutBf16) static_cast<uint16_t*>(p.out_ptr)[at + i] = static_cast<uint16_t>(v[i / 2] >> (i % 2 * 16));
                            else static_cast<uint32_t*>(p.out_ptr)[at + i] = v[i];
                        }
                    }
                    return;
                }
                uint8_t* buf = buf0 + buf_idx * kEpiBufBytes;
                // the buffer about to be filled must have been read by the store that used it last
                if (leader) {
                    if (p.epi_bufs == 2) tma_store_wait_read<1>();
                    else tma_store_wait_read<0>();
                }
                __syncwarp();
                // 64- or 128-byte rows, swizzled like the store's tensor map: 16-byte chunk index ^ ((row / 2) % 4) or ^ (row % 8)
                const uint32_t row_addr = smem_u32(buf) + lane * (4 * kValues), turn = kOut == kOutBf16 ? (lane >> 1) & 3 : lane & 7;
                #pragma unroll
                for (uint32_t j = 0; j < kValues / 4; ++j) st_shared_v4(row_addr + ((j ^ turn) << 4), v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
                fence_proxy_async_smem();
                __syncwarp();
                if (leader) {
                    if (col0 < p.n && row0 < t.m_end) {
                        if (p.accumulate) tma_reduce_add_3d(&tmap_d, buf, static_cast<int32_t>(col0), static_cast<int32_t>(row0), static_cast<int32_t>(t.gd));
                        else tma_store_3d(&tmap_d, buf, static_cast<int32_t>(col0), static_cast<int32_t>(row0), static_cast<int32_t>(t.gd));
                    }
                    tma_store_commit();
                }
                buf_idx ^= p.epi_bufs - 1;
            };
            auto scaled = [&](uint32_t x) { return p.has_alpha ? __uint_as_float(x) * p.alpha : __uint_as_float(x); };
            if constexpr (kOut == kOutBf16) {
                // the whole half leaves TMEM as bf16 pairs before the first store: the next tile's UMMAs wait for the accumulator, not for the stores
                uint32_t pairs[kWideMostSubs][16], va[16], vb[16];
                auto pack = [&](uint32_t (&v)[16], uint32_t* to) {
                    tmem_ld_wait_x16(v);
                    #pragma unroll
                    for (uint32_t i = 0; i < 8; ++i) to[i] = pack_bf16x2(scaled(v[2 * i]), scaled(v[2 * i + 1]));
                };
                #pragma unroll
                for (uint32_t s = 0; s < kWideMostSubs; ++s) {
                    if (s < subs) {
                        tmem_ld_32x32b_x16(taddr + s * 32, va);
                        tmem_ld_32x32b_x16(taddr + s * 32 + 16, vb);
                        pack(va, pairs[s]);
                        pack(vb, pairs[s] + 8);
                    }
                }
                release();
                #pragma unroll
                for (uint32_t s = 0; s < kWideMostSubs; ++s)
                    if (s < subs) store(pairs[s], s);
            } else {
                // two register sets: the TMEM load of the next 32 columns is in flight while the current ones are staged
                auto process = [&](uint32_t (&v)[32], uint32_t s) {
                    #pragma unroll
                    for (uint32_t i = 0; i < 32; ++i) v[i] = __float_as_uint(scaled(v[i]));
                    store(v, s);
                };
                uint32_t va[32], vb[32];
                tmem_ld_32x32b_x32(taddr, va);
                for (uint32_t s = 0; s < subs; s += 2) {
                    tmem_ld_wait_x32(va);
                    const bool has_b = s + 1 < subs;
                    if (has_b) tmem_ld_32x32b_x32(taddr + (s + 1) * 32, vb);
                    else release();
                    process(va, s);
                    if (has_b) {
                        tmem_ld_wait_x32(vb);
                        if (s + 2 < subs) tmem_ld_32x32b_x32(taddr + (s + 2) * 32, va);
                        else release();
                        process(vb, s + 1);
                    }
                }
            }
        }
        if (leader) tma_store_wait<0>();
        __syncwarp();
    }

    tc_fence_before();
    cluster_sync();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc<2>(tmem_base, kTmemCols);
    }
}

// Bytes of dynamic shared memory for a configuration (host side).
inline uint32_t gemm_wide_smem_bytes(uint32_t block_n, uint32_t out_kind, uint32_t stages, uint32_t sfa_words, uint32_t sfb_words, uint32_t epi_bufs) {
    const uint32_t per_stage = kBlockM * kBlockKBytes + block_n * kBlockKBytes + 512 * sfa_words + 2 * 512 * ((block_n + 127) / 128) * sfb_words;
    return 1024 + stages * per_stage + kWideEpiWarps * epi_bufs * epilogue_buf_bytes(out_kind) + (3 * kMaxStages + 5) * 8 + 16;
}

}  // namespace dg
