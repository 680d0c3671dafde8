// Second tile family of the block-scaled GEMM: the WEIGHT rows ride the UMMA M dimension (128 per CTA, 256 per CTA pair) and
// the activation rows the UMMA N dimension, whose width follows the rows a tile really has.
//
// What it is for: problems with few activation rows per weight matrix (expert groups of up to a few hundred rows).  The first
// family pads a group to 128 or 256 rows on UMMA M; here a group of r rows costs r rounded up to 32 columns of tensor work, and
// every weight byte passes through an SM once per tile: above 256 rows (288 by the rule, up to 320 where DG_BLOCK_N asks for it) a
// k-step is two UMMAs (256 + the rest) on the same weights.  A group of R rows is cut into ceil(R / BLOCK_N) tiles of about equal
// height, because a narrow tile is bound by its weight stream and by the issue of its instructions (~450 cycles per 128 bytes of
// K), not by its tensor time.
//
// Roles of the 384-thread CTA (one per SM, persistent): warp 0 loads weights, warp 3 activations, warp 2 loads and re-orders the
// scale words into a ring of its own, warp 1 issues the UMMAs, warps 4-11 are the epilogue: two per TMEM quadrant, taking turns
// at its 32-row chunks (a chunk is a chain of dependent steps, ~1000 cycles; with short K one warp could not keep up).  The
// accumulator holds D transposed (TMEM lane = output column, TMEM column = output row):
//   bf16  tcgen05.ld.16x256b gives every lane column pairs of one lane row, stmatrix.trans turns 8 x 8 blocks round on the way
//         through shared memory, 64 bytes of a row per four lanes
//   f32   lane-per-column loads, 128 bytes of a row per store instruction
//   e4m3  as bf16 into shared memory, then a row of 32 columns (a scale block) per lane
// Two accumulators of up to 320 columns and the scale columns do not fit 512 TMEM columns side by side, so the second one starts
// at acc_stride < block_n: tiles wider than that overlap the other buffer.  The epilogue drains those columns first (buffer 0
// from its last 32 columns down, buffer 1 upwards) and reports them separately, so that the next tile's UMMAs start while the
// rest is still being stored; narrower tiles never wait.
// K ranges, one per CTA (pair), for dense problems where DG_SWAP=1 pins this family (by its rule it gets none): every range writes
// its f32 accumulator to a workspace in the epilogue's register order, the last range of a tile to arrive (a counter per tile)
// adds them in range order and stores the tile.  Nobody waits for anybody, the sum does not depend on who is last, and there is no second launch.
#pragma once
#include "dg_gemm_kernel.cuh"
#include "dg_ring.cuh"

namespace dg {

constexpr uint32_t kSwapThreads = 384;
constexpr uint32_t kSwapEpiWarps = 8;
constexpr uint32_t kSwapMaxRows = 320;    // of a tile
constexpr uint32_t kSwapTailRows = 16;    // per CTA and box, for the rows of a tile beyond 256
constexpr uint32_t kSwapSfSlots = 4;      // ring of scale words, fetched ahead of the k-block that needs them

struct SwapTile {
    uint32_t m0;               // first weight row (output column)
    uint32_t n0, valid, n;     // first activation row, rows of the tile, UMMA N of all its parts (rows rounded up)
    uint32_t rows;             // rows that are written
    uint32_t ga, gb, gd;       // group coordinate of the weights, of the activations and of D
    uint32_t kb0, kb1;         // k-block range
    uint32_t index, split;     // output tile and K range
};

// Walks the tile list of one CTA (pair); every role runs its own copy and sees the same sequence.  kTable: the kernel keeps a table of
// the groups in shared memory.
template <bool kTable>
struct SwapScheduler {
    const GemmParams& p;
    bool grouped;
    uint32_t step, tile_m, worker, num_workers, num_m_blocks, total_kb, iter;
    uint32_t cur_group, cum_begin, row_start, rows, tile_rows, num_tiles;
    const uint4* table;      // shared memory: (row_start, rows, num_tiles, tile_rows) of the first table_groups groups

    DG_DEVICE SwapScheduler(const GemmParams& params, uint32_t ctas, uint32_t block_k_elems) : p(params) {
        tile_m = kBlockM * ctas;
        worker = blockIdx.x / ctas;
        num_workers = gridDim.x / ctas;
        num_m_blocks = (p.m + tile_m - 1) / tile_m;
        total_kb = (p.k + block_k_elems - 1) / block_k_elems;
        iter = 0;
        cur_group = 0;
        cum_begin = 0;
        row_start = 0;
        grouped = p.gemm_type == kGemmContiguous || p.gemm_type == kGemmMasked;
        step = grouped ? 32 : 16 * ctas;
        if (!grouped) set_rows(p.n);
    }
    // What needs the group table: call once, after groups_ready().  The constructor belongs before it, where its time is hidden.
    DG_DEVICE void start(const uint4* group_table) {
        if constexpr (kTable) table = group_table;
        if (grouped) load_group();
    }
    DG_DEVICE void set_rows(uint32_t r) {
        // tiles of one range of rows meet at multiples of 32 rows (16 for BLOCK_N = 16)
        rows = r;
        const uint32_t grid = p.block_n < 32 ? 16u : 32u, most = p.block_n / grid * grid;
        num_tiles = r <= p.block_n ? (r != 0 ? 1u : 0u) : (r + most - 1) / most;
        tile_rows = num_tiles > 1 ? ((r + num_tiles - 1) / num_tiles + grid - 1) / grid * grid : r;
    }
    // rows and tiles of a group, from global memory
    DG_DEVICE void read_group(uint32_t g) {
        if (p.gemm_type == kGemmContiguous) {
            const uint32_t prev_end = g == 0 ? 0u : ld_ro(p.grouped_layout + g - 1);
            uint32_t end = ld_ro(p.grouped_layout + g);
            end = end < p.n ? end : p.n;
            row_start = (prev_end + p.mk_alignment - 1) / p.mk_alignment * p.mk_alignment;
            set_rows(end > row_start ? end - row_start : 0u);
        } else {
            const int32_t valid = static_cast<int32_t>(ld_ro(p.grouped_layout + g));
            set_rows(valid <= 0 ? 0u : (static_cast<uint32_t>(valid) < p.n ? static_cast<uint32_t>(valid) : p.n));
        }
    }
    DG_DEVICE void load_group() {
        if (cur_group >= p.num_groups) return;
        if constexpr (kTable) {
            if (cur_group < p.table_groups) {
                const uint4 x = table[cur_group];
                row_start = x.x;
                rows = x.y;
                num_tiles = x.z;
                tile_rows = x.w;
                return;
            }
        }
        read_group(cur_group);
    }
    DG_DEVICE bool next(SwapTile& t) {
        uint32_t idx = worker + (iter++) * num_workers;
        t.split = 0;
        t.kb0 = 0;
        t.kb1 = total_kb;
        uint32_t nb, mb;
        if (p.gemm_type == kGemmNormal || p.gemm_type == kGemmBatched) {
            if (p.num_splits > 1) {
                // K ranges of one tile next to each other; k-blocks dealt out evenly, no range empty
                t.split = idx % p.num_splits;
                idx /= p.num_splits;
                t.kb0 = t.split * total_kb / p.num_splits;
                t.kb1 = (t.split + 1) * total_kb / p.num_splits;
            }
            const uint32_t per_group = num_m_blocks * num_tiles;
            if (idx >= per_group * p.num_groups) return false;
            const uint32_t g = idx / per_group, r = idx - g * per_group;
            nb = r / num_m_blocks;
            mb = r - nb * num_m_blocks;      // weight blocks fastest: the tiles in flight share the activation rows
            t.ga = t.gb = t.gd = g;
        } else {
            while (true) {
                if (cur_group >= p.num_groups) return false;
                const uint32_t end = cum_begin + num_tiles * num_m_blocks;
                if (idx < end) break;
                cum_begin = end;
                ++cur_group;
                load_group();
            }
            const uint32_t in_group = idx - cum_begin;
            nb = in_group / num_m_blocks;
            mb = in_group - nb * num_m_blocks;
            t.ga = cur_group;
            t.gb = t.gd = p.gemm_type == kGemmContiguous ? 0u : cur_group;
        }
        t.index = idx;
        t.m0 = mb * tile_m;
        t.n0 = row_start + nb * tile_rows;
        const uint32_t left = rows - nb * tile_rows;
        t.valid = left < tile_rows ? left : tile_rows;
        t.n = (t.valid + step - 1) / step * step;
        // like the first family's 32-row store boxes, a group's last rows go out with what follows them up to a multiple of 32: rows of
        // the group's own padding (mask_rows: the neighbour may start there, nothing but valid rows)
        t.rows = t.valid;
        if (grouped && p.mask_rows == 0) t.rows = t.n < p.n - t.n0 ? t.n : p.n - t.n0;
        return true;
    }
};

// 16 TMEM lanes x 32 consecutive 32-bit columns in the layout of 8 x 8 matrix fragments: register 4 j + i of lane t holds TMEM
// lane t / 4 + 8 (i / 2), column 8 j + 2 (t % 4) + i % 2.
DG_DEVICE void tmem_ld_16x256b_x4(uint32_t taddr, uint32_t* r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
          "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
// Four 8 x 8 blocks of 16-bit elements, each stored transposed: lane 8 q + i gives the address of row i of block q.
DG_DEVICE void stmatrix_x4_trans(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
DG_DEVICE uint4 ld_shared_v4(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
    return v;
}
DG_DEVICE uint32_t ld_shared_u16(uint32_t addr) {
    uint16_t v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr) : "memory");
    return v;
}

// staging bytes of one epilogue warp: 32 output rows x 32 columns (f32 goes out straight from registers)
constexpr uint32_t swap_epi_buf_bytes(uint32_t out_kind) { return out_kind == kOutF32 ? 0u : 2048u; }

// Kernels with a group table: the form that the grouped layouts get by the rule.  In the others, which the dense problems get, its code
// costs 2 % (5 x 17888 x 9216: 31.0 -> 31.8 us).
__host__ __device__ constexpr bool swap_has_table(uint32_t ctas, uint32_t halves) { return ctas == 2 && halves == 1; }

// Activation rows of a stage, per CTA and slab: the first 256 rows of a tile, and the rows beyond.
__host__ __device__ inline uint32_t swap_main_rows(uint32_t block_n, uint32_t ctas) { return (block_n < 256 ? block_n : 256) / ctas; }
__host__ __device__ inline uint32_t swap_tail_rows(uint32_t block_n, uint32_t ctas) {
    return block_n <= 256 ? 0u : ((block_n - 256) / ctas + kSwapTailRows - 1) / kSwapTailRows * kSwapTailRows;
}
// A tile with at most this many rows per CTA takes the smaller box.
__host__ __device__ inline uint32_t swap_part_rows(uint32_t main_rows) { return main_rows >= 64 ? (main_rows / 2 + 7) / 8 * 8 : main_rows; }

// tmap_b brings swap_main_rows rows of the activations (and, with wide_k, both slabs of a stage), tmap_b_part swap_part_rows of
// one slab, tmap_b_tail kSwapTailRows of one slab.
template <uint32_t kFmt, uint32_t kOut, uint32_t kCtas, uint32_t kHalves>
__global__ void __launch_bounds__(kSwapThreads, 1)
dg_gemm_swap_kernel(const __grid_constant__ GemmParams p, const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                    const __grid_constant__ CUtensorMap tmap_sfa, const __grid_constant__ CUtensorMap tmap_sfb,
                    const __grid_constant__ CUtensorMap tmap_b_part, const __grid_constant__ CUtensorMap tmap_b_tail) {
    constexpr bool kMXF4 = kFmt == kFmtMxf4, kScaled = kFmt != kFmtBf16;
    constexpr uint32_t kHalfElems = kMXF4 ? 256 : 128;      // K elements of one 128-byte slab
    constexpr uint32_t kBlockKElems = kHalves * kHalfElems;
    constexpr bool kTable = swap_has_table(kCtas, kHalves);
    using Scheduler = SwapScheduler<kTable>;
    constexpr uint32_t kEpiBufBytes = swap_epi_buf_bytes(kOut);
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));

    const uint32_t warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const uint32_t cta_rank = kCtas == 2 ? cluster_cta_rank() : 0u;
    const uint32_t block_n = p.block_n;
    const uint32_t sf_block_n = (block_n + 127) / 128 * 128;
    SfPlan plan_a = sf_plan(p.gran_a, kBlockKElems), plan_b = sf_plan(p.gran_b, kBlockKElems);
    const uint32_t new_words = plan_a.period < plan_b.period ? plan_a.period : plan_b.period;
    const uint32_t sf_period = scale_period(p.num_stages, new_words);      // k-blocks between two loads of scale words
    if (sf_period != new_words) plan_a.period = plan_b.period = sf_period;
    const uint32_t sfa_bytes = 512 * plan_a.words, sfb_bytes = sf_block_n * 4 * plan_b.words;
    const uint32_t main_rows = swap_main_rows(block_n, kCtas), tail_rows = swap_tail_rows(block_n, kCtas);
    constexpr uint32_t a_half = kBlockM * kBlockKBytes, a_bytes = a_half * kHalves;
    const uint32_t b_half = main_rows * kBlockKBytes, tail_half = tail_rows * kBlockKBytes;
    const uint32_t b_bytes = (b_half + tail_half) * kHalves;      // main rows of every slab, then the tail rows of every slab
    const uint32_t num_stages = p.num_stages;

    // shared memory carve-up (every tile base stays 1024-byte aligned)
    uint8_t* smem_a = smem;
    uint8_t* smem_b = smem_a + num_stages * a_bytes;
    uint8_t* smem_epi = smem_b + num_stages * b_bytes;
    uint8_t* smem_sf = smem_epi + kSwapEpiWarps * kEpiBufBytes;      // kSwapSfSlots x (weight words, activation words)
    const uint32_t sf_slot_bytes = sfa_bytes + sfb_bytes;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem_sf + kSwapSfSlots * sf_slot_bytes);
    uint64_t* bar_full = bars;                       // operands and scale words of a stage in place (pair: both CTAs', on rank 0)
    uint64_t* bar_empty = bars + kMaxStages;         // the UMMAs reading a stage finished
    uint64_t* bar_sf_raw = bars + 2 * kMaxStages;    // scale words of a slot landed (per CTA)
    uint64_t* bar_sf_empty = bar_sf_raw + kSwapSfSlots;     // ... and have been copied to TMEM
    uint64_t* bar_tmem_full = bar_sf_empty + kSwapSfSlots;
    uint64_t* bar_tmem_empty = bar_tmem_full + 2;
    uint64_t* bar_tmem_edge = bar_tmem_full + 4;     // the columns shared with the other accumulator are in registers
    uint64_t* bar_tc = bar_tmem_full + 6;            // the UMMAs of a k-block finished (only with a duty cycle below 100 %)
    uint64_t* bar_table = bar_tmem_full + 7;         // the group table is in shared memory
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar_tmem_full + 8);
    volatile uint32_t* abort_flag = tmem_slot + 1;
    volatile uint32_t* last_flag = tmem_slot + 2;
    uint4* const group_table = reinterpret_cast<uint4*>((reinterpret_cast<uintptr_t>(tmem_slot + 3) + 15) & ~uintptr_t(15));

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < num_stages; ++s) {
            // the two producer warps (their bytes are counted on the same barrier) and, for the block-scaled kinds, one arrival per CTA
            // for the scale words: by the scale warp on k-blocks that bring new ones, else by the weight producer in its stead, so that
            // the UMMA warp has one barrier to wait for
            mbar_init(bar_full + s, 2 + (kScaled ? kCtas : 0u));
            mbar_init(bar_empty + s, 1);
        }
        for (uint32_t s = 0; s < kSwapSfSlots; ++s) {
            mbar_init(bar_sf_raw + s, 1);
            mbar_init(bar_sf_empty + s, 1);
        }
        for (uint32_t e = 0; e < 2; ++e) {
            mbar_init(bar_tmem_full + e, 1);
            mbar_init(bar_tmem_empty + e, kSwapEpiWarps * kCtas);
            mbar_init(bar_tmem_edge + e, kSwapEpiWarps * kCtas);
        }
        mbar_init(bar_tc, 1);
        mbar_init(bar_table, kSwapEpiWarps);
        *abort_flag = 0;
        fence_mbar_init();
        tma_prefetch_desc(&tmap_a);
        tma_prefetch_desc(&tmap_b);
        tma_prefetch_desc(&tmap_b_part);
        if constexpr (kScaled) {
            tma_prefetch_desc(&tmap_sfa);
            tma_prefetch_desc(&tmap_sfb);
        }
    }
    if (warp == 1) {
        tmem_alloc<kCtas>(tmem_slot, kTmemCols);
        tmem_relinquish<kCtas>();
    }
    tc_fence_before();
    if constexpr (kCtas == 2) cluster_sync(); else __syncthreads();
    tc_fence_after();
    // Every role waits for the previous kernel itself, after what it can do without global memory: its first instructions have to
    // come from memory too, ~1000 cycles that pass while that kernel still runs.
    griddep_launch_dependents();
    // Grouped layouts: the epilogue warps, which have nothing to do yet, bring the groups' rows and tiles into shared memory.  Every
    // role walks the groups one after the other, two to five of them between two tiles; fetched from global memory (~700 cycles each)
    // they stopped the weight loads for that long, where a tile of 16 k-blocks takes 9000 cycles (masked groups of up to 32 rows, 2048 x
    // 2048: 128 of them 114.7 -> 103.9 us; of up to 64 rows, 64 of them 62.1 -> 57.1; contiguous 256 x 128 rows, 2048 x 3584: 397 ->
    // 375).  Read from the table or not in turn, 4-64 masked groups of up to 128 rows and K of 2048-7168 gain 1-10 %, most with many groups
    // and short K.
    auto groups_ready = [&]() {
        griddep_wait();
        if constexpr (kTable) return p.table_groups == 0 || mbar_wait(bar_table, 0, abort_flag, p.status, 0x680);
        else return true;
    };
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t tmem_sfa = tmem_base + p.acc_stride + block_n;
    const uint32_t tmem_sfb = tmem_sfa + 4 * plan_a.words;

    if (warp == 0) {
        // ------------------------------------------------------------ weights: one lane, one or two loads per stage
        if (elect_one()) {
            Scheduler sched(p, kCtas, kBlockKElems);
            SwapTile t;
            uint32_t stage = 0, phase = 0;
            bool ok = true;
            const uint32_t full_addr = kCtas == 2 ? mapa_u32(smem_u32(bar_full), 0) : 0u;
            const uint64_t policy = p.stream_a ? l2_policy_evict_first() : l2_policy_evict_normal();
            const uint32_t tx = (a_bytes >> p.tx_shift_a) * kCtas;
            const bool expects = cta_rank == 0, wide = p.wide_k != 0;
            ok = groups_ready();
            sched.start(group_table);
            while (ok && sched.next(t)) {
                const int32_t row = static_cast<int32_t>(t.m0 + cta_rank * kBlockM), g = static_cast<int32_t>(t.ga);
                for (uint32_t kb = t.kb0; kb < t.kb1; ++kb) {
                    if (!mbar_wait(bar_empty + stage, phase ^ 1, abort_flag, p.status, 0x100 + stage)) { ok = false; break; }
                    if (expects) mbar_arrive_expect_tx(bar_full + stage, tx);
                    if (kScaled && (kb & (sf_period - 1)) != 0 && kb != t.kb0) {
                        if constexpr (kCtas == 1) mbar_arrive(bar_full + stage);
                        else mbar_arrive_remote(bar_full + stage, 0);
                    }
                    uint8_t* dst = smem_a + stage * a_bytes;
                    if (wide) {
                        if constexpr (kCtas == 1) tma_load_4d_hint(dst, &tmap_a, bar_full + stage, 0, row, static_cast<int32_t>(kb * 2), g, policy);
                        else tma_load_4d_2cta_hint(dst, &tmap_a, full_addr + stage * 8, 0, row, static_cast<int32_t>(kb * 2), g, policy);
                    } else {
                        #pragma unroll
                        for (uint32_t h = 0; h < kHalves; ++h) {
                            const int32_t kx = static_cast<int32_t>(kb * kBlockKElems + h * kHalfElems);
                            if constexpr (kCtas == 1) tma_load_3d_hint(dst + h * a_half, &tmap_a, bar_full + stage, kx, row, g, policy);
                            else tma_load_3d_2cta_hint(dst + h * a_half, &tmap_a, full_addr + stage * 8, kx, row, g, policy);
                        }
                    }
                    if (++stage == num_stages) { stage = 0; phase ^= 1; }
                }
            }
        }
        __syncwarp();
    } else if (warp == 3) {
        // ------------------------------------------------------------ activations: few large boxes, even where a tile needs fewer rows
        // (a load costs its issuing lane ~70 cycles whatever its size)
        if (elect_one()) {
            Scheduler sched(p, kCtas, kBlockKElems);
            SwapTile t;
            uint32_t stage = 0, phase = 0;
            bool ok = true;
            const uint32_t full_addr = kCtas == 2 ? mapa_u32(smem_u32(bar_full), 0) : 0u;
            const uint32_t part_rows = swap_part_rows(main_rows);
            const bool expects = cta_rank == 0, wide = p.wide_k != 0;
            constexpr uint32_t kTailBytes = kSwapTailRows * kBlockKBytes;
            ok = groups_ready();
            sched.start(group_table);
            while (ok && sched.next(t)) {
                // a pair's UMMA takes the first half of its N rows from rank 0 and the second half from rank 1
                const uint32_t n_main = t.n < 256 ? t.n : 256u, my_rows = n_main / kCtas, my_tail = (t.n - n_main) / kCtas;
                const int32_t row = static_cast<int32_t>(t.n0 + cta_rank * my_rows), g = static_cast<int32_t>(t.gb);
                const int32_t row_tail = static_cast<int32_t>(t.n0 + n_main + cta_rank * my_tail);
                const bool full = my_rows > part_rows || part_rows == main_rows;
                const uint32_t tails = (my_tail + kSwapTailRows - 1) / kSwapTailRows;
                const uint32_t tx = (((full ? main_rows : part_rows) * kBlockKBytes + tails * kTailBytes) * kHalves * kCtas) >> p.tx_shift_b;
                for (uint32_t kb = t.kb0; kb < t.kb1; ++kb) {
                    if (!mbar_wait(bar_empty + stage, phase ^ 1, abort_flag, p.status, 0x180 + stage)) { ok = false; break; }
                    if (expects) mbar_arrive_expect_tx(bar_full + stage, tx);
                    uint8_t* dst = smem_b + stage * b_bytes;
                    if (full && wide) {
                        if constexpr (kCtas == 1) tma_load_4d(dst, &tmap_b, bar_full + stage, 0, row, static_cast<int32_t>(kb * 2), g);
                        else tma_load_4d_2cta(dst, &tmap_b, full_addr + stage * 8, 0, row, static_cast<int32_t>(kb * 2), g);
                    } else {
                        const CUtensorMap* map = full ? &tmap_b : &tmap_b_part;
                        #pragma unroll
                        for (uint32_t h = 0; h < kHalves; ++h) {
                            const int32_t kx = static_cast<int32_t>(kb * kBlockKElems + h * kHalfElems);
                            if constexpr (kCtas == 1) tma_load_3d(dst + h * b_half, map, bar_full + stage, kx, row, g);
                            else tma_load_3d_2cta(dst + h * b_half, map, full_addr + stage * 8, kx, row, g);
                        }
                    }
                    if (tails != 0) {
                        #pragma unroll
                        for (uint32_t h = 0; h < kHalves; ++h) {
                            const int32_t kx = static_cast<int32_t>(kb * kBlockKElems + h * kHalfElems);
                            uint8_t* dst_tail = dst + kHalves * b_half + h * tail_half;
                            for (uint32_t j = 0; j < tails; ++j) {
                                const int32_t r = row_tail + static_cast<int32_t>(j * kSwapTailRows);
                                if constexpr (kCtas == 1) tma_load_3d(dst_tail + j * kTailBytes, &tmap_b_tail, bar_full + stage, kx, r, g);
                                else tma_load_3d_2cta(dst_tail + j * kTailBytes, &tmap_b_tail, full_addr + stage * 8, kx, r, g);
                            }
                        }
                    }
                    if (++stage == num_stages) { stage = 0; phase ^= 1; }
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------------------------------------- UMMA issuer
        if (cta_rank == 0) {
            Scheduler sched(p, kCtas, kBlockKElems);
            SwapTile t;
            uint32_t stage = 0, phase = 0, it = 0, tc_phase = 0, prev_n = 0, slot = 0;
            bool ok = true;
            const bool leader_lane = elect_one();
            // Everything a stage needs is an add away from values computed here: descriptors are (low word moving with the stage, constant
            // high word), the instruction descriptor carries the scale byte of the slab (per-128 scales) or of the UMMA (per-32 scales).
            const uint32_t desc_hi = static_cast<uint32_t>(make_smem_desc(0, 0, 1024, 2) >> 32), sf_hi = static_cast<uint32_t>(make_smem_desc(0, 0, 128, 0) >> 32);
            const uint32_t a_lo0 = smem_u32(smem_a) >> 4, b_lo0 = smem_u32(smem_b) >> 4, sf_lo0 = smem_u32(smem_sf) >> 4;
            const uint32_t b_step = b_bytes >> 4, b_half_step = b_half >> 4, tail_off = (kHalves * b_half) >> 4, tail_half_step = tail_half >> 4;
            const uint32_t sf_step = sf_slot_bytes >> 4, sfb_off = sfa_bytes >> 4;
            const bool per128_a = p.gran_a == 128, per128_b = p.gran_b == 128;
            const uint32_t slab_ids = kMXF4 ? 0u : ((per128_a ? 1u << 29 : 0u) | (per128_b ? 1u << 4 : 0u));
            const uint32_t umma_ids = kMXF4 ? 0u : ((per128_a ? 0u : 1u << 29) | (per128_b ? 0u : 1u << 4));
            const uint32_t per_word = sf_block_n / 128;
            // scale columns of slab h (per-32 scales of e4m3: one word per slab; e2m1: one word per two UMMAs)
            const uint32_t sfa_slab = kMXF4 ? 8u : (per128_a ? 0u : 4u), sfb_slab = kMXF4 ? 8u * per_word : (per128_b ? 0u : 4u * per_word);
            const uint32_t sfa_cols[2] = {tmem_sfa, tmem_sfa + sfa_slab}, sfb_cols[2] = {tmem_sfb, tmem_sfb + sfb_slab};
            const bool throttled = p.tc_util < 100;
            ok = groups_ready();
            if constexpr (kTable) ok = __all_sync(0xFFFFFFFFu, ok);
            sched.start(group_table);
            while (ok && sched.next(t)) {
                const uint32_t e = it & 1, acc_phase = (it >> 1) & 1;
                if (!mbar_wait_warp(bar_tmem_empty + e, acc_phase ^ 1, abort_flag, p.status, 0x200 + e)) break;
                // does this tile share columns with the one before, in the other accumulator?
                if (it > 0 && (e == 0 ? t.n : prev_n) > p.acc_stride)
                    if (!mbar_wait_warp(bar_tmem_edge + (e ^ 1), ((it - 1) >> 1) & 1, abort_flag, p.status, 0x280 + e)) break;
                ++it;
                prev_n = t.n;
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + e * p.acc_stride;
                const uint32_t used = (t.n + 127) / 128;
                const uint32_t n_main = t.n < 256 ? t.n : 256u, n_tail = t.n - n_main;
                const uint32_t idesc0 = kScaled ? make_idesc_block_scaled(kBlockM * kCtas, n_main, kMXF4 ? 1u : p.fmt_a, kMXF4 ? 1u : p.fmt_b)
                                                : make_idesc_bf16(kBlockM * kCtas, n_main);
                const uint32_t tail_idesc = ((n_main - n_tail) >> 3) << 17;      // what to subtract for the N of the tail
                for (uint32_t kb = t.kb0; kb < t.kb1; ++kb) {
                    const bool need_sf = kScaled && ((kb & (sf_period - 1)) == 0 || kb == t.kb0);
                    if (!mbar_wait_warp(bar_full + stage, phase, abort_flag, p.status, 0x300 + stage)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t a_lo = a_lo0 + stage * (a_bytes >> 4), b_lo = b_lo0 + stage * b_step;
                    const uint32_t sfa_lo = sf_lo0 + slot * sf_step, sfb_lo = sfa_lo + sfb_off;
                    const bool last = kb + 1 == t.kb1;
                    const bool need_a = need_sf && ((kb & (plan_a.period - 1)) == 0 || kb == t.kb0), need_b = need_sf && ((kb & (plan_b.period - 1)) == 0 || kb == t.kb0);
                    // operands computed by the whole warp, ahead of the single-lane region: warp-uniform values stay in uniform registers
                    uint32_t idescs[kHalves][4];
                    uint64_t a_descs[kHalves], b_descs[kHalves], t_descs[kHalves];
                    #pragma unroll
                    for (uint32_t h = 0; h < kHalves; ++h) {
                        #pragma unroll
                        for (uint32_t k = 0; k < 4; ++k)
                            idescs[h][k] = kMXF4 ? idesc_with_sf_ids(idesc0, (k & 1) * 2, (k & 1) * 2) : idesc0 + ((kb * kHalves + h) & 3) * slab_ids + k * umma_ids;
                        a_descs[h] = desc64(a_lo + h * (a_half >> 4), desc_hi);
                        b_descs[h] = desc64(b_lo + h * b_half_step, desc_hi);
                        t_descs[h] = desc64(b_lo + tail_off + h * tail_half_step, desc_hi);
                    }
                    const uint64_t sfa_desc = desc64(sfa_lo, sf_hi), sfb_desc = desc64(sfb_lo, sf_hi);
                    if (leader_lane) {
                        if (need_sf) {
                            if (need_a)
                                for (uint32_t c = 0; c < plan_a.words; ++c) utccp_32x128b_warpx4<kCtas>(tmem_sfa + 4 * c, sfa_desc + c * (512 >> 4));
                            if (need_b)
                                // a word column has per_word chunks of 128 rows, of which the tile uses the first ones
                                for (uint32_t w = 0; w < plan_b.words; ++w)
                                    for (uint32_t c = w * per_word; c < w * per_word + used; ++c)
                                        utccp_32x128b_warpx4<kCtas>(tmem_sfb + 4 * c, sfb_desc + c * (512 >> 4));
                            if constexpr (kCtas == 1) umma_commit(bar_sf_empty + slot);
                            else umma_commit_2cta(bar_sf_empty + slot, static_cast<uint16_t>(3));
                        }
                        auto issue = [&](uint32_t d, const uint64_t* rows, uint32_t less, uint32_t sf_off) {
                            #pragma unroll
                            for (uint32_t h = 0; h < kHalves; ++h) {
                                #pragma unroll
                                for (uint32_t k = 0; k < kBlockKBytes / kUmmaKBytes; ++k) {
                                    const uint32_t accumulate = (h != 0 || k != 0) ? 1u : (kb != t.kb0 ? 1u : 0u);
                                    const uint64_t a_desc = a_descs[h] + k * (kUmmaKBytes >> 4), b_desc = rows[h] + k * (kUmmaKBytes >> 4);
                                    if constexpr (kMXF4)
                                        umma_block_scaled<kCtas, true>(d, a_desc, b_desc, idescs[h][k] - less, sfa_cols[h] + 4 * (k / 2),
                                                                       sfb_cols[h] + sf_off + 4 * per_word * (k / 2), accumulate);
                                    else if constexpr (kScaled)
                                        umma_block_scaled<kCtas, false>(d, a_desc, b_desc, idescs[h][k] - less, sfa_cols[h], sfb_cols[h] + sf_off, accumulate);
                                    else umma_f16<kCtas>(d, a_desc, b_desc, idesc0 - less, accumulate);
                                }
                            }
                        };
                        issue(d_tmem, b_descs, 0, 0);
                        if (n_tail != 0) issue(d_tmem + 256, t_descs, tail_idesc, 8);       // 256 rows: two chunks of scale columns further
                        if constexpr (kCtas == 1) {
                            umma_commit(bar_empty + stage);
                            if (last) umma_commit(bar_tmem_full + e);
                        } else {
                            umma_commit_2cta(bar_empty + stage, static_cast<uint16_t>(3));
                            if (last) umma_commit_2cta(bar_tmem_full + e, static_cast<uint16_t>(3));
                        }
                    }
                    __syncwarp();
                    if (throttled) {
                        // duty cycle: wait until this k-block's UMMAs are done, then idle for the requested share
                        if (leader_lane) {
                            if constexpr (kCtas == 1) umma_commit(bar_tc);
                            else umma_commit_2cta(bar_tc, static_cast<uint16_t>(1));
                        }
                        __syncwarp();
                        if (!mbar_wait_warp(bar_tc, tc_phase, abort_flag, p.status, 0x480)) { ok = false; break; }
                        tc_phase ^= 1;
                        duty_cycle_pause(p.tc_util, t.n * kHalves);
                        __syncwarp();
                    }
                    if (need_sf && ++slot == kSwapSfSlots) slot = 0;
                    if (++stage == num_stages) { stage = 0; phase ^= 1; }
                }
            }
        }
        __syncwarp();
    } else if (warp == 2) {
        // -------------------------------------------------- scale words: load, re-order, publish
        // A ring of its own, fetched up to kSwapSfSlots - 1 loads ahead: loaded together with their k-block's operands, the words were
        // re-ordered ~300 cycles after those had landed, and every stage with new words was that much later.
        if constexpr (kScaled) {
            // walks the k-blocks that need new words: `ahead` issues loads, `here` re-orders what landed
            struct Walk {
                Scheduler sched;
                SwapTile t;
                uint32_t kb;
                bool live;
            };
            auto start = [&](Walk& w) { w.live = w.sched.next(w.t); w.kb = w.live ? w.t.kb0 : 0u; };
            auto step = [&](Walk& w) {
                w.kb = (w.kb & ~(sf_period - 1)) + sf_period;
                if (w.kb >= w.t.kb1) start(w);
            };
            auto needs = [&](const Walk& w, const SfPlan& plan) { return (w.kb & (plan.period - 1)) == 0 || w.kb == w.t.kb0; };
            Walk ahead{Scheduler(p, kCtas, kBlockKElems)};
            bool ok = groups_ready();
            if constexpr (kTable) ok = __all_sync(0xFFFFFFFFu, ok);
            ahead.sched.start(group_table);
            start(ahead);
            Walk here = ahead;
            uint32_t in_slot = 0, in_phase = 0, out_slot = 0, out_phase = 0, in_flight = 0;
            uint32_t stage = 0, phase = 0;      // of the k-block `here`
            const bool leader_lane = elect_one();
            while (ok && here.live) {
                while (ahead.live && in_flight < kSwapSfSlots - 1) {      // a free slot never holds up words that have landed
                    if (!mbar_wait_warp(bar_sf_empty + in_slot, in_phase ^ 1, abort_flag, p.status, 0x400 + in_slot)) { ok = false; break; }
                    if (leader_lane) {
                        uint8_t* dst = smem_sf + in_slot * sf_slot_bytes;
                        const bool need_a = needs(ahead, plan_a), need_b = needs(ahead, plan_b);
                        const uint32_t used = (ahead.t.n + 127) / 128;
                        mbar_arrive_expect_tx(bar_sf_raw + in_slot, (need_a ? sfa_bytes : 0u) + (need_b ? used * 512 * plan_b.words : 0u));
                        if (need_a)
                            tma_load_2d(dst, &tmap_sfa, bar_sf_raw + in_slot, static_cast<int32_t>(ahead.t.m0 + cta_rank * kBlockM),
                                        static_cast<int32_t>(ahead.t.ga * p.sf_a_cols + (ahead.kb >> plan_a.shift) * plan_a.words));
                        if (need_b) {
                            const int32_t y = static_cast<int32_t>(ahead.t.gb * p.sf_b_cols + (ahead.kb >> plan_b.shift) * plan_b.words);
                            for (uint32_t w = 0; w < plan_b.words; ++w)
                                for (uint32_t c = 0; c < used; ++c)
                                    tma_load_2d(dst + sfa_bytes + (w * sf_block_n + c * 128) * 4, &tmap_sfb, bar_sf_raw + in_slot,
                                                static_cast<int32_t>(ahead.t.n0 + c * 128), y + static_cast<int32_t>(w));
                        }
                    }
                    __syncwarp();
                    ++in_flight;
                    if (++in_slot == kSwapSfSlots) { in_slot = 0; in_phase ^= 1; }
                    step(ahead);
                }
                if (!ok || !mbar_wait_warp(bar_sf_raw + out_slot, out_phase, abort_flag, p.status, 0x500 + out_slot)) { ok = false; break; }
                // word r of a 128-word chunk moves to position (r % 32) * 4 + r / 32
                auto reorder = [&](uint8_t* at) {
                    uint32_t* chunk = reinterpret_cast<uint32_t*>(at);
                    const uint32_t w0 = chunk[lane], w1 = chunk[32 + lane], w2 = chunk[64 + lane], w3 = chunk[96 + lane];
                    __syncwarp();
                    st_shared_v4(smem_u32(chunk + lane * 4), w0, w1, w2, w3);
                };
                uint8_t* words = smem_sf + out_slot * sf_slot_bytes;
                const uint32_t used = (here.t.n + 127) / 128, per_word = sf_block_n / 128;
                if (needs(here, plan_a))
                    for (uint32_t c = 0; c < plan_a.words; ++c) reorder(words + c * 512);
                if (needs(here, plan_b))
                    for (uint32_t w = 0; w < plan_b.words; ++w)
                        for (uint32_t c = 0; c < used; ++c) reorder(words + sfa_bytes + (w * per_word + c) * 512);
                fence_proxy_async_smem();
                __syncwarp();
                // the arrival belongs to the stage's present round: its previous one must be over
                if (!mbar_wait_warp(bar_empty + stage, phase ^ 1, abort_flag, p.status, 0x580 + stage)) { ok = false; break; }
                if (lane == 0) {
                    if constexpr (kCtas == 1) mbar_arrive(bar_full + stage);
                    else mbar_arrive_remote(bar_full + stage, 0);
                }
                --in_flight;
                if (++out_slot == kSwapSfSlots) { out_slot = 0; out_phase ^= 1; }
                const uint32_t next_kb = (here.kb & ~(sf_period - 1)) + sf_period, last_kb = next_kb < here.t.kb1 ? next_kb : here.t.kb1;
                for (uint32_t kb = here.kb; kb < last_kb; ++kb)
                    if (++stage == num_stages) { stage = 0; phase ^= 1; }
                step(here);
            }
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------------ epilogue
        const uint32_t ew = warp % 4, half = (warp - 4) / 4;      // TMEM lane quadrant: 32 output columns; which of its two warps
        uint8_t* const buf = smem_epi + (warp - 4) * kEpiBufBytes;
        Scheduler sched(p, kCtas, kBlockKElems);
        SwapTile t;
        uint32_t it = 0;
        if constexpr (kTable) {
            if (p.table_groups != 0) {
                griddep_wait();
                for (uint32_t g = threadIdx.x - 128; g < p.table_groups; g += kSwapEpiWarps * 32) {
                    sched.read_group(g);
                    group_table[g] = make_uint4(sched.row_start, sched.rows, sched.num_tiles, sched.tile_rows);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_table);
            }
        }
        bool ok = groups_ready();
        sched.start(group_table);
        while (sched.next(t)) {
            const uint32_t e = it & 1, acc_phase = (it >> 1) & 1;
            ++it;
            ok = ok && mbar_wait(bar_tmem_full + e, acc_phase, abort_flag, p.status, 0x600 + e);
            // with K ranges the eight warps meet below: a warp that gave up keeps coming to those meetings, so that none waits for it
            if (!ok && p.num_splits == 1) break;
            tc_fence_after();
            const uint32_t taddr = tmem_base + ((ew * 32) << 16) + e * p.acc_stride;
            const uint32_t col0 = t.m0 + cta_rank * kBlockM + ew * 32;      // first output column of this warp
            const uint32_t chunks = (t.rows + 31) / 32;
            constexpr uint32_t kElem = kOut == kOutBf16 ? 2 : (kOut == kOutF32 ? 4 : 1);
            uint8_t* const out = static_cast<uint8_t*>(p.out_ptr) + ((static_cast<size_t>(t.gd) * p.n + t.n0) * p.out_ld + col0) * kElem;
            const size_t pitch = static_cast<size_t>(p.out_ld) * kElem;
            const uint32_t cols = col0 < p.m ? (p.m - col0 < 32 ? p.m - col0 : 32u) : 0u;       // columns of this warp that exist
            auto arrive = [&](uint64_t* bar) {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    if constexpr (kCtas == 1) mbar_arrive(bar + e);
                    else mbar_arrive_remote(bar + e, 0);
                }
            };
            // 32 output rows to registers: in matrix-fragment order (lanes 0-15 of the quadrant, then 16-31), f32 one column per lane
            auto load_chunk = [&](uint32_t c, uint32_t (&v)[32]) {
                if constexpr (kOut != kOutF32) {
                    tmem_ld_16x256b_x4(taddr + c * 32, v);
                    tmem_ld_16x256b_x4(taddr + (16u << 16) + c * 32, v + 16);
                } else {
                    tmem_ld_32x32b_x32(taddr + c * 32, v);
                }
            };
            if (p.num_splits > 1) {
                // K ranges: this range's accumulator to the workspace, 16 bytes per thread and step (coalesced; read back by the same thread
                // positions), then count the range in; the last one sums all of them in range order
                const size_t tile_floats = static_cast<size_t>((block_n + 31) / 32) * 32 * kBlockM;
                const size_t first_slot = (static_cast<size_t>(t.index) * kCtas + cta_rank) * p.num_splits;
                const uint32_t et = ew * 32 + lane;       // position in the 128 lanes of the accumulator
                float4* mine = reinterpret_cast<float4*>(p.splitk_ws + (first_slot + t.split) * tile_floats);
                for (uint32_t c = half; ok && c < chunks; c += 2) {
                    uint32_t v[32];
                    load_chunk(c, v);
                    tmem_ld_wait_x32(v);
                    #pragma unroll
                    for (uint32_t i = 0; i < 8; ++i)
                        __stcg(mine + (c * 8 + i) * 128 + et, make_float4(__uint_as_float(v[4 * i]), __uint_as_float(v[4 * i + 1]), __uint_as_float(v[4 * i + 2]),
                                                                          __uint_as_float(v[4 * i + 3])));
                }
                arrive(bar_tmem_edge);
                arrive(bar_tmem_empty);
                __threadfence();
                named_bar_sync(1, kSwapEpiWarps * 32);
                if (threadIdx.x == 128) {
                    uint32_t* counter = p.splitk_counters + static_cast<size_t>(t.index) * kCtas + cta_rank;
                    const bool last = ok && atomicAdd(counter, 1u) + 1 == p.num_splits;
                    if (last) *counter = 0;        // ready for the next launch
                    __threadfence();
                    *last_flag = last ? 1u : 0u;
                }
                named_bar_sync(1, kSwapEpiWarps * 32);
                const bool last = *last_flag != 0;
                named_bar_sync(1, kSwapEpiWarps * 32);            // everyone has read the flag before the next tile may set it
                if (!last) continue;
            }
            // Chunks in an order that frees the columns shared with the other accumulator first: buffer 0 from the top, buffer 1 from the
            // bottom.  One pass of one loop per chunk: unrolled (or with two chunks in flight) this code outgrows the instruction cache.
            const bool ranges = p.num_splits > 1;
            const uint32_t loads = ranges ? chunks : (t.n + 31) / 32, edge = p.acc_edge_chunks < loads ? p.acc_edge_chunks : loads;
            bool edge_done = ranges, all_done = ranges;       // (with K ranges both were reported above)
            #pragma unroll 1
            for (uint32_t i = half; i < loads; i += 2) {
                const uint32_t c = e == 0 ? loads - 1 - i : i;
                uint32_t v[32];
                if (ranges) {
                    const size_t tile_floats = static_cast<size_t>((block_n + 31) / 32) * 32 * kBlockM;
                    const float4* first = reinterpret_cast<const float4*>(p.splitk_ws + (static_cast<size_t>(t.index) * kCtas + cta_rank) * p.num_splits * tile_floats) +
                                          c * 1024 + ew * 32 + lane;
                    #pragma unroll
                    for (uint32_t k = 0; k < 32; ++k) v[k] = 0;
                    #pragma unroll 2
                    for (uint32_t r = 0; r < p.num_splits; ++r) {
                        float4 x[8];
                        #pragma unroll
                        for (uint32_t k = 0; k < 8; ++k) x[k] = __ldcg(first + r * (tile_floats / 4) + k * 128);
                        #pragma unroll
                        for (uint32_t k = 0; k < 8; ++k) {
                            v[4 * k] = __float_as_uint(__uint_as_float(v[4 * k]) + x[k].x);
                            v[4 * k + 1] = __float_as_uint(__uint_as_float(v[4 * k + 1]) + x[k].y);
                            v[4 * k + 2] = __float_as_uint(__uint_as_float(v[4 * k + 2]) + x[k].z);
                            v[4 * k + 3] = __float_as_uint(__uint_as_float(v[4 * k + 3]) + x[k].w);
                        }
                    }
                } else {
                    load_chunk(c, v);
                    tmem_ld_wait_x32(v);
                    if (!edge_done && i + 2 >= edge) { arrive(bar_tmem_edge); edge_done = true; }
                    if (i + 2 >= loads) { arrive(bar_tmem_empty); all_done = true; }
                }
                if (c >= chunks) continue;
                // Exactly the tile's rows are written, straight from the warp: a store through TMA would hold the staging buffer for ~1000
                // cycles, longer than a chunk takes to convert.
                const uint32_t left = t.rows - c * 32, rows_here = left < 32 ? left : 32u;
                uint8_t* const dst = out + c * 32 * pitch;
                if (p.has_alpha) {
                    #pragma unroll
                    for (uint32_t k = 0; k < 32; ++k) v[k] = __float_as_uint(__uint_as_float(v[k]) * p.alpha);
                }
                if constexpr (kOut == kOutF32) {
                    // one row per instruction: 32 lanes write 128 consecutive bytes
                    float* o = reinterpret_cast<float*>(dst) + lane;
                    #pragma unroll
                    for (uint32_t r = 0; r < 32; ++r) {
                        if (r < rows_here && lane < cols) *o = p.accumulate ? *o + __uint_as_float(v[r]) : __uint_as_float(v[r]);
                        o += p.out_ld;
                    }
                    continue;
                }
                // 64-byte rows of bf16, the 16-byte pieces swizzled by (row / 2) % 4; lane 8 q + k addresses columns 8 q .. 8 q + 7 of row 8 j + k
                __syncwarp();       // the previous chunk has been read
                #pragma unroll
                for (uint32_t j = 0; j < 4; ++j) {
                    const uint32_t row = 8 * j + lane % 8;
                    stmatrix_x4_trans(smem_u32(buf) + row * 64 + (((lane / 8) ^ ((row >> 1) & 3)) << 4),
                                      pack_bf16x2(__uint_as_float(v[4 * j]), __uint_as_float(v[4 * j + 1])),
                                      pack_bf16x2(__uint_as_float(v[4 * j + 2]), __uint_as_float(v[4 * j + 3])),
                                      pack_bf16x2(__uint_as_float(v[16 + 4 * j]), __uint_as_float(v[16 + 4 * j + 1])),
                                      pack_bf16x2(__uint_as_float(v[16 + 4 * j + 2]), __uint_as_float(v[16 + 4 * j + 3])));
                }
                __syncwarp();
                if constexpr (kOut == kOutBf16) {
                    // a lane takes one 16-byte piece of every eighth row: four lanes write 64 bytes of a row
                    const uint32_t piece = lane % 4;
                    uint8_t* at = dst + (lane / 4) * pitch + piece * 16;
                    #pragma unroll
                    for (uint32_t j = 0; j < 4; ++j) {
                        const uint32_t row = 8 * j + lane / 4, from = smem_u32(buf) + row * 64 + ((piece ^ ((row >> 1) & 3)) << 4);
                        if (row < rows_here && piece * 8 + 8 <= cols) {
                            uint4 x = ld_shared_v4(from);
                            if (p.accumulate) {
                                const uint4 old = *reinterpret_cast<uint4*>(at);
                                x = make_uint4(add_bf16x2(x.x, old.x), add_bf16x2(x.y, old.y), add_bf16x2(x.z, old.z), add_bf16x2(x.w, old.w));
                            }
                            *reinterpret_cast<uint4*>(at) = x;
                        } else if (row < rows_here && piece * 8 < cols) {
                            // the matrix ends inside this piece
                            #pragma unroll 1
                            for (uint32_t k = 0; piece * 8 + k < cols; ++k) {
                                uint16_t* const o = reinterpret_cast<uint16_t*>(at) + k;
                                const uint32_t y = ld_shared_u16(from + 2 * k);
                                *o = static_cast<uint16_t>(p.accumulate ? add_bf16x2(y, *o) : y);
                            }
                        }
                        at += 8 * pitch;
                    }
                } else {
                    // a lane takes a row: bf16 values, maximum of their bit patterns, the power-of-two scale that brings it under 448,
                    // 32 bytes of e4m3 (n is a multiple of 128: the columns all exist or none does)
                    uint32_t w[16];
                    #pragma unroll
                    for (uint32_t j = 0; j < 4; ++j) {
                        const uint4 x = ld_shared_v4(smem_u32(buf) + lane * 64 + ((j ^ ((lane >> 1) & 3)) << 4));
                        w[4 * j] = x.x; w[4 * j + 1] = x.y; w[4 * j + 2] = x.z; w[4 * j + 3] = x.w;
                    }
                    uint32_t amax = 0;
                    #pragma unroll
                    for (uint32_t k = 0; k < 16; ++k) amax = max(amax, max(w[k] & 0x7FFFu, (w[k] >> 16) & 0x7FFFu));
                    const uint32_t rounded = (amax + 0x7Fu - 0x60u) >> 7;
                    uint32_t sf_exp = (rounded < 8u ? 8u : rounded) - 8u;
                    sf_exp = sf_exp < 105u ? 105u : sf_exp;
                    const float inv = __uint_as_float((254u - sf_exp) << 23);
                    if (lane < rows_here && cols != 0) {
                        uint32_t q[8];
                        #pragma unroll
                        for (uint32_t k = 0; k < 8; ++k)
                            q[k] = cvt_e4m3x4(scale_pos_zero(__uint_as_float(w[2 * k] << 16), inv), scale_pos_zero(__uint_as_float(w[2 * k] & 0xFFFF0000u), inv),
                                              scale_pos_zero(__uint_as_float(w[2 * k + 1] << 16), inv), scale_pos_zero(__uint_as_float(w[2 * k + 1] & 0xFFFF0000u), inv));
                        uint4* const o = reinterpret_cast<uint4*>(dst + lane * pitch);
                        o[0] = make_uint4(q[0], q[1], q[2], q[3]);
                        o[1] = make_uint4(q[4], q[5], q[6], q[7]);
                        if (c * 32 + lane < t.valid)
                            reinterpret_cast<uint8_t*>(p.sfd)[(static_cast<size_t>(t.gd * (p.m / 128) + col0 / 128) * p.sfd_stride + t.n0 + c * 32 + lane) * 4 + (col0 % 128) / 32] =
                                static_cast<uint8_t>(sf_exp);
                    }
                }
            }
            if (!edge_done) arrive(bar_tmem_edge);      // a tile of one chunk leaves the second warp without any
            if (!all_done) arrive(bar_tmem_empty);
        }
        __syncwarp();
    }

    tc_fence_before();
    if constexpr (kCtas == 2) cluster_sync(); else __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc<kCtas>(tmem_base, kTmemCols);
    }
}

// Bytes of dynamic shared memory the kernel needs for a configuration, without the group table (host side).
inline uint32_t gemm_swap_smem_bytes(uint32_t block_n, uint32_t ctas, uint32_t out_kind, uint32_t stages, uint32_t sfa_words, uint32_t sfb_words, uint32_t halves) {
    const uint32_t sf_block_n = (block_n + 127) / 128 * 128;
    const uint32_t per_stage = halves * (kBlockM + swap_main_rows(block_n, ctas) + swap_tail_rows(block_n, ctas)) * kBlockKBytes;
    return 1024 + stages * per_stage + kSwapEpiWarps * swap_epi_buf_bytes(out_kind) + kSwapSfSlots * (512 * sfa_words + sf_block_n * 4 * sfb_words) +
           (2 * kMaxStages + 2 * kSwapSfSlots + 8) * 8 + 32;
}
// Column where the second accumulator starts.
inline uint32_t gemm_swap_acc_stride(uint32_t block_n, uint32_t sfa_words, uint32_t sfb_words) {
    const uint32_t sf_cols = 4 * sfa_words + (block_n + 127) / 128 * 4 * sfb_words;
    const uint32_t room = kTmemCols - sf_cols - block_n;
    return room < block_n ? room / 16 * 16 : block_n;
}

}  // namespace dg
