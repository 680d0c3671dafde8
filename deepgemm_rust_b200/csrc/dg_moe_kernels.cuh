// Row movers either side of the expert-sharded grouped GEMM: they pack quantised token rows and
// their scale words into all-to-all send rows, unpack received rows into the group-contiguous
// arena (data + packed scale layout), gather result rows for the way back and reduce a token's
// expert outputs.  Byte movers: 16-byte loads/stores, one warp per row.
#pragma once
#include "dg_ptx.cuh"

namespace dg {

// dst row i = src row idx[i] (row_bytes, a multiple of 16); idx[i] < 0 writes zeros.
__global__ void __launch_bounds__(256) dg_gather_rows_kernel(const uint8_t* src, size_t src_pitch, const int32_t* idx,
                                                             uint32_t n_dst, uint32_t row_bytes, uint8_t* dst, size_t dst_pitch) {
    griddep_wait();
    griddep_launch_dependents();
    const uint32_t lane = threadIdx.x % 32;
    const uint64_t row = static_cast<uint64_t>(blockIdx.x) * (blockDim.x / 32) + threadIdx.x / 32;
    if (row >= n_dst) return;
    const int32_t s = ld_ro(idx + row);
    uint4* d = reinterpret_cast<uint4*>(dst + row * dst_pitch);
    if (s < 0) {
        for (uint32_t c = lane; c < row_bytes / 16; c += 32) d[c] = make_uint4(0, 0, 0, 0);
        return;
    }
    const uint4* p = reinterpret_cast<const uint4*>(src + static_cast<size_t>(s) * src_pitch);
    for (uint32_t c = lane; c < row_bytes / 16; c += 32) d[c] = ld_ro(p + c);
}

// Send row i = [k data bytes of token idx[i] | its sf_cols scale words | zero padding up to out_pitch].
// Scale words come from the packed layout sf[c * sf_stride + token].
__global__ void __launch_bounds__(256) dg_moe_pack_rows_kernel(const uint8_t* data, uint32_t k, const uint32_t* sf,
                                                               uint32_t sf_stride, uint32_t sf_cols, const int32_t* idx, uint32_t n,
                                                               uint8_t* out, size_t out_pitch) {
    griddep_wait();
    griddep_launch_dependents();
    const uint32_t lane = threadIdx.x % 32;
    const uint64_t row = static_cast<uint64_t>(blockIdx.x) * (blockDim.x / 32) + threadIdx.x / 32;
    if (row >= n) return;
    const uint32_t tok = static_cast<uint32_t>(ld_ro(idx + row));
    const uint4* p = reinterpret_cast<const uint4*>(data + static_cast<size_t>(tok) * k);
    uint4* d = reinterpret_cast<uint4*>(out + row * out_pitch);
    for (uint32_t c = lane; c < k / 16; c += 32) d[c] = ld_ro(p + c);
    uint32_t* tail = reinterpret_cast<uint32_t*>(out + row * out_pitch + k);
    const uint32_t tail_words = static_cast<uint32_t>((out_pitch - k) / 4);
    for (uint32_t c = lane; c < tail_words; c += 32) tail[c] = c < sf_cols ? ld_ro(sf + static_cast<size_t>(c) * sf_stride + tok) : 0u;
}

// Arena row i takes received row idx[i]: data bytes to dst_data, scale words to the packed layout
// dst_sf[c * dst_sf_stride + i].  idx[i] < 0 (alignment padding) writes zero data and zero scales.
__global__ void __launch_bounds__(256) dg_moe_unpack_rows_kernel(const uint8_t* in, size_t in_pitch, uint32_t k, uint32_t sf_cols,
                                                                 const int32_t* idx, uint32_t n_dst, uint8_t* dst_data,
                                                                 uint32_t* dst_sf, uint32_t dst_sf_stride) {
    griddep_wait();
    griddep_launch_dependents();
    const uint32_t lane = threadIdx.x % 32;
    const uint64_t row = static_cast<uint64_t>(blockIdx.x) * (blockDim.x / 32) + threadIdx.x / 32;
    if (row >= n_dst) return;
    const int32_t s = ld_ro(idx + row);
    uint4* d = reinterpret_cast<uint4*>(dst_data + row * k);
    if (s < 0) {
        for (uint32_t c = lane; c < k / 16; c += 32) d[c] = make_uint4(0, 0, 0, 0);
        for (uint32_t c = lane; c < sf_cols; c += 32) dst_sf[static_cast<size_t>(c) * dst_sf_stride + row] = 0u;
        return;
    }
    const uint8_t* src = in + static_cast<size_t>(s) * in_pitch;
    const uint4* p = reinterpret_cast<const uint4*>(src);
    for (uint32_t c = lane; c < k / 16; c += 32) d[c] = ld_ro(p + c);
    const uint32_t* tail = reinterpret_cast<const uint32_t*>(src + k);
    for (uint32_t c = lane; c < sf_cols; c += 32) dst_sf[static_cast<size_t>(c) * dst_sf_stride + row] = ld_ro(tail + c);
}

// out[t, :] = bf16( sum_j w[t, j] * rows[pos[t, j], :] ), f32 accumulation in order j = 0..topk-1
// with one fused multiply-add per term; pos < 0 skips the term.  One thread owns 8 columns.
__global__ void __launch_bounds__(256) dg_moe_combine_kernel(const uint16_t* rows, size_t pitch, const int32_t* pos,
                                                             const float* w, uint32_t tokens, uint32_t topk, uint32_t n,
                                                             uint16_t* out, size_t out_pitch) {
    griddep_wait();
    griddep_launch_dependents();
    const uint32_t chunks = n / 8;
    const uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= static_cast<uint64_t>(tokens) * chunks) return;
    const uint32_t t = static_cast<uint32_t>(i / chunks), c = static_cast<uint32_t>(i % chunks);
    float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (uint32_t j = 0; j < topk; ++j) {
        const int32_t p = ld_ro(pos + static_cast<size_t>(t) * topk + j);
        if (p < 0) continue;
        const float wj = ld_ro(w + static_cast<size_t>(t) * topk + j);
        const uint4 v = ld_ro(reinterpret_cast<const uint4*>(rows + static_cast<size_t>(p) * pitch) + c);
        const uint32_t u[4] = {v.x, v.y, v.z, v.w};
        #pragma unroll
        for (uint32_t q = 0; q < 4; ++q) {
            acc[2 * q] = fmaf(wj, __uint_as_float(u[q] << 16), acc[2 * q]);
            acc[2 * q + 1] = fmaf(wj, __uint_as_float(u[q] & 0xFFFF0000u), acc[2 * q + 1]);
        }
    }
    uint4 o;
    o.x = pack_bf16x2(acc[0], acc[1]);
    o.y = pack_bf16x2(acc[2], acc[3]);
    o.z = pack_bf16x2(acc[4], acc[5]);
    o.w = pack_bf16x2(acc[6], acc[7]);
    reinterpret_cast<uint4*>(out + static_cast<size_t>(t) * out_pitch)[c] = o;
}

// ---------------------------------------------------------------------------------------------
// Expert-parallel exchange over peer memory.  Every rank owns num_experts / world consecutive
// experts and exposes three buffers to its peers: the group-contiguous arena (e4m3 rows), the
// arena's packed scale words, and the result rows of its last grouped GEMM.  A step:
//   rank pairs    stable position of every (token, j) pair among this rank's pairs for its expert
//   block scan    per-expert totals of this rank (exchanged with a small all-gather)
//   layout        from all ranks' totals: where each expert's group starts on its owner, where this
//                 rank's rows go inside it, and the owner's group-end table for the grouped GEMM
//   dispatch      every pair's row and scale words are written straight to their arena row on the
//                 owner (plain stores to peer memory; no send buffer, no unpack pass)
//   combine       every token reads its topk result rows from the owners' result buffers and
//                 reduces them (plain loads from peer memory; no gather pass, no receive buffer)
// Cross-rank ordering (arena complete before the GEMM reads it, results complete before the
// combine reads them) is the host's job: a collective on the same stream between the steps.
// None of these kernels waits on another rank.
// ---------------------------------------------------------------------------------------------
constexpr uint32_t kEpChunk = 256;   // pairs per block of the ranking kernel

// local_rank[p] = number of earlier pairs of the same chunk with the same expert;
// block_hist[b * num_experts + e] = pairs of chunk b routed to expert e.  Expert ids outside
// [0, num_experts) are dropped (rank -1): such a pair is neither sent nor reduced.
// A warp's lanes with the same expert find one another in one instruction, the warps of a chunk take turns at its histogram (a walk over
// the earlier pairs of the chunk, up to 255 of them, took 1.5 us longer).
// kWhole: one block takes all chunks in turn and leaves what the scan below leaves, the pairs of the chunks before b in block_hist and
// the totals in counts: one launch instead of two, for the few chunks of a decode step.
template <bool kWhole>
__global__ void __launch_bounds__(kEpChunk) dg_ep_rank_pairs_kernel(const int32_t* expert_of_pair, uint32_t pairs, uint32_t num_experts,
                                                                    int32_t* local_rank, uint32_t* block_hist, uint32_t* counts) {
    griddep_wait();
    griddep_launch_dependents();
    extern __shared__ uint32_t ep_hist[];
    const uint32_t tid = threadIdx.x, lane = tid % 32, warp = tid / 32;
    for (uint32_t i = tid; i < num_experts; i += kEpChunk) ep_hist[i] = 0;
    const uint32_t first = kWhole ? 0u : blockIdx.x, past = kWhole ? (pairs + kEpChunk - 1) / kEpChunk : first + 1;
    auto expert = [&](uint32_t chunk) { return chunk * kEpChunk + tid < pairs ? ld_ro(expert_of_pair + chunk * kEpChunk + tid) : -1; };
    int32_t next = first < past ? expert(first) : -1;
    for (uint32_t chunk = first; chunk < past; ++chunk) {
        const int32_t e = next < 0 || static_cast<uint32_t>(next) >= num_experts ? -1 : next;
        if (chunk + 1 < past) next = expert(chunk + 1);
        const uint32_t same = __match_any_sync(0xFFFFFFFFu, e), before = __popc(same & ((1u << lane) - 1));
        uint32_t* const hist = block_hist + static_cast<size_t>(chunk) * num_experts;
        __syncthreads();
        const uint32_t start = e >= 0 ? ep_hist[e] : 0u;
        if constexpr (kWhole)
            for (uint32_t i = tid; i < num_experts; i += kEpChunk) hist[i] = ep_hist[i];
        uint32_t rank = 0;
        for (uint32_t w = 0; w < kEpChunk / 32; ++w) {
            __syncthreads();
            if (warp == w) {
                const uint32_t base = e >= 0 ? ep_hist[e] : 0u;
                __syncwarp();
                if (e >= 0 && before == 0) ep_hist[e] = base + __popc(same);
                rank = base - start + before;
            }
        }
        const uint32_t p = chunk * kEpChunk + tid;
        if (p < pairs) local_rank[p] = e >= 0 ? static_cast<int32_t>(rank) : -1;
    }
    __syncthreads();
    uint32_t* const totals = kWhole ? counts : block_hist + static_cast<size_t>(blockIdx.x) * num_experts;
    for (uint32_t i = tid; i < num_experts; i += kEpChunk) totals[i] = ep_hist[i];
}

// Exclusive scan over chunks, per expert, in place; counts[e] = this rank's pairs for expert e.  One warp per expert:
// 32 chunks per round (independent loads, shuffle scan), so a scan over hundreds of chunks costs a handful of memory
// round trips instead of one per chunk.
__global__ void __launch_bounds__(256) dg_ep_block_scan_kernel(uint32_t* block_hist, uint32_t num_blocks, uint32_t num_experts,
                                                               uint32_t* counts) {
    griddep_wait();
    griddep_launch_dependents();
    const uint32_t lane = threadIdx.x % 32;
    const uint32_t e = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
    if (e >= num_experts) return;
    uint32_t running = 0;
    for (uint32_t b0 = 0; b0 < num_blocks; b0 += 32) {
        const uint32_t b = b0 + lane;
        const size_t at = static_cast<size_t>(b) * num_experts + e;
        const uint32_t v = b < num_blocks ? block_hist[at] : 0u;
        uint32_t inc = v;                                     // inclusive scan over the 32 lanes
        #pragma unroll
        for (uint32_t d = 1; d < 32; d *= 2) {
            const uint32_t up = __shfl_up_sync(0xFFFFFFFFu, inc, d);
            if (lane >= d) inc += up;
        }
        if (b < num_blocks) block_hist[at] = running + inc - v;
        running += __shfl_sync(0xFFFFFFFFu, inc, 31);
    }
    if (lane == 0) counts[e] = running;
}

// all_counts: (world, num_experts) pairs per source rank and expert.  One block.
//   pair_base[e]   arena row (on the owner of e) of this rank's first pair for expert e
//   group_ends[l]  one past the last valid arena row of local expert l (the grouped GEMM's table)
//   totals[0..3]   arena rows in use on this rank (groups padded to `alignment`), valid rows on this
//                  rank, 1 if any owner's arena would exceed `capacity` rows (dispatch then drops the
//                  rows that do not fit), largest arena in use on any rank
// slot_rows != 0 selects the masked layout instead: local expert l owns the fixed slot of rows [l * slot_rows,
// (l + 1) * slot_rows), group_ends[l] is then its valid row count (the masked GEMM's masked_m), and the overflow flag is
// raised when some expert receives more than slot_rows rows (or the slots exceed `capacity`).
__global__ void __launch_bounds__(1024) dg_ep_layout_kernel(const uint32_t* all_counts, uint32_t world, uint32_t rank, uint32_t num_experts,
                                                            uint32_t alignment, uint32_t capacity, uint32_t slot_rows, uint32_t* pair_base,
                                                            uint32_t* group_ends, uint32_t* totals) {
    griddep_wait();
    griddep_launch_dependents();
    extern __shared__ uint32_t ep_smem[];
    uint32_t* rows_of = ep_smem;                  // [num_experts] rows of the expert over all source ranks
    uint32_t* before_me = ep_smem + num_experts;  // [num_experts] rows from lower source ranks
    uint32_t* start_of = ep_smem + 2 * num_experts;
    __shared__ uint32_t arena_rows[1024];
    const uint32_t local = num_experts / world;
    for (uint32_t e = threadIdx.x; e < num_experts; e += blockDim.x) {
        uint32_t total = 0, before = 0;
        for (uint32_t s = 0; s < world; ++s) {
            const uint32_t c = ld_ro(all_counts + static_cast<size_t>(s) * num_experts + e);
            if (s < rank) before += c;
            total += c;
        }
        rows_of[e] = total;
        before_me[e] = before;
    }
    __syncthreads();
    __shared__ uint32_t slot_overflow;
    if (threadIdx.x == 0) slot_overflow = 0;
    __syncthreads();
    // one warp per owner: padded group sizes scanned 32 experts at a time
    const uint32_t lane = threadIdx.x % 32;
    for (uint32_t owner = threadIdx.x / 32; owner < world; owner += blockDim.x / 32) {
        uint32_t running = 0, valid = 0;
        for (uint32_t l0 = 0; l0 < local; l0 += 32) {
            const uint32_t l = l0 + lane, e = owner * local + l;
            const uint32_t r = l < local ? rows_of[e] : 0u;
            const uint32_t padded = slot_rows ? (l < local ? slot_rows : 0u) : (r + alignment - 1) / alignment * alignment;
            if (slot_rows && r > slot_rows) slot_overflow = 1;
            uint32_t inc = padded, sum_r = r;
            #pragma unroll
            for (uint32_t d = 1; d < 32; d *= 2) {
                const uint32_t up = __shfl_up_sync(0xFFFFFFFFu, inc, d);
                if (lane >= d) inc += up;
                sum_r += __shfl_xor_sync(0xFFFFFFFFu, sum_r, d);
            }
            if (l < local) {
                const uint32_t start = running + inc - padded;
                start_of[e] = start;
                if (owner == rank) group_ends[l] = slot_rows ? r : start + r;
            }
            running += __shfl_sync(0xFFFFFFFFu, inc, 31);
            valid += sum_r;
        }
        if (lane == 0) {
            arena_rows[owner] = running;
            if (owner == rank) { totals[0] = running; totals[1] = valid; }
        }
    }
    __syncthreads();
    for (uint32_t e = threadIdx.x; e < num_experts; e += blockDim.x) pair_base[e] = start_of[e] + before_me[e];
    if (threadIdx.x == 0) {
        uint32_t largest = 0;
        for (uint32_t s = 0; s < world; ++s) largest = arena_rows[s] > largest ? arena_rows[s] : largest;
        totals[2] = (largest > capacity || slot_overflow) ? 1u : 0u;
        totals[3] = largest;
    }
}

// Warp loads (512 bytes) of a row that one warp of the dispatch holds, at most.  Eight take the per-token kernel from 64 to 76 registers
// (8192 tokens, top-8: 7168 bytes 93.8 -> 92.7 us, but 2048 bytes 28.9 -> 30.8; 1024 tokens x 7168 bytes 11.8 -> 15.6).
constexpr uint32_t kEpPieceLoads = 7;

struct EpDispatchParams {
    const int32_t* expert_of_pair;   // (pairs)
    const int32_t* local_rank;       // (pairs)
    const uint32_t* block_base;      // (chunks, num_experts) exclusive scan of the chunk histograms
    const uint32_t* pair_base;       // (num_experts)
    const uint8_t* data;             // (tokens, k) e4m3 rows of this rank's tokens
    const uint32_t* sf;              // packed scale words sf[c * sf_stride + token]
    uint8_t* const* peer_data;       // [world] arena of each rank, (capacity, k)
    uint32_t* const* peer_sf;        // [world] arena scale words, sf[c * peer_sf_stride + row]
    int32_t* pos_of_pair;            // (pairs) arena row on the owner, -1 if dropped
    uint32_t pairs, topk, k, sf_cols, sf_stride, peer_sf_stride, num_experts, experts_per_rank, capacity;
    uint32_t pieces, piece_loads;    // a token's row is cut into `pieces` of piece_loads warp loads, one warp each
    uint32_t slot_rows;              // masked layout: rows per expert slot (0: contiguous layout); the arena's scale words are then
                                     // laid out per slot, sf[(slot * sf_cols + c) * peer_sf_stride + row in slot]
};

// Arena row of a pair that has a rank among its expert's pairs, -1 if it does not fit; where its data and scale words go.
DG_DEVICE int32_t ep_arena_row(const EpDispatchParams& p, uint32_t pair, uint32_t local_rank, uint8_t*& dst, uint32_t*& dst_sf) {
    const uint32_t e = static_cast<uint32_t>(ld_ro(p.expert_of_pair + pair));
    const uint32_t row = ld_ro(p.pair_base + e) + ld_ro(p.block_base + static_cast<size_t>(pair / kEpChunk) * p.num_experts + e) + local_rank;
    const uint32_t owner = e / p.experts_per_rank, slot = e - owner * p.experts_per_rank;
    const uint32_t in_slot = row - slot * p.slot_rows;      // masked layout only
    if (row >= p.capacity || (p.slot_rows != 0 && in_slot >= p.slot_rows)) return -1;
    dst = p.peer_data[owner] + static_cast<size_t>(row) * p.k;
    dst_sf = p.peer_sf[owner] + (p.slot_rows ? static_cast<size_t>(slot) * p.sf_cols * p.peer_sf_stride + in_slot : row);
    return static_cast<int32_t>(row);
}

// Few tokens: one warp per (pair, piece of its token's row); grid.y is the piece.  Bound by the chain of dependent loads that leads to
// the arena row, beside which the piece is already on its way.  Top-8, 7168-byte rows: 16 tokens 2.1 us, 128 tokens 3.3 (a warp per
// token's piece, which stores to its experts' rows one after the other: 4.1 and 4.5; a warp per pair with a whole row, fetched after the
// chain: 3.5 and 3.7); 2048-byte rows 2.0 and 2.4 (3.5 and 3.6; 2.2 and 2.4).
__global__ void __launch_bounds__(256) dg_ep_dispatch_pairs_kernel(const EpDispatchParams p) {
    griddep_wait();
    griddep_launch_dependents();
    const uint32_t lane = threadIdx.x % 32, vecs = p.k / 16;
    const uint32_t piece_words = (p.sf_cols + p.pieces - 1) / p.pieces;
    for (uint64_t at = blockIdx.x * 8 + threadIdx.x / 32; at < p.pairs; at += gridDim.x * 8) {
        const uint32_t pair = static_cast<uint32_t>(at), tok = pair / p.topk;
        const int32_t lr = ld_ro(p.local_rank + pair);
        for (uint32_t piece = blockIdx.y; piece < p.pieces; piece += gridDim.y) {
            const uint4* src = reinterpret_cast<const uint4*>(p.data + static_cast<size_t>(tok) * p.k);
            const uint32_t first = piece * p.piece_loads * 32 + lane, past = (piece + 1) * p.piece_loads * 32, end = past < vecs ? past : vecs;
            const uint32_t word0 = piece * piece_words, words = word0 + piece_words < p.sf_cols ? word0 + piece_words : p.sf_cols;
            uint4 v[kEpPieceLoads];
            #pragma unroll
            for (uint32_t i = 0; i < kEpPieceLoads; ++i) {
                if (i >= p.piece_loads) break;
                if (first + 32 * i < end) v[i] = ld_ro(src + first + 32 * i);
            }
            const uint32_t word = word0 + lane;
            uint32_t x = 0;
            if (word < words) x = ld_ro(p.sf + static_cast<size_t>(word) * p.sf_stride + tok);
            uint8_t* dst = nullptr;
            uint32_t* dst_sf = nullptr;
            const int32_t row = lr < 0 ? -1 : ep_arena_row(p, pair, static_cast<uint32_t>(lr), dst, dst_sf);
            if (piece == 0 && lane == 0) p.pos_of_pair[pair] = row;
            if (row < 0) continue;
            uint4* to = reinterpret_cast<uint4*>(dst);
            #pragma unroll
            for (uint32_t i = 0; i < kEpPieceLoads; ++i) {
                if (i >= p.piece_loads) break;
                if (first + 32 * i < end) to[first + 32 * i] = v[i];
            }
            if (word < words) dst_sf[static_cast<size_t>(word) * p.peer_sf_stride] = x;
            for (uint32_t w = word + 32; w < words; w += 32)
                dst_sf[static_cast<size_t>(w) * p.peer_sf_stride] = ld_ro(p.sf + static_cast<size_t>(w) * p.sf_stride + tok);
        }
    }
}

// Many tokens: one warp per (token, up to 32 of its experts, piece of its row): the piece is read once and stored to the experts' arena
// rows.  A lane per expert works out where its copy goes; the whole warp then stores to one row after the other.  Bound by the stores
// (topk x k bytes per token): 8192 tokens, top-8: rows of 7168 bytes 94 us (a warp per pair, which reads every token top-k times from L2 and looks
// its row up as often: 118), 5120 bytes 69 (94), 4096 bytes 55 (71), 2048 bytes 29 (50).
// In both kernels the grid may be smaller than the work (warps stride over it), which lets a caller leave room on every SM for a
// kernel running beside this one.
__global__ void __launch_bounds__(256) dg_ep_dispatch_tokens_kernel(const EpDispatchParams p) {
    griddep_wait();
    griddep_launch_dependents();
    const uint32_t lane = threadIdx.x % 32, vecs = p.k / 16;
    const uint32_t parts = (p.topk + 31) / 32;
    const uint32_t units = p.pairs / p.topk * parts * p.pieces;      // fits 32 bits (checked by the host), the next one of a warp need not
    for (uint64_t at = blockIdx.x * 8 + threadIdx.x / 32; at < units; at += static_cast<uint64_t>(gridDim.x) * 8) {
        const uint32_t unit = static_cast<uint32_t>(at);
        const uint32_t row_part = unit / p.pieces, piece = unit - row_part * p.pieces;
        const uint32_t tok = row_part / parts, j0 = (row_part - tok * parts) * 32, here = p.topk - j0 < 32 ? p.topk - j0 : 32;
        const uint4* src = reinterpret_cast<const uint4*>(p.data + static_cast<size_t>(tok) * p.k);
        const uint32_t first = piece * p.piece_loads * 32 + lane, past = (piece + 1) * p.piece_loads * 32, end = past < vecs ? past : vecs;
        uint4 v[kEpPieceLoads];      // on its way while the rows are looked up
        #pragma unroll
        for (uint32_t i = 0; i < kEpPieceLoads; ++i)
            if (first + 32 * i < end) v[i] = ld_ro(src + first + 32 * i);
        // where the copy of expert j0 + lane goes: null if it is dropped
        uint8_t* dst = nullptr;
        uint32_t* dst_sf = nullptr;
        if (lane < here) {
            const uint32_t pair = tok * p.topk + j0 + lane;
            const int32_t lr = ld_ro(p.local_rank + pair);
            const int32_t row = lr < 0 ? -1 : ep_arena_row(p, pair, static_cast<uint32_t>(lr), dst, dst_sf);
            if (piece == 0) p.pos_of_pair[pair] = row;
        }
        const uint64_t dst_bits = reinterpret_cast<uint64_t>(dst), sf_bits = reinterpret_cast<uint64_t>(dst_sf);
        for (uint32_t j = 0; j < here; ++j) {
            uint4* to = reinterpret_cast<uint4*>(__shfl_sync(0xFFFFFFFFu, dst_bits, j));
            if (to == nullptr) continue;
            #pragma unroll
            for (uint32_t i = 0; i < kEpPieceLoads; ++i)
                if (first + 32 * i < end) to[first + 32 * i] = v[i];
        }
        // scale words: one (word, expert) per lane and step, the steps dealt out over the pieces
        const uint32_t words = p.sf_cols * here;
        for (uint32_t i0 = piece * 32; i0 < words; i0 += p.pieces * 32) {
            const uint32_t i = i0 + lane, w = i / here, j = i - w * here;
            uint32_t* to = reinterpret_cast<uint32_t*>(__shfl_sync(0xFFFFFFFFu, sf_bits, j));
            if (i < words && to != nullptr) to[static_cast<size_t>(w) * p.peer_sf_stride] = ld_ro(p.sf + static_cast<size_t>(w) * p.sf_stride + tok);
        }
    }
}

struct EpCombineParams {
    const int32_t* expert_of_pair;    // (tokens, topk)
    const int32_t* pos_of_pair;       // (tokens, topk) result row on the owner, < 0 skips the term
    const float* weights;             // (tokens, topk)
    const uint16_t* const* peer_rows; // [world] bf16 result rows of each rank, (capacity, pitch)
    uint16_t* out;                    // (tokens, out_pitch) bf16
    size_t pitch, out_pitch;
    uint32_t tokens, topk, n, experts_per_rank;
    uint32_t segments;                // of a token's row, one warp each
};

// out[t, :] = bf16( sum_j w[t, j] * rows_of_owner(t, j)[pos[t, j], :] ): the same ordered fused multiply-add
// chain as dg_moe_combine_kernel, reading each term from the rank that computed it.  One warp per (token, segment of its row), a lane
// 8 columns at a time: where the token's top-k rows are is worked out once per warp, a lane per row (every thread looking up all of
// them for its 8 columns cost 32 loads beside the 8 that move data).  Bound by reading topk x n x 2 bytes per token, and so by the loads
// in flight: 32 warps per SM (at most 64 registers; without the bound the compiler takes 79), and nothing done for rows beyond the top-k
// (which branches skip as a whole).  8192 tokens x 7168 columns, top-8: 236 us with a thread per 8 columns, 220 by pieces with 79
// registers and 8 rows whatever top-k is, 163.5 now; 1024 tokens 33.5, 36.9, 24.3; 128 tokens 5.7, 5.2, 4.1, of them with top-2 3.4, 4.2, 2.6.
__global__ void __launch_bounds__(256, 4) dg_ep_combine_kernel(const EpCombineParams p) {
    griddep_wait();
    griddep_launch_dependents();
    const uint32_t lane = threadIdx.x % 32;
    const uint32_t chunks = p.n / 8, per_segment = ((chunks + 31) / 32 + p.segments - 1) / p.segments * 32;
    const uint32_t units = p.tokens * p.segments, warps = gridDim.x * 8;      // fit 32 bits (checked by the host); a unit and a stride need not
    constexpr uint32_t kDeep = 8;      // rows whose loads are in flight before the first use
    for (uint32_t unit = blockIdx.x * 8 + threadIdx.x / 32; unit < units; unit = units - unit > warps ? unit + warps : units) {
        const uint32_t t = unit / p.segments, segment = unit - t * p.segments;
        const uint32_t first = segment * per_segment, end = first + per_segment < chunks ? first + per_segment : chunks;
        auto look_up = [&](uint32_t j, uint64_t& row_bits, float& weight) {
            row_bits = 0;
            weight = 0.0f;
            if (lane < kDeep && j + lane < p.topk) {
                const size_t at = static_cast<size_t>(t) * p.topk + j + lane;
                const int32_t row = ld_ro(p.pos_of_pair + at);
                const int32_t expert = ld_ro(p.expert_of_pair + at);
                weight = ld_ro(p.weights + at);
                if (row >= 0) row_bits = reinterpret_cast<uint64_t>(p.peer_rows[static_cast<uint32_t>(expert) / p.experts_per_rank] + static_cast<size_t>(row) * p.pitch);
            }
        };
        uint64_t row_bits;
        float weight;
        look_up(0, row_bits, weight);
        for (uint32_t c0 = first; c0 < end; c0 += 32) {
            const uint32_t c = c0 + lane;
            float2 acc[4] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
            for (uint32_t j0 = 0; j0 < p.topk; j0 += kDeep) {
                if (p.topk > kDeep) look_up(j0, row_bits, weight);
                const uint32_t here = p.topk - j0 < kDeep ? p.topk - j0 : kDeep;
                uint4 v[kDeep];
                #pragma unroll
                for (uint32_t u = 0; u < kDeep; ++u) {
                    if (u >= here) break;
                    const uint4* row = reinterpret_cast<const uint4*>(__shfl_sync(0xFFFFFFFFu, row_bits, u));
                    if (row != nullptr && c < end) v[u] = *(row + c);
                }
                #pragma unroll
                for (uint32_t u = 0; u < kDeep; ++u) {
                    if (u >= here) break;
                    if (__shfl_sync(0xFFFFFFFFu, row_bits, u) == 0) continue;
                    const float wj = __shfl_sync(0xFFFFFFFFu, weight, u);
                    const uint32_t w[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
                    #pragma unroll
                    for (uint32_t q = 0; q < 4; ++q)
                        acc[q] = __ffma2_rn(make_float2(wj, wj), make_float2(__uint_as_float(w[q] << 16), __uint_as_float(w[q] & 0xFFFF0000u)), acc[q]);
                }
            }
            if (c < end) {
                uint4 o;
                o.x = pack_bf16x2(acc[0].x, acc[0].y);
                o.y = pack_bf16x2(acc[1].x, acc[1].y);
                o.z = pack_bf16x2(acc[2].x, acc[2].y);
                o.w = pack_bf16x2(acc[3].x, acc[3].y);
                reinterpret_cast<uint4*>(p.out + static_cast<size_t>(t) * p.out_pitch)[c] = o;
            }
        }
    }
}

}  // namespace dg
