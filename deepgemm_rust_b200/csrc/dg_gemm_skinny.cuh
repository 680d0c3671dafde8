// Dense e4m3 GEMM with per-128 scales for a handful of activation rows (decode-time projections through small matrices).
//
// What bounds such a call is not the weight stream but everything around it: with the tiles of the first family 8 x 2112 x 7168 took
// 10.5 us, of which the 15 MB of weights are 2.4: the start-up of a kernel with tensor maps, TMEM and rings, its drain, f32 planes of the
// K ranges, and a second launch that sums them.  Here a block owns 16 weight rows (output columns) over the whole of K; its warps deal
// the K blocks out among themselves and bring them from global memory straight to registers, where a 16-byte piece of a row is a lane's share of two
// warp-wide matrix instructions (e4m3 in, f32 sums); the warps' sums meet in shared memory.  One launch, no workspace, nothing set up
// before the first load.  Quantiser and GEMM together: 8 x 2112 x 7168 12.1 -> 8.0 us, which is what the host needs for the two calls;
// 3 x 6664 x 4608 16.5 -> 10.7.  (With the codes turned into f16 first, for the instruction of half the depth: the same error, up to 6 %
// slower.)  With more rows or weights the latency of plain loads shows, and the tensor-memory kernels are the better ones.
//
// A K block of 128 is multiplied on its own, scaled by the two power-of-two scales and added to f32 sums.  The order of K inside a block
// is the same for both operands and otherwise free, so that a lane's 16-byte pieces of a row are its share of the fragments.
#pragma once
#include "dg_ptx.cuh"

namespace dg {

constexpr uint32_t kSkinnyCols = 16;      // weight rows (output columns) of a block

struct SkinnyParams {
    const uint8_t* a;          // activations (m, a_ld) e4m3
    const uint8_t* b;          // weights (n, b_ld) e4m3
    const uint32_t* sfa;       // packed UE8M0 words: [word column * stride + row]
    const uint32_t* sfb;
    void* out;                 // (m, out_ld) bf16 or f32
    uint32_t m, n, k_blocks, a_ld, b_ld, sfa_stride, sfb_stride, out_ld;
    uint32_t has_alpha, accumulate;
    float alpha;
};

// Shared memory of a block, in the kernel's static array (host side).
constexpr uint32_t skinny_smem_bytes(uint32_t row_tiles, uint32_t warps) { return warps * row_tiles * 8 * (kSkinnyCols + 1) * 4; }

DG_DEVICE void mma_16x8x32_e4m3(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.f32.e4m3.e4m3.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// x * 2^(e - 254) for the sum e of two UE8M0 exponents, in two steps that stay inside the range of f32 wherever the result does.
DG_DEVICE float scale_by_exponents(float x, uint32_t ea, uint32_t eb) {
    const int32_t e = static_cast<int32_t>(ea + eb) - 254, h = e >> 1;
    const float y = x * __uint_as_float(static_cast<uint32_t>(h + 127) << 23) * __uint_as_float(static_cast<uint32_t>(e - h + 127) << 23);
    return ea == 255 || eb == 255 ? __uint_as_float(0x7FC00000u) : y;      // 255 is NaN
}

// kTiles: activation rows in tiles of 8.  kWarps of a block share K.
template <uint32_t kTiles, uint32_t kWarps, bool kF32>
__global__ void __launch_bounds__(kWarps * 32, 16 / kWarps) dg_gemm_skinny_kernel(const __grid_constant__ SkinnyParams p) {
    __shared__ float sums[kWarps][kTiles * 8][kSkinnyCols + 1];
    griddep_wait();
    griddep_launch_dependents();
    const uint32_t warp = threadIdx.x / 32, lane = threadIdx.x % 32, g = lane / 4, t = lane % 4;
    const uint32_t n0 = blockIdx.x * kSkinnyCols;
    // rows beyond the matrix read the last one; what they give is not stored
    const uint32_t w_row[2] = {min(n0 + g, p.n - 1), min(n0 + g + 8, p.n - 1)};
    const uint8_t* w_at[2] = {p.b + static_cast<size_t>(w_row[0]) * p.b_ld + t * 16, p.b + static_cast<size_t>(w_row[1]) * p.b_ld + t * 16};
    float acc[kTiles][4];
    #pragma unroll
    for (uint32_t i = 0; i < kTiles; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.0f;
    struct Block {      // what a lane holds of a K block
        uint4 w[2][2], x[kTiles][2];
        uint32_t w_sf[2], x_sf[kTiles][2];
    };
    auto load = [&](Block& c, uint32_t kb) {
        const size_t k0 = static_cast<size_t>(kb) * 128;
        #pragma unroll
        for (uint32_t r = 0; r < 2; ++r)
            #pragma unroll
            for (uint32_t j = 0; j < 2; ++j) c.w[r][j] = ld_ro(reinterpret_cast<const uint4*>(w_at[r] + k0 + j * 64));
        #pragma unroll
        for (uint32_t r = 0; r < 2; ++r) c.w_sf[r] = ld_ro(p.sfb + static_cast<size_t>(kb / 4) * p.sfb_stride + w_row[r]);
        #pragma unroll
        for (uint32_t i = 0; i < kTiles; ++i) {
            const uint8_t* x_at = p.a + static_cast<size_t>(min(i * 8 + g, p.m - 1)) * p.a_ld + t * 16 + k0;
            #pragma unroll
            for (uint32_t j = 0; j < 2; ++j) c.x[i][j] = ld_ro(reinterpret_cast<const uint4*>(x_at + j * 64));
            #pragma unroll
            for (uint32_t v = 0; v < 2; ++v) c.x_sf[i][v] = ld_ro(p.sfa + static_cast<size_t>(kb / 4) * p.sfa_stride + min(i * 8 + 2 * t + v, p.m - 1));
        }
    };
    auto multiply = [&](const Block& c, uint32_t kb) {
        float d[kTiles][4];
        #pragma unroll
        for (uint32_t i = 0; i < kTiles; ++i) d[i][0] = d[i][1] = d[i][2] = d[i][3] = 0.0f;
        #pragma unroll
        for (uint32_t j = 0; j < 2; ++j) {
            const uint32_t w0[4] = {c.w[0][j].x, c.w[0][j].y, c.w[0][j].z, c.w[0][j].w}, w1[4] = {c.w[1][j].x, c.w[1][j].y, c.w[1][j].z, c.w[1][j].w};
            #pragma unroll
            for (uint32_t q = 0; q < 4; q += 2)
                #pragma unroll
                for (uint32_t i = 0; i < kTiles; ++i) {
                    const uint32_t y[4] = {c.x[i][j].x, c.x[i][j].y, c.x[i][j].z, c.x[i][j].w};
                    mma_16x8x32_e4m3(d[i], w0[q], w1[q], w0[q + 1], w1[q + 1], y[q], y[q + 1]);
                }
        }
        const uint32_t shift = 8 * (kb & 3);
        #pragma unroll
        for (uint32_t i = 0; i < kTiles; ++i)
            #pragma unroll
            for (uint32_t v = 0; v < 4; ++v)
                acc[i][v] += scale_by_exponents(d[i][v], (c.w_sf[v / 2] >> shift) & 0xFF, (c.x_sf[i][v % 2] >> shift) & 0xFF);
    };
    Block now;
    if constexpr (kTiles <= 2) {
        // the next K block of the warp is on its way while the present one is multiplied
        Block next;
        if (warp < p.k_blocks) load(now, warp);
        for (uint32_t kb = warp; kb < p.k_blocks; kb += 2 * kWarps) {
            const bool second = kb + kWarps < p.k_blocks;
            if (second) load(next, kb + kWarps);
            multiply(now, kb);
            if (kb + 2 * kWarps < p.k_blocks) load(now, kb + 2 * kWarps);
            if (second) multiply(next, kb + kWarps);
        }
    } else {
        #pragma unroll 1
        for (uint32_t kb = warp; kb < p.k_blocks; kb += kWarps) {
            load(now, kb);
            multiply(now, kb);
        }
    }
    #pragma unroll
    for (uint32_t i = 0; i < kTiles; ++i)
        #pragma unroll
        for (uint32_t v = 0; v < 4; ++v) sums[warp][i * 8 + 2 * t + v % 2][g + 8 * (v / 2)] = acc[i][v];
    __syncthreads();
    // A thread per output, its sums added in the order of the warps; all of a thread's outputs before the first is stored.  Accumulation adds in memory, as the
    // first family's TMA reduction does: calls on two streams may add into one output.
    constexpr uint32_t kOutputs = kTiles * 8 * kSkinnyCols, kEach = (kOutputs + kWarps * 32 - 1) / (kWarps * 32);
    static_assert(kEach == 1 || kOutputs % (kWarps * 32) == 0, "a thread has all of its outputs or none");
    float out[kEach];
    #pragma unroll
    for (uint32_t i = 0; i < kEach; ++i) {
        const uint32_t o = threadIdx.x + i * kWarps * 32, row = o / kSkinnyCols, col = o % kSkinnyCols;
        if (o >= kOutputs) return;
        out[i] = 0.0f;
        #pragma unroll
        for (uint32_t w = 0; w < kWarps; ++w) out[i] += sums[w][row][col];
        if (p.has_alpha) out[i] *= p.alpha;
    }
    #pragma unroll
    for (uint32_t i = 0; i < kEach; ++i) {
        const uint32_t o = threadIdx.x + i * kWarps * 32, row = o / kSkinnyCols, col = o % kSkinnyCols;
        if (row >= p.m || n0 + col >= p.n) continue;
        const size_t at = static_cast<size_t>(row) * p.out_ld + n0 + col;
        if constexpr (kF32) {
            float* d = static_cast<float*>(p.out) + at;
            if (p.accumulate) red_add_f32(d, out[i]);
            else *d = out[i];
        } else {
            uint16_t* d = static_cast<uint16_t*>(p.out) + at;
            const uint16_t y = static_cast<uint16_t>(pack_bf16x2(out[i], 0.0f));
            if (p.accumulate) red_add_bf16(d, y);
            else *d = y;
        }
    }
}

}  // namespace dg
