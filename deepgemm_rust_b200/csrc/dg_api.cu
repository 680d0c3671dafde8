// Host side of the C ABI declared in include/dgb200.h: context, argument validation, tile
// configuration, tensor-map encoding and kernel launches.  No CPU compute path exists here:
// every entry point either launches sm_100a kernels or returns an error.
#include <cuda.h>
#include <cuda_runtime.h>
#include <unistd.h>

#include <atomic>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <new>
#include <string>

#include "../../include/dgb200.h"
#include "dg_cast_kernels.cuh"
#include "dg_gemm_kernel.cuh"
#include "dg_gemm_swap.cuh"
#include "dg_gemm_f32scale.cuh"
#include "dg_gemm_wide.cuh"
#include "dg_gemm_skinny.cuh"
#include "dg_moe_kernels.cuh"

namespace {

thread_local std::string g_last_error;

int fail(int code, const char* fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    g_last_error = buf;
    return code;
}

#define DG_CUDA(expr)                                                                            \
    do {                                                                                         \
        cudaError_t e_ = (expr);                                                                 \
        if (e_ != cudaSuccess) return fail(DG_ERR_DRIVER, "%s: %s", #expr, cudaGetErrorString(e_)); \
    } while (0)

std::atomic<uint32_t> g_mk_alignment{128};

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                   const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled_fn() {
    static EncodeTiledFn fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess)
            p = nullptr;
        return reinterpret_cast<EncodeTiledFn>(p);
    }();
    return fn;
}

constexpr uint32_t kSmemCapacity = 232448;  // 227 KB opt-in maximum per CTA on sm_100

uint32_t align4(uint32_t x) { return (x + 3) / 4 * 4; }
uint32_t ceil_div(uint32_t a, uint32_t b) { return (a + b - 1) / b; }

}  // namespace

// A device buffer that grows on demand.
struct ScratchBuffer {
    void* ptr = nullptr;
    size_t bytes = 0;
    bool captured = false;      // a captured graph may hold its address: it stays until the context goes
};
struct ScratchBlock {
    void* ptr;
    ScratchBlock* next;
};

// What the calls of one stream share: they run one after the other.
struct Scratch {
    cudaStream_t stream = nullptr;
    bool orphaned = false;              // the stream was the context's own and is destroyed; another may get its handle
    ScratchBuffer group_ends;           // group-end table of the contiguous layout
    ScratchBuffer splitk_ws;            // f32 partial products of K-split GEMMs
    ScratchBuffer splitk_counters;      // K ranges that have arrived, per tile (swapped tile family); zero between launches
    ScratchBuffer bridge_sf[2];         // packed scale words built from f32 scales by the f32-scale entry points
    Scratch* next = nullptr;
};

struct dg_ctx {
    int ordinal = 0;
    cudaStream_t stream = nullptr;
    bool owns_stream = false;
    int num_sms = 0;
    dg::Status* status = nullptr;       // device word block the kernels report into
    Scratch first;                      // one set per stream the context has been used on
    Scratch* scratch = &first;          // of `stream`
    ScratchBlock* replaced = nullptr;   // outgrown buffers that a captured graph may still use
};

extern "C" {

const char* dg_last_error(void) { return g_last_error.c_str(); }

static int ctx_create(int ordinal, void* stream, bool adopt, dg_ctx** out) {
    if (out == nullptr) return fail(DG_ERR_SHAPE, "null output pointer");
    int count = 0;
    cudaError_t e = cudaGetDeviceCount(&count);
    if (e != cudaSuccess || count == 0)
        return fail(DG_ERR_DRIVER, "no CUDA device available (%s); this library has no CPU path", cudaGetErrorString(e));
    if (ordinal < 0 || ordinal >= count) return fail(DG_ERR_SHAPE, "device ordinal %d out of range (0..%d)", ordinal, count - 1);
    DG_CUDA(cudaSetDevice(ordinal));
    cudaDeviceProp prop;
    DG_CUDA(cudaGetDeviceProperties(&prop, ordinal));
    if (prop.major != 10)
        return fail(DG_ERR_UNSUPPORTED, "device %d is sm_%d%d; these kernels are built for sm_100a only", ordinal, prop.major, prop.minor);
    if (encode_tiled_fn() == nullptr) return fail(DG_ERR_DRIVER, "cuTensorMapEncodeTiled not found in the driver");
    dg_ctx* c = new dg_ctx();
    c->ordinal = ordinal;
    c->num_sms = prop.multiProcessorCount;
    if (adopt) {
        c->stream = static_cast<cudaStream_t>(stream);
    } else {
        if (cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking) != cudaSuccess) { delete c; return fail(DG_ERR_DRIVER, "cudaStreamCreate failed"); }
        c->owns_stream = true;
    }
    c->first.stream = c->stream;
    if (cudaMalloc(&c->status, sizeof(dg::Status)) != cudaSuccess || cudaMemset(c->status, 0, sizeof(dg::Status)) != cudaSuccess) {
        delete c;
        return fail(DG_ERR_DRIVER, "allocating the device status word failed");
    }
    *out = c;
    return DG_OK;
}

int dg_ctx_create(int ordinal, dg_ctx** out) { return ctx_create(ordinal, nullptr, false, out); }
int dg_ctx_create_on_stream(int ordinal, void* cuda_stream, dg_ctx** out) { return ctx_create(ordinal, cuda_stream, true, out); }

int dg_ctx_destroy(dg_ctx* ctx) {
    if (ctx == nullptr) return DG_OK;
    cudaSetDevice(ctx->ordinal);
    if (ctx->status) cudaFree(ctx->status);
    for (Scratch *set = &ctx->first, *next; set != nullptr; set = next) {
        next = set->next;
        for (ScratchBuffer* b : {&set->group_ends, &set->splitk_ws, &set->splitk_counters, &set->bridge_sf[0], &set->bridge_sf[1]})
            if (b->ptr) cudaFree(b->ptr);
        if (set != &ctx->first) delete set;
    }
    while (ScratchBlock* block = ctx->replaced) {
        ctx->replaced = block->next;
        cudaFree(block->ptr);
        delete block;
    }
    if (ctx->owns_stream && ctx->stream) cudaStreamDestroy(ctx->stream);
    delete ctx;
    return DG_OK;
}

int dg_ctx_check_status(dg_ctx* ctx) {
    if (ctx == nullptr) return fail(DG_ERR_SHAPE, "null context");
    dg::Status st;
    DG_CUDA(cudaMemcpy(&st, ctx->status, sizeof(st), cudaMemcpyDeviceToHost));
    if (st.code != 0) {
        cudaMemset(ctx->status, 0, sizeof(st));
        for (Scratch* set = &ctx->first; set != nullptr; set = set->next)
            if (set->splitk_counters.ptr) cudaMemset(set->splitk_counters.ptr, 0, set->splitk_counters.bytes);   // the kernel may have left some
        return fail(DG_ERR_TIMEOUT, "a device-side wait ran out: block %u, site 0x%x, parity %u", st.block, st.site, st.extra);
    }
    return DG_OK;
}

int dg_ctx_sync(dg_ctx* ctx) {
    if (ctx == nullptr) return fail(DG_ERR_SHAPE, "null context");
    DG_CUDA(cudaStreamSynchronize(ctx->stream));
    return dg_ctx_check_status(ctx);
}

int dg_ctx_num_sms(const dg_ctx* ctx, int* out) {
    if (ctx == nullptr || out == nullptr) return fail(DG_ERR_SHAPE, "null argument");
    *out = ctx->num_sms;
    return DG_OK;
}
void* dg_ctx_stream(const dg_ctx* ctx) { return ctx ? ctx->stream : nullptr; }
int dg_ctx_set_stream(dg_ctx* ctx, void* cuda_stream) {
    if (ctx == nullptr) return fail(DG_ERR_SHAPE, "null context");
    const cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
    // work queued on the old stream may still run beside the new stream's: that one gets scratch of its own
    const bool ends = ctx->owns_stream && ctx->stream;
    Scratch* set = ctx->scratch;
    if (ends || stream != ctx->stream)
        for (set = &ctx->first; set != nullptr; set = set->next)
            if (set->stream == stream && !set->orphaned && !(ends && set == ctx->scratch)) break;
    if (set == nullptr) {
        set = new (std::nothrow) Scratch;
        if (set == nullptr) return fail(DG_ERR_DRIVER, "out of host memory");
        set->stream = stream;
        set->next = ctx->first.next;
        ctx->first.next = set;
    }
    if (ends) {
        ctx->scratch->orphaned = true;
        cudaStreamDestroy(ctx->stream);
    }
    ctx->owns_stream = false;
    ctx->stream = stream;
    ctx->scratch = set;
    return DG_OK;
}

// ------------------------------------------------------------------ size helpers / knobs
uint32_t dg_sf_packed_cols(uint32_t k, uint32_t gran_k) { return gran_k ? ceil_div(k, gran_k * 4) : 0; }
uint32_t dg_sf_aligned_rows(uint32_t rows) { return align4(rows); }
size_t dg_sf_words(uint32_t rows, uint32_t k, uint32_t gran_k, uint32_t num_groups) {
    const uint32_t g = num_groups ? num_groups : 1;
    return static_cast<size_t>(dg_sf_packed_cols(k, gran_k)) * g * align4(rows / g);
}

int dg_set_mk_alignment_for_contiguous_layout(uint32_t value) {
    if (value < 16 || value > 256 || (value & (value - 1)) != 0)
        return fail(DG_ERR_SHAPE, "mk alignment must be a power of two in [16, 256], got %u", value);
    g_mk_alignment.store(value);
    return DG_OK;
}
uint32_t dg_get_mk_alignment_for_contiguous_layout(void) { return g_mk_alignment.load(); }
uint32_t dg_get_theoretical_mk_alignment_for_contiguous_layout(uint32_t arch_major) { return arch_major == 10 ? 256u : 128u; }

// ------------------------------------------------------------------------- heuristics
// Tile choice for 148 SMs / 227 KB shared memory / 512 TMEM columns.  In the first tile family A rows ride the UMMA M dimension (128
// per CTA); BLOCK_N is picked from the widths the epilogue of the output type can store, minimising waves x per-tile cost; stages
// fill the shared memory left over.  prefer_swapped says which problems the second family gets, with weight rows on UMMA M.
// What the launcher needs to know about a choice (the public dg_config describes the same choice in the reference's terms).
struct KernelPlan {
    bool swap;                 // weights on the UMMA M dimension, activation rows on UMMA N
    uint32_t ctas, umma_n, halves, stages, accum, smem;
    uint32_t splits;           // K ranges: summed by a second kernel (first tile family) or by the last range to arrive (swapped)
    uint32_t tiles;
    uint32_t epi_bufs;         // staging buffers of an epilogue warp (first tile family)
    uint32_t block_n2;         // wide tiles: columns of the second half (0: not a wide tile)
    uint32_t table_groups;     // groups whose rows and tiles are kept in shared memory (swapped family)
    uint32_t skinny_warps;     // the kernel for a handful of rows: warps of its blocks (0: another kernel)
};
// What a call rules out that its description does not tell: K ranges (the caller adds into the output: their sum is written, not added), wide
// tiles (no bf16 operands), the kernel for a handful of rows (neither bf16 operands nor a duty cycle).
constexpr uint32_t kNoKRanges = 1, kNoWideTiles = 2, kNoSkinny = 4;
static int search_config(const dg_desc* d, uint32_t limits, dg_config* out, KernelPlan* plan);
int dg_best_config(const dg_desc* d, dg_config* out) {
    KernelPlan plan;
    return search_config(d, 0, out, &plan);
}

// What the DG_* knobs say, as a hash of their text (0 if none is set); they may change between two calls.
// One pass over the environment takes 50 ns; asking for every knob by name 54 ns each.
static uint64_t knob_signature() {
    uint64_t h = 0;
    for (char** e = environ; e != nullptr && *e != nullptr; ++e) {
        if ((*e)[0] != 'D' || (*e)[1] != 'G' || (*e)[2] != '_') continue;
        for (const char* c = *e; *c != 0; ++c) h = (h ^ static_cast<unsigned char>(*c)) * 0x100000001B3ull;
        h = (h ^ '\n') * 0x100000001B3ull + 1;
    }
    return h;
}

// search_config with the choices of recent problems remembered: the search walks ~500 candidates (3.7 us on a B200 host, more
// than the launch itself), and a program asks for the same few problems again and again.  The choice is a function of the
// description, the alignment and the knobs alone.  One small table per thread, overwritten on collision.
static int choose_config(const dg_desc* d, uint32_t limits, dg_config* out, KernelPlan* plan) {
    struct Key {
        dg_desc desc;
        uint32_t limits, alignment;
        uint32_t knobs[2];
    };
    struct Entry {
        bool used;
        Key key;
        dg_config cfg;
        KernelPlan plan;
    };
    constexpr uint32_t kEntries = 64;
    static thread_local Entry table[kEntries];
    const uint64_t knobs = knob_signature();
    const Key key = {*d, limits, g_mk_alignment.load(), {static_cast<uint32_t>(knobs), static_cast<uint32_t>(knobs >> 32)}};
    static_assert(sizeof(Key) == 18 * sizeof(uint32_t), "compared and hashed as 18 words");
    uint32_t words[18], hash = 0;
    memcpy(words, &key, sizeof(key));
    for (uint32_t w : words) hash = (hash ^ w) * 0x9E3779B1u;
    Entry& e = table[(hash >> 16) % kEntries];
    if (!e.used || memcmp(&e.key, &key, sizeof(key)) != 0) {
        const int rc = search_config(d, limits, &e.cfg, &e.plan);
        e.used = rc == DG_OK;
        if (rc) return rc;
        e.key = key;
    }
    *out = e.cfg;
    *plan = e.plan;
    return DG_OK;
}

// Rows of a group of the contiguous layout, as far as the host knows them: the arena's rows include the alignment padding.
static double contiguous_rows(uint32_t m, uint32_t groups) {
    const double per_group = static_cast<double>(m) / groups, padding = g_mk_alignment.load() / 2.0;
    return per_group > padding ? per_group - padding : per_group;
}
static double group_rows(const dg_desc* d) {
    if (d->gemm_type == DG_GEMM_M_GROUPED_CONTIGUOUS) return contiguous_rows(d->m, d->num_groups ? d->num_groups : 1);
    if (d->gemm_type == DG_GEMM_M_GROUPED_MASKED) return d->expected_m < d->m ? d->expected_m : d->m;
    return d->m;
}

// Is the swapped family the better one for this problem?  Measured on B200 over 920 grouped problems (4-128 groups of 4-1200 rows,
// equal and skewed, n 128-7168, k 1024-7168), both families side by side.  It wins where a group's rows fit one tile and there is
// enough to stream (masked 32 x <= 256 rows, 4096 x 7168: 247 -> 199 us; contiguous 256 x 256 rows: 486 -> 430 us at 4096 x 7168,
// 263 -> 237 us at 7168 x 2048).  It loses
//   with few tiles: below half a wave of pair tiles (masked) or one wave (contiguous) it took 1.2-1.3 times as long over 300 problems,
//     because its tiles are 256 weight rows wide where the first family goes down to 32;
//   with short K, where its start-up and the transposed epilogue show: below 2048 bytes 1.17-1.24 times on average (34 x 64 rows,
//     1792 x 1024: 22 -> 31 us).  Up to 28 slabs of 128 bytes it is the better one for e4m3 output (the first family then has
//     tiles of 128 and 256 columns only), for masked groups with 4096 columns and two waves, and for contiguous groups of 160-320
//     rows (one tile of its, two of the other's); else it takes up to 1.4 times as long (20 x 36 rows, 1792 x 2048: 17.9 -> 24.5 us);
//   with fewer than 2048 columns in the contiguous layout (up to 1.4 times: 28 x 40 rows, 1088 x 6144: 54 -> 75 us);
//   with groups of two tiles and more, which fill the first family's 256-row tiles as well (900 rows: 750 -> 808 us).
// With these lines it is chosen for a third of them; on average they take 0.95 (masked) and 0.99 (contiguous) of the first family's
// time, at most 1.34; chosen wherever K had 2048 bytes and groups up to 450 rows it was 0.99 and 1.02, at most 2.0.
// Only with per-128 scales on both sides: a per-32 operand (every e2m1 one) brings new scale words with each k-block, which one
// warp re-orders for a narrow tile.  Over 90 grouped problems with one it took 1.6 to 4.9 times as long as the first family
// (64 x 12 rows, 1984 x 3072, e4m3 x e2m1: 72 -> 222 us), over 20 dense ones up to 1.7 times (2 x 11992 x 10752: 34 -> 57 us).
static bool prefer_swapped(const dg_desc* d) {
    if (d->cd_dtype == DG_OUT_SWIGLU_FP8) return false;
    if (d->a_bits != 8 || d->b_bits != 8 || d->gran_a != 128 || d->gran_b != 128) return false;
    const uint32_t sms = d->num_sms ? d->num_sms : 148, slabs = ceil_div(d->k, 128), groups = d->num_groups ? d->num_groups : 1;
    if (d->gemm_type == DG_GEMM_M_GROUPED_MASKED || d->gemm_type == DG_GEMM_M_GROUPED_CONTIGUOUS) {
        const double rows = group_rows(d), waves = static_cast<double>(groups) * ceil_div(d->n, 256) / (sms / 2.0);
        if (d->k < 2048 || rows > 450.0) return false;
        if (d->gemm_type == DG_GEMM_M_GROUPED_MASKED) return waves >= 0.5 && (d->cd_dtype == DG_OUT_FP8 || slabs >= 28 || (waves >= 2.0 && d->n >= 4096));
        // (an arena with fewer rows per group than the alignment is one of mostly empty groups, about which nothing was measured)
        return waves >= 1.0 && d->n >= 2048 && (slabs >= 28 || (rows >= 160.0 && rows <= 320.0)) && d->m / groups >= g_mk_alignment.load();
    }
    // Dense e4m3, a few rows: where the weight blocks alone fill half of the SMs in one wave (four fifths above 32 rows), a CTA streams
    // its 128 weight rows without K ranges and without a second launch (8 x 17056 x 8192: 41 -> 26 us; 28 x 9872 x 4608: 17.2 -> 15.4;
    // 53 x 18600 x 10240: 38 -> 34).  With more than one wave or more rows the first family's K ranges are as fast or
    // faster.
    const uint32_t blocks = ceil_div(d->n, 128);
    // With fewer blocks it still wins where K is short: it takes 4.4 us + 0.31 us per 128 bytes of K whatever n is, the K ranges with
    // their second launch 8.2 us + 0.17 us per MB of weights (up to 32 rows and from 25 blocks on, 13 problems: 3680 x 2048
    // 12.2 -> 8.9 us, 5208 x 1536 10.6 -> 8.6, 9040 x 2560 15.3 -> 10.6; 0.99 to 1.44 times as fast; with fewer blocks 0.88 times).
    const bool short_k = 6 * blocks >= sms && slabs * 0.31 < 3.8 + 0.17 * blocks * slabs * (128 * 128 / 1e6);
    return d->gemm_type == DG_GEMM_NORMAL && blocks <= sms &&
           ((d->m <= 32 && (2 * blocks >= sms || short_k)) || (d->m <= 64 && 5 * blocks >= 4 * sms));
}

// Is the kernel for a handful of activation rows (dg_gemm_skinny.cuh) the one for this problem?  Measured against the other kernels over 1263
// problems (m 1-32, n 16-343744, k 128-62464), the GEMM alone, in a loop and in a graph of 24, weights from DRAM.  What bounds it is the latency of plain
// loads: a warp's rounds of K blocks, times the waves of blocks (four of four warps fit an SM).  Inside the lines below it takes 0.73 of the
// others' time on average and 1.10 at most (16 x 512 x 12288); behind the activation quantiser, where its shorter start-up shows, 0.93 and 1.03 at most over the
// 69 problems nearest to the lines, 0.88 at most with weights in L2.  The figures are of the graphs, or of both launches where it says so.
//   Up to 8 rows it wins to 64 MB (5 x 4472 x 13312: 17.4 -> 14.4 us; 1 x 6144 x 9728: 17.3 -> 17.3), to 44 where the swapped family
//     fills the SMs (8 x 16384 x 2560: 11.6 -> 11.0), and to 16384 of K (8 x 256 x 16384: 8.7 -> 8.2, x 32768: 10.5 -> 14.8), 24576 where blocks of 16 warps
//     take more than half of the SMs (8 x 1280 x 24576: 13.0 -> 12.7; 8 x 1024 x 28672: 13.2 -> 13.7).
//   9-16 rows: while the blocks fit at once to 24 MB (16 x 9472 x 2304: 9.9 -> 8.7) and 7168 of K (16 x 2400 x 6656: 10.6 -> 10.6), with 16 warps
//     12288 (16 x 1024 x 12288: 9.8 -> 9.7; 16 x 512: 8.7 -> 9.6, with the quantiser 12.5 -> 12.1), or 10240 with so few blocks that K ranges occupy more SMs (16 x 16 x
//     10240: 7.2 -> 7.1, x 12288: 7.2 -> 8.1); in two waves two rounds of K (16 x 18432 x 1024: 8.8 -> 8.1, x 1152: 9.5 -> 9.9), in more one, or two full ones
//     (16 x 28672 x 512: 8.6 -> 7.6, x 640: 9.3 -> 10.8; 16 x 22528 x 1024: 9.9 -> 9.9, with the quantiser 12.6 -> 12.5, x 896: 9.3 -> 9.6).
//   17-32 rows, whose K blocks are not prefetched: to 8 MB and 4096 of K (32 x 3072 x 2560: 9.5 -> 8.5), with four warps two rounds
//     of K (32 x 6144 x 1024: 6.7 -> 6.8, with the quantiser 10.3 -> 9.0, x 1280: 7.5 -> 8.3), in two waves one round (32 x 12288 x 512: 6.7 -> 6.7, x 640: 7.3 -> 9.7).
//   More short blocks than 14 (7) per SM: 8 x 65536 x 128 9.0 -> 9.2, 8 x 343744 x 128 30.7 -> 42.4, 32 x 32768 x 128 6.8 -> 10.2.
static bool prefer_skinny(const dg_desc* d) {
    if (d->gemm_type != DG_GEMM_NORMAL || d->k % 128 != 0 || (d->cd_dtype != DG_OUT_BF16 && d->cd_dtype != DG_OUT_F32)) return false;
    if (d->a_bits != 8 || d->b_bits != 8 || d->gran_a != 128 || d->gran_b != 128 || d->major_a_mn || d->major_b_mn) return false;
    const uint32_t sms = d->num_sms ? d->num_sms : 148;
    const double mb = static_cast<double>(d->n) * d->k * 1e-6;
    const uint32_t blocks = ceil_div(d->n, dg::kSkinnyCols);
    bool few = false;
    if (d->m <= 8) few = blocks <= 14 * sms && mb <= (2 * ceil_div(d->n, 128) >= sms ? 44.0 : 64.0) && d->k <= (blocks <= sms && 2 * blocks > sms ? 24576u : 16384u);
    else if (d->m <= 16 && blocks <= 4 * sms) few = mb <= 24.0 && d->k <= (blocks > sms ? 7168u : (blocks >= 32 ? 12288u : 10240u));
    else if (d->m <= 16) few = blocks <= 14 * sms && mb <= 24.0 && (d->k <= 512 || (d->k <= 1024 && (blocks <= 8 * sms || d->k % 512 == 0)));
    else if (d->m <= 32 && blocks <= 4 * sms) few = mb <= 8.0 && d->k <= (blocks <= 2 * sms ? 4096u : 1024u);
    else if (d->m <= 32) few = blocks <= 7 * sms && mb <= 6.3 && d->k <= 512;
    if (!few || knob_signature() == 0) return few;
    // DG_SKINNY=0 turns it off, and so does a knob that asks for something of another kernel
    for (const char* knob : {"DG_SWAP", "DG_BLOCK_N", "DG_CTAS", "DG_STAGES", "DG_SPLITS", "DG_K_SLABS"})
        if (getenv(knob)) return false;
    const char *skinny = getenv("DG_SKINNY"), *wide = getenv("DG_WIDE_TILE");
    return !(skinny && atoi(skinny) == 0) && !(wide && atoi(wide) != 0);
}
// Warps of its blocks.  Blocks of 16 columns that all fit at once share K among as many warps as there are; with more blocks it is
// several of them per SM that keep loads in flight (8 x 2112 x 7168 with 4 / 8 / 16 warps: 9.5 / 8.1 / 8.0 us; 1 x 4096 x 7168: 12.7 / 10.7 / 11.6;
// 16 x 7168 x 2048: 8.4 / 9.4 / 11.5).
static uint32_t skinny_warps(uint32_t n, uint32_t sms) {
    const uint32_t blocks = ceil_div(n, dg::kSkinnyCols);
    return blocks <= sms ? 16 : (blocks <= 2 * sms ? 8 : 4);
}
static uint32_t skinny_row_tiles(uint32_t m) { return m <= 8 ? 1 : (m <= 16 ? 2 : 4); }      // of 8 activation rows
static void skinny_config(const dg_desc* d, dg_config* out, KernelPlan* plan) {
    memset(plan, 0, sizeof(*plan));
    plan->skinny_warps = skinny_warps(d->n, d->num_sms ? d->num_sms : 148);
    plan->splits = 1;
    plan->tiles = ceil_div(d->n, dg::kSkinnyCols);
    const uint32_t row_tiles = skinny_row_tiles(d->m);
    out->swap_ab = 0;
    out->block_m = 8 * row_tiles;
    out->block_n = dg::kSkinnyCols;
    out->block_k = 128;
    out->cluster_m = out->cluster_n = 1;
    out->num_stages = row_tiles <= 2 ? 2 : 1;      // K blocks that a warp has in registers
    out->num_accum_stages = 1;
    out->smem_size = plan->smem = dg::skinny_smem_bytes(row_tiles, plan->skinny_warps);
    out->num_tiles = plan->tiles;
    out->num_splits = 1;
}
const char* dg_kernel_name(const dg_desc* d) {
    dg_config cfg;
    KernelPlan plan;
    if (search_config(d, 0, &cfg, &plan)) return nullptr;
    if (plan.skinny_warps != 0) return "dg_gemm_skinny_kernel";
    return plan.swap ? "dg_gemm_swap_kernel" : (plan.block_n2 != 0 ? "dg_gemm_wide_kernel" : "dg_gemm_kernel");
}

// How a dense problem's tiles of two halves are dealt out to the CTA pairs.
struct WideWaves {
    uint32_t whole;      // tiles computed whole, in full waves
    uint32_t units;      // those, and single halves
    uint32_t halves;     // length of the schedule in halves
};
static WideWaves wide_waves(uint32_t m, uint32_t n, uint32_t block_n, uint32_t pairs) {
    const uint32_t across = ceil_div(n, block_n), m_blocks = ceil_div(m, 256), tiles = m_blocks * (across / 2), all = m_blocks * across;
    WideWaves w;
    const uint32_t waves = all / (2 * pairs), full = waves * pairs < tiles ? waves * pairs : tiles, rest = all - 2 * full;
    // What is left over the full waves goes out as single halves, at most two per pair: whole tiles and the halves without a second one do not
    // deal out evenly.
    w.whole = full;
    w.units = full + rest;
    w.halves = 2 * waves + (all == 2 * pairs * waves ? 0 : (rest <= pairs ? 1 : 2));
    return w;
}

// Wide tiles (dg_gemm_wide.cuh) for a problem that costs `other` in the first family's other tiles; false if those are the better ones (or
// the only ones, of width `other_n`, `other_columns` of them for each CTA or pair), unless `forced`.
// Contiguous groups of 450 rows on, where the first 256 rows of each alone make 1.3 waves of tiles (3.5 where K is below 20 slabs): an arena may be sized for far
// more rows than it holds, and what the device finds is what decides.  Both tiles measured in three ways: under the power cap (bursts of 0.3-0.5 s a side,
// balanced), and single passes in turn after a 256 MB fill and after 20 ms of idling.  24 problems below 3.5 waves (k 2560-7168, n 1152-7104, 8-50 groups) take 0.96,
// 0.95 and 0.96 of the other tiles' time with a full arena, 0.98, 1.01 and 1.00 with 3 % of it live, up to 1.07, 1.08 and 1.19 (14 groups of 48 rows, 3200 x 3584: 48.7 ->
// 52.1 us); 18 above (k 2048-7168, 22-64 groups) 0.96, 0.99 and 0.99 full, 0.98, 0.99 and 0.97 with 3 %.  With fewer tiles it was up to 1.32 (8 groups of 47
// rows in 13696, 1600 x 7168: 28.5 -> 35.2 us).  K below 16 slabs loses too (23 groups of 4211 rows, 1152 x 1024, single
// passes: 1.01; of 1052: 1.14), and so do tiles that cover more columns than the others do, unless K is long: 1.03 to 1.05 times as
// many, full and 3 % live, take 0.99 and 1.02 under load, 1.03 and 1.06 after a fill at 20 slabs of K, 0.98, 0.99, 1.00 and 1.01 at 24-32 (12 problems), 0.95,
// 0.99, 0.94 and 1.01 from 40 on.
// Dense problems by cost, within lines.  Of 180 that the cost alone picks (m 200-8192, n 512-16384, k 1024-16384) the 75 inside take 0.96, 0.97 and 0.98 of
// the other tiles' time, measured in the same ways, up to 1.00, 1.01 and 1.02; the others 0.99, 1.03 and 1.03, up to 1.09, 1.16 and 1.13:
//   f32 outputs of two e2m1 operands (22 of them: 1.02, 1.06 and 1.06), whose stores take longer than the UMMAs of their K;
//   short K, by the drain of two accumulators per tile: below 32 slabs with an e4m3 operand (23: 1.00, 1.03, 1.04), 16 with two of e2m1 (22: 0.96, 1.04, 0.98);
//   an even number of halves per pair, which ends in two single halves on one accumulator (8 or 10 of them, e4m3: 1.00, 1.01, 1.02), unless there are
//     many, or two e2m1 operands have a long K;
//   more columns for a pair to work through than `other_columns` (2607 x 6624 x 10240, e4m3 x e2m1: 1.01, 1.03, 1.05).
// Halves of 160 columns were slower than both (5841 x 3720 x 11776 mxfp4: 114 -> 124 us).  Masked and batched problems, and e4m3 operands with per-32
// scales, were not measured and keep the other tiles.
static bool search_wide(const dg_desc* d, uint32_t sms, double other, uint32_t other_n, uint32_t other_columns, bool forced, dg_config* out, KernelPlan* plan) {
    if (d->cd_dtype != DG_OUT_BF16 && d->cd_dtype != DG_OUT_F32) return false;
    if (d->major_a_mn || d->major_b_mn || sms < 2 || d->gemm_type == DG_GEMM_BATCHED) return false;
    if (!forced && (d->gemm_type == DG_GEMM_M_GROUPED_MASKED || (d->a_bits == 8 && d->gran_a != 128) || (d->b_bits == 8 && d->gran_b != 128))) return false;
    const uint32_t block_k = d->a_bits == 4 && d->b_bits == 4 ? 256 : 128, groups = d->num_groups ? d->num_groups : 1, pairs = sms / 2;
    const uint32_t sfa_words = 4 * d->gran_a >= block_k ? 1 : block_k / (4 * d->gran_a), sfb_words = 4 * d->gran_b >= block_k ? 1 : block_k / (4 * d->gran_b);
    const uint32_t total_kb = ceil_div(d->k, block_k);
    const bool dense = d->gemm_type == DG_GEMM_NORMAL;
    bool found = false, chosen = false;
    double best = 0;
    for (uint32_t most = 224; most >= 192; most -= 32) {
        uint32_t bn = most, bn2 = most, tiles;
        double halves;
        if (dense) {
            const WideWaves w = wide_waves(d->m, d->n, bn, pairs);
            tiles = w.units;
            halves = w.halves;
        } else {
            // a group's columns in tiles of about equal width
            if (most != 224) break;
            const uint32_t across = ceil_div(d->n, 2 * most), width = ceil_div(ceil_div(d->n, across), 32) * 32;
            bn = ceil_div(width / 2, 32) * 32;
            bn2 = width - bn;
            if (bn2 == 0) break;
            tiles = static_cast<uint32_t>(groups * (group_rows(d) / 256 + 0.5) * across + 0.999);
            halves = 2.0 * ceil_div(tiles, pairs);
        }
        if (bn + bn2 + 4 * sfa_words + 8 * ceil_div(bn, 128) * sfb_words > 512) continue;
        uint32_t epi_bufs = 2, stages = 4;
        auto smem = [&]() { return dg::gemm_wide_smem_bytes(bn, d->cd_dtype, stages, sfa_words, sfb_words, epi_bufs); };
        if (smem() > kSmemCapacity) epi_bufs = 1;
        while (stages < dg::kMaxStages && smem() <= kSmemCapacity) ++stages;
        while (stages > 3 && smem() > kSmemCapacity) --stages;
        if (smem() > kSmemCapacity) continue;
        const double cost = halves * (total_kb * (2.0 * bn + 130.0) + 1500.0 + (d->cd_dtype == DG_OUT_F32 ? 1000.0 : 0.0)) + 8000.0;
        const uint32_t across = ceil_div(d->n, bn + bn2);
        const bool wider = across * (bn + bn2) > (total_kb >= 40 ? 1.06 : (total_kb >= 24 ? 1.04 : 1.02)) * (ceil_div(d->n, other_n) * other_n);
        const bool odd = static_cast<uint32_t>(halves) % 2 != 0;
        bool inside;
        if (!dense) inside = (total_kb >= 20 ? 10 * groups * across >= 13 * pairs : total_kb >= 16 && 2 * groups * across >= 7 * pairs) && group_rows(d) >= 450.0 && !wider;
        else if (block_k == 256) inside = d->cd_dtype == DG_OUT_BF16 && total_kb >= 16 && (odd || (total_kb >= 24 && halves >= 8));
        else inside = total_kb >= 32 && (halves >= 11 || (odd && total_kb >= 48));
        if (found && cost >= best) continue;
        found = true;
        best = cost;
        chosen = forced || (inside && !(dense && (halves < 5 || cost >= other || halves * bn > 1.05 * other_columns)));
        plan->swap = false;
        plan->ctas = 2; plan->umma_n = bn; plan->block_n2 = bn2; plan->halves = 1; plan->stages = stages; plan->accum = 1;
        plan->splits = 1; plan->tiles = tiles; plan->epi_bufs = epi_bufs; plan->table_groups = plan->skinny_warps = 0;
        plan->smem = smem();
        out->swap_ab = 0;
        out->block_m = 256;
        out->block_n = bn;            // of each of the tile's two accumulators
        out->block_k = block_k;
        out->cluster_m = 2;
        out->cluster_n = 1;
        out->num_stages = stages;
        out->num_accum_stages = 2;
        out->smem_size = plan->smem;
        out->num_tiles = tiles;
        out->num_splits = 1;
    }
    return chosen;
}

// Tile choice of the swapped family; false if nothing fits (or the DG_* knobs leave nothing).
static bool search_swapped(const dg_desc* d, uint32_t sms, dg_config* out, KernelPlan* plan) {
    const char *force_n = getenv("DG_BLOCK_N"), *force_ctas = getenv("DG_CTAS"), *force_stages = getenv("DG_STAGES");
    const char *force_splits = getenv("DG_SPLITS"), *force_halves = getenv("DG_K_SLABS");
    const bool mxf4 = d->a_bits == 4 && d->b_bits == 4;
    const uint32_t half_k = mxf4 ? 256 : 128, groups = d->num_groups ? d->num_groups : 1;
    const bool dense = d->gemm_type == DG_GEMM_NORMAL || d->gemm_type == DG_GEMM_BATCHED;
    double best_cost = 0;
    bool found = false;
    for (uint32_t halves = 1; halves <= 2; ++halves) {
        if (force_halves && static_cast<uint32_t>(atoi(force_halves)) != halves) continue;
        const uint32_t block_k = half_k * halves;
        // kernel operand A is the caller's b (weights), kernel operand B the caller's a (activation rows)
        const uint32_t sfa_words = 4 * d->gran_b >= block_k ? 1 : block_k / (4 * d->gran_b);
        const uint32_t sfb_words = 4 * d->gran_a >= block_k ? 1 : block_k / (4 * d->gran_a);
        const uint32_t total_kb = ceil_div(d->k, block_k);
        for (uint32_t ctas = 1; ctas <= 2; ++ctas) {
            if (force_ctas && static_cast<uint32_t>(atoi(force_ctas)) != ctas) continue;
            if (ctas == 2 && sms < 2) continue;
            // the dense problems the rule above picks: one CTA per weight block, two slabs, no K ranges (those, pairs and one slab only
            // where DG_SWAP=1 pins the family: in the dense problems it was measured on, the first family's K ranges are the faster ones)
            const bool picked = d->gemm_type == DG_GEMM_NORMAL && !getenv("DG_SWAP");
            if (picked && ((halves == 1 && !force_halves) || (ctas == 2 && !force_ctas))) continue;
            // grouped layouts: pairs and one slab per stage measured best at every size (MoE layer of 256 experts: 3.88 ms against 4.28
            // with two slabs; single CTAs 5-15 % slower)
            if (d->gemm_type != DG_GEMM_NORMAL && d->gemm_type != DG_GEMM_BATCHED && ((halves == 2 && !force_halves) || (ctas == 1 && !force_ctas && sms >= 2))) continue;
            const uint32_t step = dense ? 16 * ctas : 32, workers = sms / ctas;
            const double rows = group_rows(d);
            // tile height: everything a dense problem has up to 256 rows; where groups vary, twice what is expected and at least 64, in the
            // contiguous layout 288 rather than 256 for groups around that size, half of which are a little above.
            // A masked problem's expected rows are a hint about the mean only, and a hot group's weights pass through an SM once per tile:
            // with a hint of 1, tiles of 64 rows took up to 2.0 times as long as the first family (15 groups of up to 336 rows,
            // 3712 x 3072: 59 -> 99 us).  So at least 128 rows, and a quarter of the slot.  128 rows cost nothing where the hint is right
            // (1-16 rows, 30 problems: 0.99 of the time on average; 256 rows took 3 % more in a decode step of 62 experts x 2 rows).
            uint32_t bn;
            if (dense) bn = d->m <= 256 ? ceil_div(d->m, step) * step : 256;
            else bn = ceil_div(static_cast<uint32_t>(2 * rows) + 1, 32) * 32;
            if (!dense && bn < 64) bn = 64;
            if (d->gemm_type == DG_GEMM_M_GROUPED_MASKED) {
                const uint32_t least = d->m / 4 > 128 ? ceil_div(d->m / 4, 32) * 32 : 128, slot = ceil_div(d->m, 32) * 32;
                if (bn < least) bn = least;
                if (bn > slot) bn = slot;
            }
            if (bn > 256) bn = d->gemm_type == DG_GEMM_M_GROUPED_CONTIGUOUS && halves == 1 ? 288 : 256;
            if (force_n) bn = static_cast<uint32_t>(atoi(force_n));
            if (bn == 0 || bn > dg::kSwapMaxRows || (bn > 256 && bn % 32 != 0) || (bn > 256 && dense) || bn % step != 0) continue;
            const uint32_t sf_cols = 4 * sfa_words + ceil_div(bn, 128) * 4 * sfb_words;
            if (bn + sf_cols > 512) continue;
            const uint32_t m_blocks = ceil_div(d->n, 128 * ctas);
            const uint32_t most_rows = bn < 32 ? bn : bn / 32 * 32;         // of a tile that has a neighbour
            const double row_tiles = rows <= bn ? 1.0 : (dense ? static_cast<double>(ceil_div(d->m, most_rows)) : rows / most_rows + 0.5);
            const double tile_rows = rows / row_tiles;
            const uint32_t tiles = static_cast<uint32_t>(groups * row_tiles * m_blocks + 0.999);
            const uint32_t most_splits = d->gemm_type == DG_GEMM_NORMAL && !picked ? 16 : 1;
            for (uint32_t splits = 1; splits <= most_splits; ++splits) {
                if (force_splits && static_cast<uint32_t>(atoi(force_splits)) != splits) continue;
                if (splits > 1 && total_kb < 2 * splits) continue;       // at least two k-blocks per range
                if (splits > 1 && !force_splits && static_cast<uint64_t>(tiles) * splits > workers) continue;
                uint32_t stages = force_stages ? static_cast<uint32_t>(atoi(force_stages)) : dg::kMaxStages;
                if (stages > dg::kMaxStages) stages = dg::kMaxStages;
                auto smem = [&](uint32_t st) { return dg::gemm_swap_smem_bytes(bn, ctas, d->cd_dtype, st, sfa_words, sfb_words, halves); };
                while (stages > 1 && smem(stages) > kSmemCapacity) --stages;
                if (smem(stages) > kSmemCapacity || (stages < 2 && !force_stages)) continue;
                const double mma = 4.0 * (tile_rows > 66.0 ? tile_rows * 0.5 : 33.0);
                const double feed = (16384.0 + tile_rows / ctas * 128.0) / 70.0;
                const double per_kb = (halves * (mma > feed ? mma : feed) + 150.0) * (stages < 3 ? 1.5 : 1.0);   // two stages do not cover a load's latency
                const double kb_per = static_cast<double>(total_kb) / splits;
                const double waves = splits > 1 || dense ? ceil_div(tiles * splits, workers) : static_cast<double>(tiles) / workers;
                // decides only where DG_SWAP=1 pins the family for a dense or batched problem, between pairs, slabs and K ranges: by its
                // rule every problem has one candidate here
                const double cost = waves * (kb_per * per_kb + 800.0) + (splits > 1 ? 2500.0 + splits * tile_rows * 8.0 : 0.0);
                if (!found || cost < best_cost * (1.0 - 1e-9)) {
                    found = true;
                    best_cost = cost;
                    plan->swap = true;
                    plan->ctas = ctas; plan->umma_n = bn; plan->halves = halves; plan->stages = stages; plan->accum = 2;
                    plan->splits = splits; plan->tiles = tiles; plan->smem = smem(stages);
                    // the group table takes what the stages leave of the shared memory
                    const uint32_t room = !dense && dg::swap_has_table(ctas, halves) ? (kSmemCapacity - plan->smem) / 16 : 0;
                    plan->table_groups = groups < room ? groups : room;
                    plan->block_n2 = plan->skinny_warps = 0;
                    plan->smem += plan->table_groups * 16;
                    out->swap_ab = 1;
                    out->block_m = bn;            // activation rows per tile (an upper bound: a tile's UMMA N follows its rows)
                    out->block_n = 128 * ctas;    // weight rows per tile
                    out->block_k = block_k;
                    out->cluster_m = 1;
                    out->cluster_n = ctas;
                    out->num_stages = stages;
                    out->num_accum_stages = 2;
                    out->smem_size = plan->smem;
                    out->num_tiles = tiles;
                    out->num_splits = splits;
                }
            }
        }
    }
    return found;
}

static int search_config(const dg_desc* d, uint32_t limits, dg_config* out, KernelPlan* plan) {
    if (d == nullptr || out == nullptr) return fail(DG_ERR_SHAPE, "null argument");
    if ((d->a_bits != 8 && d->a_bits != 4) || (d->b_bits != 8 && d->b_bits != 4)) return fail(DG_ERR_SHAPE, "operand bits must be 8 or 4");
    if ((d->major_a_mn && d->a_bits == 4) || (d->major_b_mn && d->b_bits == 4)) return fail(DG_ERR_SHAPE, "FP4 operands must be K-major");
    if (!(limits & kNoSkinny) && prefer_skinny(d)) {
        skinny_config(d, out, plan);
        return DG_OK;
    }
    // two packed e2m1 operands run on kind::mxf4 (256 elements per 128-byte slab); an e4m3 x e2m1 pair runs on
    // kind::mxf8f6f4 with the e2m1 side expanded to one code per byte by the TMA load (128 elements per slab)
    const bool mxf4 = d->a_bits == 4 && d->b_bits == 4;
    const uint32_t half_k = mxf4 ? 256 : 128;     // K elements of one 128-byte slab
    const uint32_t sms = d->num_sms ? d->num_sms : 148;
    const uint32_t groups = d->num_groups ? d->num_groups : 1;
    // the fused gate/up activation writes block_n / 2 columns per tile in 32-column scale blocks: widths of 64
    const bool swiglu = d->cd_dtype == DG_OUT_SWIGLU_FP8;
    const uint32_t step = d->cd_dtype == DG_OUT_FP8 ? 128 : (swiglu ? 64 : 32);
    const uint32_t align = g_mk_alignment.load();
    const char* force_n = getenv("DG_BLOCK_N");
    const char* force_ctas = getenv("DG_CTAS");
    const char* force_stages = getenv("DG_STAGES");

    const char* force_splits = getenv("DG_SPLITS");
    const char* force_halves = getenv("DG_K_SLABS");
    const bool pinned = force_n || force_ctas || force_stages || force_splits || force_halves;
    uint32_t best_n = 0, best_accum = 0, best_tiles = 0, best_ctas = 0, best_stages = 0, best_splits = 1, best_halves = 1, best_epi_bufs = 2;
    double best_cost = 0;
    // a stage holds one or two 128-byte K slabs per operand; two slabs halve the per-stage bookkeeping per UMMA
    for (uint32_t halves = 1; halves <= 2; ++halves) {
    if (force_halves && static_cast<uint32_t>(atoi(force_halves)) != halves) continue;
    const uint32_t block_k = half_k * halves;
    const uint32_t sfa_words = 4 * d->gran_a >= block_k ? 1 : block_k / (4 * d->gran_a);
    const uint32_t sfb_words = 4 * d->gran_b >= block_k ? 1 : block_k / (4 * d->gran_b);
    for (uint32_t ctas = 1; ctas <= 2; ++ctas) {
        if (force_ctas && static_cast<uint32_t>(atoi(force_ctas)) != ctas) continue;
        const uint32_t tile_m = 128 * ctas;
        // contiguous layout: a tile may run past its group's end into the next groups' rows; those rows are computed but
        // never stored (stores are 32 rows tall and stop at the group end; an alignment of 16 switches the last box of a
        // group to row-exact stores), so every alignment from 16 to 256 works with 128- and 256-row tiles
        if (ctas == 2 && sms < 2) continue;
        if (swiglu && ctas != 2) continue;        // gate rows on one CTA of the pair, up rows on the other
        // expected row-tiles.  Grouped layouts: a group of r valid rows needs ceil(r / tile_m) tiles, on average
        // r / tile_m + 1/2 when group sizes are spread out; the contiguous arena's m includes about half an alignment of
        // padding per group.
        double m_blocks;
        if (d->gemm_type == DG_GEMM_M_GROUPED_CONTIGUOUS) {
            const double per_group = groups ? static_cast<double>(d->m) / groups : d->m;
            const double valid = per_group > align / 2.0 ? per_group - align / 2.0 : per_group;
            m_blocks = groups > 1 ? groups * (valid / tile_m + 0.5) : ceil_div(d->m, tile_m);
        } else if (d->gemm_type == DG_GEMM_M_GROUPED_MASKED) {
            const double e = d->expected_m ? d->expected_m : d->m;
            m_blocks = groups * (e / tile_m + 0.5);
        } else {
            m_blocks = groups * ceil_div(d->m, tile_m);
        }
        const uint32_t workers = sms / ctas;
        for (uint32_t bn = step; bn <= 256; bn += step) {
            if (bn % (16 * ctas) != 0) continue;
            if (d->major_b_mn && (bn / ctas) % 128 != 0) continue;    // an MN-major B tile is made of whole 128-row boxes per CTA
            if (force_n && static_cast<uint32_t>(atoi(force_n)) != bn) continue;
            const uint32_t sf_cols = 4 * sfa_words + ceil_div(bn, 128) * 4 * sfb_words;
            if (bn + sf_cols > 512) continue;
            const uint32_t accum = 2 * bn + sf_cols <= 512 ? 2 : 1;
            if (swiglu && accum == 1 && !force_n) continue;   // its epilogue is long: only worth it behind a second accumulator
            const uint32_t tiles = static_cast<uint32_t>(m_blocks * ceil_div(d->n, bn) + 0.999);
            // cycles per tile, fitted to measurements on B200 (dense 4096x7168x4096, every width, 1 and 2 CTAs):
            // per k-block max(UMMA time, load time) + ~150 of issue-side overhead, where one UMMA (K = 32 bytes) takes
            // max(~118, bn / 2) cycles and a CTA receives its A tile (16 KB) plus bn/ctas rows of B at ~77 bytes per cycle;
            // a single-buffered accumulator exposes the whole epilogue (~10.5 cycles per column).
            const uint32_t total_kb = ceil_div(d->k, block_k);
            // Dense problems have constants of their own.  For one wave they were fitted to 205 problems (m 1-4096, n 512-16384, k 1024-16384,
            // e4m3 / mixed / mxfp4, every width, K ranges; the choice is 2 % off the best of these tiles on average, 4 % with the others): a
            // scale copy costs 40 cycles, a tile 2900 from its first load to its last store, of which the last one's epilogue is exposed.
            // (Fitted when the copies were loops and f32 outputs of a single tile were staged in two buffers; both are cheaper since.)
            // What was not in that fit keeps the constants and the choices it had before it, which measured better there: batched problems
            // (60 of them, 1.01 times as long on average with the fitted constants, 1.22 at worst: 10 x 420 x 1792 x 512, f32), and
            // e4m3 operands with per-32 scales (30 problems, 1.02 and 1.28: 972 x 8704 x 1024, f32).
            const bool fitted = d->gemm_type == DG_GEMM_NORMAL && !swiglu && (d->a_bits == 4 || d->gran_a == 128) && (d->b_bits == 4 || d->gran_b == 128);
            const double least_mma = fitted ? 103.0 : 118.0;
            const double mma = 4.0 * (bn * 0.5 > least_mma ? bn * 0.5 : least_mma);
            const double feed = (16384.0 + bn / ctas * 128.0) / 77.0;
            const double epilogue = swiglu ? (accum == 1 ? 40.0 * bn : 1.0 * bn) : (accum == 1 ? (fitted ? 9.7 : 10.5) * bn : (fitted ? 5.2 * bn : 1.0 * bn));
            const double copies = (4 * d->gran_a > block_k ? static_cast<double>(block_k) / (4 * d->gran_a) : sfa_words) +
                                  (4 * d->gran_b > block_k ? static_cast<double>(block_k) / (4 * d->gran_b) : sfb_words) * ceil_div(bn, 128);
            const double per_kb = halves * (mma > feed ? mma : feed) + (fitted ? 234.0 + 40.0 * copies : 150.0);
            // K ranges (dense GEMMs with f32-summable outputs only): each range is a multiple of 4 k-blocks so scale words
            // never straddle ranges; the partial sums cost a second small kernel (launch + S reads of the M x N f32 tile set)
            const bool may_split = d->gemm_type == DG_GEMM_NORMAL && d->cd_dtype != DG_OUT_FP8 && !swiglu && d->n % 4 == 0 && !(limits & kNoKRanges);
            for (uint32_t splits = 1; splits <= 16; ++splits) {
                if (splits > 1 && (!may_split || (halves > 1 && !fitted))) break;
                if (force_splits && static_cast<uint32_t>(atoi(force_splits)) != splits) continue;
                const uint32_t unit = 4 / halves;      // a range is whole scale words: four slabs
                uint32_t kb_per = ceil_div(ceil_div(total_kb, splits), unit) * unit;
                if (splits > 1 && (kb_per < 2 * unit || kb_per * (splits - 1) >= total_kb)) continue;   // every range non-empty, at least 8 k-blocks
                if (splits == 1) kb_per = total_kb;
                // K ranges store f32 partials whatever the caller's output type: size the staging buffers for that
                const uint32_t kernel_out = splits > 1 ? static_cast<uint32_t>(DG_OUT_F32) : d->cd_dtype;
                uint32_t stages = force_stages ? static_cast<uint32_t>(atoi(force_stages)) : dg::kMaxStages;
                if (stages > dg::kMaxStages) stages = dg::kMaxStages;
                // f32 staging takes 32 KB; with half of it three stages of two slabs fit 256-column tiles
                const uint32_t most_stages = stages;
                uint32_t epi_bufs = 2;
                auto smem = [&]() { return dg::gemm_smem_bytes(bn, ctas, kernel_out, stages, sfa_words, sfb_words, halves, epi_bufs); };
                while (stages > 1 && smem() > kSmemCapacity) --stages;
                if (fitted && stages < 3 && most_stages >= 3 && kernel_out == DG_OUT_F32) {
                    stages = most_stages;
                    epi_bufs = 1;
                    while (stages > 1 && smem() > kSmemCapacity) --stages;
                }
                if (stages < 1 || smem() > kSmemCapacity) continue;
                if (stages < 3 && !force_stages) continue;
                const uint32_t waves = ceil_div(tiles * splits, workers);
                const double tile_cost = kb_per * per_kb + (splits > 1 ? (fitted ? 3.6 : 2.0) * bn : epilogue) + (fitted ? 2855.0 : 600.0);
                const double plane_bytes = static_cast<double>(splits) * d->m * d->n * 4.0;
                const double reduce = (splits > 1 ? (fitted ? 4450.0 + plane_bytes / 1507.0 : 9000.0 + plane_bytes / 3000.0) : 0.0) +
                                      (fitted ? 4.5 * bn + (ctas == 2 ? 280.0 : 0.0) : 0.0);
                // every CTA pulls its A slab (16 KB) and its share of B from L2 for each 128 bytes of K; with many small groups
                // (weights read once, little reuse) that aggregate stream, ~9000 bytes per cycle on this part (11000 with the reuse of
                // dense problems), is the limit
                const double l2_bytes = static_cast<double>(tiles) * ctas * ceil_div(d->k, half_k) * (16384.0 + bn / ctas * 128.0);
                const double l2_floor = l2_bytes / (fitted ? 11140.0 : 9000.0);
                double compute = waves * tile_cost;
                if (fitted && splits == 1 && waves > 1) {
                    // A further wave starts while the one before it is stored: with two accumulators only the longer of main loop and stores
                    // counts, with one the epilogue comes on top; f32 tiles store twice the bytes.  Over 152 problems of several waves
                    // (m 512-8192, n 1536-24576, k 512-8192, bf16 and f32 outputs, 20 tiles each) the choice is 1.1 % off the best of them,
                    // 3.8 % with the first wave's cost for every wave, which took 256-column tiles and their exposed epilogues where narrower
                    // ones are faster: 2894 x 6144 x 1024 20.0 -> 26.7 us, 7467 x 3448 x 2560 with f32 output 63.6 -> 80.2.
                    const double loop = kb_per * per_kb, store = kernel_out == DG_OUT_F32 ? 2.0 * bn : 1.0 * bn;
                    const double hidden = loop + bn > 10.0 * store ? loop + bn : 10.0 * store;
                    compute = tile_cost + (waves - 1.0) * ((accum == 1 ? loop + 12.0 * store : hidden) + 1000.0);
                }
                const double cost = (compute > l2_floor ? compute : l2_floor) + reduce;
                if (best_n == 0 || cost < best_cost * (1.0 - 1e-9)) {
                    best_n = bn; best_cost = cost; best_accum = accum; best_tiles = tiles; best_ctas = ctas; best_stages = stages;
                    best_splits = splits; best_halves = halves; best_epi_bufs = epi_bufs;
                }
            }
        }
    }
    }
    // ---- the swapped family: weight rows on UMMA M, activation rows on UMMA N
    {
        const char* force_swap = getenv("DG_SWAP");
        const bool forced = force_swap && atoi(force_swap) != 0, forbidden = force_swap && atoi(force_swap) == 0;
        const bool applies = !swiglu && !d->major_a_mn && !d->major_b_mn;
        if (applies && !forbidden && (forced || prefer_swapped(d))) {
            if (search_swapped(d, sms, out, plan)) return DG_OK;
            if (forced) return fail(DG_ERR_SHAPE, "no tile configuration of the swapped family fits (DG_BLOCK_N=%s DG_CTAS=%s)", force_n ? force_n : "",
                                    force_ctas ? force_ctas : "");
        }
    }
    if (best_n == 0) return fail(DG_ERR_SHAPE, "no tile configuration fits (DG_BLOCK_N=%s DG_CTAS=%s)", force_n ? force_n : "", force_ctas ? force_ctas : "");
    {
        const char* wide = getenv("DG_WIDE_TILE");       // 0: never, 1: wherever they apply
        const bool forced = wide && atoi(wide) != 0, forbidden = (wide && atoi(wide) == 0) || (limits & kNoWideTiles) || pinned;
        if (!forbidden && search_wide(d, sms, best_cost, best_n, ceil_div(best_tiles, sms / best_ctas) * best_n, forced, out, plan)) return DG_OK;
    }
    const uint32_t stages = best_stages;
    plan->block_n2 = plan->skinny_warps = 0;
    plan->swap = false;
    plan->ctas = best_ctas; plan->umma_n = best_n; plan->halves = best_halves; plan->stages = best_stages; plan->accum = best_accum;
    plan->splits = best_splits; plan->tiles = best_tiles; plan->table_groups = 0;
    out->swap_ab = 0;
    out->block_m = 128 * best_ctas;
    out->block_n = best_n;
    const uint32_t block_k = half_k * best_halves;
    const uint32_t sfa_words = 4 * d->gran_a >= block_k ? 1 : block_k / (4 * d->gran_a);
    const uint32_t sfb_words = 4 * d->gran_b >= block_k ? 1 : block_k / (4 * d->gran_b);
    out->block_k = block_k;
    out->cluster_m = best_ctas;
    out->cluster_n = 1;
    out->num_stages = stages;
    out->num_accum_stages = best_accum;
    out->smem_size = dg::gemm_smem_bytes(best_n, best_ctas, best_splits > 1 ? static_cast<uint32_t>(DG_OUT_F32) : d->cd_dtype, stages, sfa_words,
                                         sfb_words, best_halves, best_epi_bufs);
    plan->epi_bufs = best_epi_bufs;
    out->num_tiles = best_tiles;
    out->num_splits = best_splits;
    plan->smem = out->smem_size;
    return DG_OK;
}

}  // extern "C"

namespace {

// ----------------------------------------------------------------------- tensor maps
int encode_map(CUtensorMap* map, CUtensorMapDataType dtype, uint32_t rank, const void* base, const uint64_t* dims,
               const uint64_t* strides_bytes, const uint32_t* box, CUtensorMapSwizzle swizzle, const char* what) {
    cuuint64_t gdim[4], gstride[3];
    cuuint32_t gbox[4], estride[4] = {1, 1, 1, 1};
    for (uint32_t i = 0; i < rank; ++i) { gdim[i] = dims[i]; gbox[i] = box[i]; }
    for (uint32_t i = 0; i + 1 < rank; ++i) gstride[i] = strides_bytes[i];
    if (reinterpret_cast<uintptr_t>(base) % 16 != 0) return fail(DG_ERR_SHAPE, "%s: base address must be 16-byte aligned", what);
    for (uint32_t i = 0; i + 1 < rank; ++i)
        if (gstride[i] % 16 != 0) return fail(DG_ERR_SHAPE, "%s: stride %llu bytes is not a multiple of 16", what, (unsigned long long)gstride[i]);
    CUresult r = encode_tiled_fn()(map, dtype, rank, const_cast<void*>(base), gdim, gstride, gbox, estride, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(DG_ERR_DRIVER, "cuTensorMapEncodeTiled(%s) failed with %d", what, static_cast<int>(r));
    return DG_OK;
}

int check_operand(const dg_lp_operand* op, const char* name, uint32_t total_rows, uint32_t groups) {
    if (op == nullptr || op->data == nullptr || op->sf == nullptr) return fail(DG_ERR_SHAPE, "%s: null operand", name);
    if (op->bits != 8 && op->bits != 4) return fail(DG_ERR_SHAPE, "invalid bits %u", op->bits);
    if (op->gran_k != 32 && op->gran_k != 128) return fail(DG_ERR_SHAPE, "invalid gran_k %u", op->gran_k);
    if (op->major_mn && op->bits == 4) return fail(DG_ERR_SHAPE, "%s: FP4 operands must be K-major", name);
    if (op->bits == 4 && (op->k % 128 != 0 || op->ld % 128 != 0)) return fail(DG_ERR_SHAPE, "FP4 k and ld must be multiples of 128");
    if (op->bits == 4 && op->gran_k != 32) return fail(DG_ERR_UNSUPPORTED, "FP4 operands need gran_k = 32");
    if (op->k == 0 || op->k % op->gran_k != 0) return fail(DG_ERR_SHAPE, "k (%u) must be a multiple of the SF granularity (%u)", op->k, op->gran_k);
    if (op->major_mn) {
        // (groups, k, ld) bytes: the rows of a group are contiguous, ld is the pitch between two k
        const uint32_t g = groups ? groups : 1;
        if (op->ld < total_rows / g) return fail(DG_ERR_SHAPE, "%s: MN-major ld (%u) smaller than the rows of a group (%u)", name, op->ld, total_rows / g);
        if (op->ld % 16 != 0) return fail(DG_ERR_SHAPE, "%s: MN-major pitch %u bytes must be a multiple of 16", name, op->ld);
        const size_t need = static_cast<size_t>(g) * op->k * op->ld;
        if (op->data_len < need) return fail(DG_ERR_SHAPE, "data buffer too small: %zu < %zu", op->data_len, need);
        const size_t sf_words = dg_sf_words(total_rows, op->k, op->gran_k, groups);
        if (op->sf_len < sf_words) return fail(DG_ERR_SHAPE, "sf buffer too small: %zu < %zu", op->sf_len, sf_words);
        return DG_OK;
    }
    if (op->ld < op->k) return fail(DG_ERR_SHAPE, "%s: ld (%u) smaller than k (%u)", name, op->ld, op->k);
    const uint32_t row_bytes = op->bits == 4 ? op->ld / 2 : op->ld;
    if (row_bytes % 16 != 0) return fail(DG_ERR_SHAPE, "%s: row pitch %u bytes must be a multiple of 16", name, row_bytes);
    const size_t storage = static_cast<size_t>(total_rows) * row_bytes;
    if (op->data_len < storage) return fail(DG_ERR_SHAPE, "data buffer too small: %zu < %zu", op->data_len, storage);
    const size_t sf_need = dg_sf_words(total_rows, op->k, op->gran_k, groups);
    if (op->sf_len < sf_need) return fail(DG_ERR_SHAPE, "sf buffer too small: %zu < %zu", op->sf_len, sf_need);
    return DG_OK;
}

struct Problem {
    uint32_t type;
    uint32_t m;            // rows per group (contiguous: whole arena)
    uint32_t n, k, groups;
    uint32_t expected_m;
    const uint32_t* layout;
    bool bf16 = false;     // operands are bf16 rows described as 2k bytes each; no scale factors (dg_bf16_gemm)
};

// DG_PDL=0 launches every kernel fully serialised (for comparisons and debugging).
bool pdl_enabled() {
    static const bool on = [] { const char* v = getenv("DG_PDL"); return !(v && strcmp(v, "0") == 0); }();
    return on;
}

bool print_configs() {
    static const bool on = [] { const char* v = getenv("DG_PRINT_CONFIGS"); return v && strcmp(v, "0") != 0; }();
    return on;
}

// Launches a kernel that calls griddep_wait() itself before its first access to global memory, so that its start-up overlaps the
// end of the kernel before it in the stream.  (Also the cheaper launch for the host: 2.0 us against 2.4 us measured for the
// fully serialised form.)  Grids of more than 4096 blocks are launched serialised: early blocks move in beside a persistent
// GEMM, whose SMs are then stuck with its shared-memory carve-out (a small L1) until the grid is through; on an MoE layer of
// 8192 tokens that cost the activation and combine kernels more (40 us of 4.9 ms) than the ~2 us of overlap bring.
// Returns the launch's own result: cudaGetLastError would also hand out what an earlier call that failed had left behind.
template <typename... Params, typename... Args>
cudaError_t launch(void (*kernel)(Params...), dim3 grid, uint32_t threads, size_t smem, cudaStream_t stream, Args... args) {
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() && static_cast<uint64_t>(grid.x) * grid.y * grid.z <= 4096 ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

// The opt-in to the full shared-memory carve-out is per kernel instantiation and per device; the first
// call also makes the runtime load that kernel's image.
// kSlabs: 0 the first tile family, kWideTiles its wide tiles, else the swapped family with that many K slabs per stage.
constexpr uint32_t kWideTiles = 3;
template <uint32_t kFmt, uint32_t kOut, uint32_t kCtas, uint32_t kSlabs>
constexpr auto gemm_kernel() {
    if constexpr (kSlabs == kWideTiles) return &dg::dg_gemm_wide_kernel<kFmt, kOut>;
    else if constexpr (kSlabs != 0) return &dg::dg_gemm_swap_kernel<kFmt, kOut, kCtas, kSlabs>;
    else return &dg::dg_gemm_kernel<kFmt, kOut, kCtas>;
}
template <uint32_t kFmt, uint32_t kOut, uint32_t kCtas, uint32_t kSlabs = 0>
cudaError_t configure_kernel() {
    static std::atomic<uint64_t> configured{0};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 64 && (configured.load() & (1ull << dev))) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(gemm_kernel<kFmt, kOut, kCtas, kSlabs>(), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(kSmemCapacity));
    if (e == cudaSuccess && dev < 64) configured.fetch_or(1ull << dev);
    return e;
}

template <uint32_t kFmt, uint32_t kOut, uint32_t kCtas, uint32_t kSlabs = 0>
cudaError_t launch_kernel(const dg::GemmParams& p, uint32_t grid, uint32_t smem, cudaStream_t stream, const CUtensorMap* maps) {
    auto kernel = gemm_kernel<kFmt, kOut, kCtas, kSlabs>();
    cudaError_t e = configure_kernel<kFmt, kOut, kCtas, kSlabs>();
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(grid, 1, 1);
    cfg.blockDim = dim3(kSlabs == kWideTiles ? dg::kWideThreads : (kSlabs != 0 ? dg::kSwapThreads : dg::kNumThreads), 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kCtas;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    // the kernel waits for its predecessor itself (griddep_wait) after its set-up: let the two overlap
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
    if constexpr (kSlabs != 0 && kSlabs != kWideTiles) return cudaLaunchKernelEx(&cfg, kernel, p, maps[0], maps[1], maps[2], maps[3], maps[5], maps[6]);
    else return cudaLaunchKernelEx(&cfg, kernel, p, maps[0], maps[1], maps[2], maps[3], maps[4]);
}

template <uint32_t kFmt, uint32_t kCtas, uint32_t kSlabs>
cudaError_t launch_swapped_by_out(int kind, const dg::GemmParams& p, uint32_t grid, uint32_t smem, cudaStream_t stream, const CUtensorMap* maps) {
    if (kind == DG_OUT_BF16) return launch_kernel<kFmt, dg::kOutBf16, kCtas, kSlabs>(p, grid, smem, stream, maps);
    if (kind == DG_OUT_F32) return launch_kernel<kFmt, dg::kOutF32, kCtas, kSlabs>(p, grid, smem, stream, maps);
    if constexpr (kFmt != dg::kFmtBf16)
        if (kind == DG_OUT_FP8) return launch_kernel<kFmt, dg::kOutFp8, kCtas, kSlabs>(p, grid, smem, stream, maps);
    return cudaErrorInvalidValue;
}
template <uint32_t kFmt>
cudaError_t launch_swapped(const KernelPlan& plan, int kind, const dg::GemmParams& p, uint32_t grid, cudaStream_t stream, const CUtensorMap* maps) {
    if (plan.ctas == 2)
        return plan.halves == 2 ? launch_swapped_by_out<kFmt, 2, 2>(kind, p, grid, plan.smem, stream, maps)
                                : launch_swapped_by_out<kFmt, 2, 1>(kind, p, grid, plan.smem, stream, maps);
    return plan.halves == 2 ? launch_swapped_by_out<kFmt, 1, 2>(kind, p, grid, plan.smem, stream, maps)
                            : launch_swapped_by_out<kFmt, 1, 1>(kind, p, grid, plan.smem, stream, maps);
}

template <uint32_t kFmt, uint32_t kCtas>
cudaError_t launch_by_out(int kind, const dg::GemmParams& p, uint32_t grid, uint32_t smem, cudaStream_t stream, const CUtensorMap* maps) {
    if (kind == DG_OUT_BF16) return launch_kernel<kFmt, dg::kOutBf16, kCtas>(p, grid, smem, stream, maps);
    if (kind == DG_OUT_F32) return launch_kernel<kFmt, dg::kOutF32, kCtas>(p, grid, smem, stream, maps);
    if constexpr (kFmt == dg::kFmtMxf8f6f4 && kCtas == 2)
        if (kind == DG_OUT_SWIGLU_FP8) return launch_kernel<kFmt, dg::kOutSwiGluFp8, kCtas>(p, grid, smem, stream, maps);
    if constexpr (kFmt != dg::kFmtBf16)
        if (kind == DG_OUT_FP8) return launch_kernel<kFmt, dg::kOutFp8, kCtas>(p, grid, smem, stream, maps);
    return cudaErrorInvalidValue;
}

template <uint32_t kFmt>
cudaError_t launch_wide(int kind, const dg::GemmParams& p, uint32_t grid, uint32_t smem, cudaStream_t stream, const CUtensorMap* maps) {
    if (kind == DG_OUT_BF16) return launch_kernel<kFmt, dg::kOutBf16, 2, kWideTiles>(p, grid, smem, stream, maps);
    return launch_kernel<kFmt, dg::kOutF32, 2, kWideTiles>(p, grid, smem, stream, maps);
}

template <uint32_t kFmt>
cudaError_t configure_contiguous_kernels_of() {
    cudaError_t e = configure_kernel<kFmt, dg::kOutBf16, 2, kWideTiles>();
    if (e == cudaSuccess) e = configure_kernel<kFmt, dg::kOutF32, 2, kWideTiles>();
    if (e == cudaSuccess) e = configure_kernel<kFmt, dg::kOutBf16, 1>();
    if (e == cudaSuccess) e = configure_kernel<kFmt, dg::kOutBf16, 2>();
    if (e == cudaSuccess) e = configure_kernel<kFmt, dg::kOutF32, 1>();
    if (e == cudaSuccess) e = configure_kernel<kFmt, dg::kOutF32, 2>();
    if (e == cudaSuccess) e = configure_kernel<kFmt, dg::kOutBf16, 1, 1>();
    if (e == cudaSuccess) e = configure_kernel<kFmt, dg::kOutBf16, 1, 2>();
    if (e == cudaSuccess) e = configure_kernel<kFmt, dg::kOutBf16, 2, 1>();
    if (e == cudaSuccess) e = configure_kernel<kFmt, dg::kOutBf16, 2, 2>();
    if (e == cudaSuccess) e = configure_kernel<kFmt, dg::kOutF32, 1, 1>();
    if (e == cudaSuccess) e = configure_kernel<kFmt, dg::kOutF32, 1, 2>();
    if (e == cudaSuccess) e = configure_kernel<kFmt, dg::kOutF32, 2, 1>();
    if (e == cudaSuccess) e = configure_kernel<kFmt, dg::kOutF32, 2, 2>();
    return e;
}
// Everything dg_m_grouped_fp8_fp4_gemm_contiguous[_ends] can launch, configured (and loaded) for the current device.
cudaError_t configure_contiguous_kernels() {
    cudaError_t e = configure_contiguous_kernels_of<dg::kFmtMxf8f6f4>();
    if (e == cudaSuccess) e = configure_contiguous_kernels_of<dg::kFmtMxf4>();
    if (e == cudaSuccess) e = configure_kernel<dg::kFmtMxf8f6f4, dg::kOutSwiGluFp8, 2>();
    cudaFuncAttributes fa;
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, dg::dg_group_ends_kernel);
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, dg::dg_group_ends_scan_kernel);
    return e;
}

// Makes a scratch buffer of the context's present stream at least `bytes` long (all zero when it is new, if `zeroed`).  The stream may
// be capturing: allocations are then made in the relaxed mode, outside the graph, and a buffer whose address went into a graph is
// never freed before the context, so that the graph can be replayed after the buffer was outgrown.
int reserve(dg_ctx* ctx, ScratchBuffer* buf, size_t bytes, bool zeroed = false) {
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    const bool capturing = cudaStreamIsCapturing(ctx->stream, &status) != cudaSuccess || status != cudaStreamCaptureStatusNone;
    if (buf->bytes < bytes) {
        DG_CUDA(cudaSetDevice(ctx->ordinal));
        if (buf->ptr && (buf->captured || capturing)) {
            ScratchBlock* block = new (std::nothrow) ScratchBlock{buf->ptr, ctx->replaced};
            if (block == nullptr) return fail(DG_ERR_DRIVER, "out of host memory");
            ctx->replaced = block;
        } else if (buf->ptr) {
            cudaFree(buf->ptr);
        }
        *buf = ScratchBuffer();
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        DG_CUDA(cudaThreadExchangeStreamCaptureMode(&mode));
        void* ptr = nullptr;
        cudaError_t e = cudaMalloc(&ptr, bytes);
        if (e == cudaSuccess && zeroed) {
            cudaStream_t side = nullptr;        // not the context's stream: a captured fill would only run with the graph
            e = cudaStreamCreateWithFlags(&side, cudaStreamNonBlocking);
            if (e == cudaSuccess) e = cudaMemsetAsync(ptr, 0, bytes, side);
            if (e == cudaSuccess) e = cudaStreamSynchronize(side);
            if (side) cudaStreamDestroy(side);
            if (e != cudaSuccess) cudaFree(ptr);
        }
        cudaThreadExchangeStreamCaptureMode(&mode);
        if (e != cudaSuccess) return fail(DG_ERR_DRIVER, "allocating %zu bytes of scratch: %s", bytes, cudaGetErrorString(e));
        buf->ptr = ptr;
        buf->bytes = bytes;
    }
    buf->captured |= capturing;
    return DG_OK;
}

int launch_skinny(dg_ctx* ctx, const dg_lp_operand* a, const dg_lp_operand* b, const dg_out* out, const dg_epilogue& e, const Problem& pr, uint32_t warps) {
    const uint32_t tiles = skinny_row_tiles(pr.m);
    // what the tensor maps of the other kernels ask for
    if (reinterpret_cast<uintptr_t>(a->data) % 16 != 0 || reinterpret_cast<uintptr_t>(b->data) % 16 != 0 || reinterpret_cast<uintptr_t>(a->sf) % 16 != 0 ||
        reinterpret_cast<uintptr_t>(b->sf) % 16 != 0 || reinterpret_cast<uintptr_t>(out->buf) % 16 != 0)
        return fail(DG_ERR_SHAPE, "operands, scales and output must be 16-byte aligned");
    dg::SkinnyParams p = {static_cast<const uint8_t*>(a->data), static_cast<const uint8_t*>(b->data), a->sf, b->sf, out->buf, pr.m, pr.n, pr.k / 128,
                          a->ld, b->ld, align4(pr.m), align4(pr.n), out->ld, e.has_alpha ? 1u : 0u, e.accumulate ? 1u : 0u, e.alpha};
    DG_CUDA(cudaSetDevice(ctx->ordinal));
    const bool f32 = out->kind == DG_OUT_F32;
    const dim3 grid(ceil_div(pr.n, dg::kSkinnyCols));
    auto run = [&](auto kernel, uint32_t warps) { return launch(kernel, grid, warps * 32, 0, ctx->stream, p); };
    auto with_warps = [&](auto count) {
        constexpr uint32_t kWarps = decltype(count)::value;
        if (tiles == 4) return f32 ? run(dg::dg_gemm_skinny_kernel<4, kWarps, true>, kWarps) : run(dg::dg_gemm_skinny_kernel<4, kWarps, false>, kWarps);
        if (tiles == 1) return f32 ? run(dg::dg_gemm_skinny_kernel<1, kWarps, true>, kWarps) : run(dg::dg_gemm_skinny_kernel<1, kWarps, false>, kWarps);
        return f32 ? run(dg::dg_gemm_skinny_kernel<2, kWarps, true>, kWarps) : run(dg::dg_gemm_skinny_kernel<2, kWarps, false>, kWarps);
    };
    if (print_configs()) fprintf(stderr, "[dgb200] few rows: m=%u n=%u k=%u -> block=%ux%u warps=%u\n", pr.m, pr.n, pr.k, 8 * tiles, dg::kSkinnyCols, warps);
    const cudaError_t ce = warps == 4 ? with_warps(std::integral_constant<uint32_t, 4>()) : (warps == 8 ? with_warps(std::integral_constant<uint32_t, 8>()) : with_warps(std::integral_constant<uint32_t, 16>()));
    if (ce != cudaSuccess) return fail(DG_ERR_DRIVER, "kernel launch failed: %s", cudaGetErrorString(ce));
    return DG_OK;
}

int launch_gemm(dg_ctx* ctx, const dg_lp_operand* a, const dg_lp_operand* b, const dg_out* out, const dg_epilogue* epi, const Problem& pr) {
    if (out == nullptr || out->buf == nullptr) return fail(DG_ERR_SHAPE, "null output");
    if (out->kind < DG_OUT_BF16 || out->kind > DG_OUT_SWIGLU_FP8) return fail(DG_ERR_SHAPE, "invalid output kind %d", out->kind);
    dg_epilogue e = {1.0f, 0, 0, 100};
    if (epi) e = *epi;
    const bool swiglu = out->kind == DG_OUT_SWIGLU_FP8;
    const bool fp8_out = out->kind == DG_OUT_FP8 || swiglu;
    if (fp8_out && (e.has_alpha || e.accumulate))
        return fail(DG_ERR_SHAPE, "the FP8-quantized output cannot combine alpha/accumulation");
    if (swiglu) {
        if (pr.bf16 || a->bits != 8 || b->bits != 8 || b->gran_k != 128)
            return fail(DG_ERR_UNSUPPORTED, "the fused gate/up activation takes e4m3 operands with per-128 weight scales");
        if (pr.n % 256 != 0) return fail(DG_ERR_SHAPE, "gate|up weights: rows per group (%u) must be 2 x a multiple of 128", pr.n);
    }
    if (e.accumulate && e.has_alpha) return fail(DG_ERR_SHAPE, "alpha and accumulation are mutually exclusive");
    const bool any_mn = !pr.bf16 && (a->major_mn || b->major_mn);
    if (any_mn && swiglu) return fail(DG_ERR_UNSUPPORTED, "the fused gate/up activation takes K-major operands");
    if (a->k != b->k) return fail(DG_ERR_SHAPE, "a.k (%u) != b.k (%u)", a->k, b->k);
    if (pr.m == 0 || pr.n == 0) return DG_OK;
    const bool contiguous = pr.type == DG_GEMM_M_GROUPED_CONTIGUOUS;
    const uint32_t a_groups = contiguous || pr.type == DG_GEMM_NORMAL ? 1 : pr.groups;
    const uint32_t b_groups = pr.type == DG_GEMM_NORMAL ? 1 : pr.groups;
    int rc = pr.bf16 ? DG_OK : check_operand(a, "a", pr.m * a_groups, a_groups);
    if (rc) return rc;
    rc = pr.bf16 ? DG_OK : check_operand(b, "b", pr.n * b_groups, b_groups);
    if (rc) return rc;
    const uint32_t d_rows = pr.m * a_groups;
    const uint32_t d_elem = out->kind == DG_OUT_F32 ? 4 : (fp8_out ? 1 : 2);
    const uint32_t n_out = swiglu ? pr.n / 2 : pr.n;     // output columns (the fused activation halves them)
    if (out->ld < n_out) return fail(DG_ERR_SHAPE, "output ld (%u) smaller than n (%u)", out->ld, n_out);
    if ((static_cast<size_t>(out->ld) * d_elem) % 16 != 0) return fail(DG_ERR_SHAPE, "output row pitch must be a multiple of 16 bytes");
    if (out->buf_len < static_cast<size_t>(d_rows - 1) * out->ld + n_out) return fail(DG_ERR_SHAPE, "output buffer too small");
    if (fp8_out) {
        if (out->sfd == nullptr) return fail(DG_ERR_SHAPE, "FP8 output needs sfd");
        if (n_out % 128 != 0) return fail(DG_ERR_SHAPE, "FP8 output needs n to be a multiple of 128");
        if (out->sfd_len < static_cast<size_t>(n_out / 128) * a_groups * align4(pr.m)) return fail(DG_ERR_SHAPE, "sfd buffer too small");
    }
    const uint32_t align = g_mk_alignment.load();
    if (swiglu && contiguous && align % 32 != 0)
        return fail(DG_ERR_UNSUPPORTED, "the fused gate/up activation needs an mk alignment of at least 32");

    dg_desc desc = {pr.type, pr.m, pr.n, pr.k, pr.groups, pr.expected_m, a->bits, b->bits, a->gran_k, b->gran_k,
                    static_cast<uint32_t>(out->kind), static_cast<uint32_t>(ctx->num_sms), (!pr.bf16 && a->major_mn) ? 1u : 0u,
                    (!pr.bf16 && b->major_mn) ? 1u : 0u};
    const uint32_t tc_util = (e.tc_util == 0 || e.tc_util > 100) ? 100 : e.tc_util;      // 0 means "unset", as in ops_sm100.rs:518-522
    dg_config cfg;
    KernelPlan plan;
    rc = choose_config(&desc, (e.accumulate ? kNoKRanges : 0u) | (pr.bf16 ? kNoWideTiles : 0u) | (pr.bf16 || tc_util < 100 ? kNoSkinny : 0u), &cfg, &plan);
    if (rc) return rc;
    if (plan.skinny_warps != 0) return launch_skinny(ctx, a, b, out, e, pr, plan.skinny_warps);
    const bool swap = plan.swap;
    // the swapped family's kernel takes the operands with their roles exchanged: its operand A (UMMA M side) is the weights
    const dg_lp_operand* ka = swap ? b : a;
    const dg_lp_operand* kb = swap ? a : b;
    const uint32_t ka_rows = swap ? pr.n : pr.m, kb_rows = swap ? pr.m : pr.n;              // per group
    const uint32_t ka_groups = swap ? b_groups : a_groups, kb_groups = swap ? a_groups : b_groups;
    if (print_configs())
        fprintf(stderr, "[dgb200] type=%u m=%u n=%u k=%u groups=%u -> swap_ab=%u block=%ux%ux%u ctas=%u stages=%u accum=%u smem=%u tiles~%u splits=%u\n",
                pr.type, pr.m, pr.n, pr.k, pr.groups, cfg.swap_ab, cfg.block_m, cfg.block_n, cfg.block_k, plan.ctas, cfg.num_stages,
                cfg.num_accum_stages, cfg.smem_size, cfg.num_tiles, cfg.num_splits);

    const bool mxf4 = a->bits == 4 && b->bits == 4;
    const uint32_t block_k = cfg.block_k;
    const uint32_t splits = plan.splits;
    const uint32_t ws_pitch = align4(pr.n);
    if (splits > 1) {
        // first family: one (m, n) plane per range; swapped family: one accumulator per tile, CTA of the pair and range
        rc = reserve(ctx, &ctx->scratch->splitk_ws, sizeof(float) * (swap ? static_cast<size_t>(plan.tiles) * plan.ctas * splits * ceil_div(plan.umma_n, 32) * 32 * dg::kBlockM
                                                                 : static_cast<size_t>(splits) * pr.m * ws_pitch));
        if (rc) return rc;
        const uint32_t counters = plan.tiles * plan.ctas;
        if (swap) rc = reserve(ctx, &ctx->scratch->splitk_counters, sizeof(uint32_t) * (counters < 1024 ? 1024 : counters), true);
        if (rc) return rc;
    }
    float* const splitk_ws = static_cast<float*>(ctx->scratch->splitk_ws.ptr);
    const uint32_t sfa_words = 4 * ka->gran_k >= block_k ? 1 : block_k / (4 * ka->gran_k);
    const uint32_t sfb_words = 4 * kb->gran_k >= block_k ? 1 : block_k / (4 * kb->gran_k);
    const uint32_t sf_block_n = ceil_div(plan.umma_n, 128) * 128;

    CUtensorMap maps[7];
    bool wide_k = false;
    {
        // packed e2m1 stays packed in shared memory for kind::mxf4 (16U4_ALIGN8B) and is expanded to one code per byte
        // for the mixed kind (16U4_ALIGN16B); dims and boxes of both are in logical 4-bit elements, pitches in bytes
        auto map_dtype = [&](uint32_t bits) {
            return bits == 8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : (mxf4 ? CU_TENSOR_MAP_DATA_TYPE_16U4_ALIGN8B : CU_TENSOR_MAP_DATA_TYPE_16U4_ALIGN16B);
        };
        const uint64_t a_pitch = ka->bits == 4 ? ka->ld / 2 : ka->ld, b_pitch = kb->bits == 4 ? kb->ld / 2 : kb->ld;
        uint64_t dims[3] = {pr.k, ka_rows, ka_groups};
        uint64_t strides[2] = {a_pitch, a_pitch * ka_rows};
        const uint32_t slab = mxf4 ? 256u : 128u;    // one 128-byte slab of K per TMA box
        uint32_t box[3] = {slab, dg::kBlockM, 1};
        if (!pr.bf16 && ka->major_mn) {
            // (groups, k, ld): rows innermost; a box is 128 rows x one slab of K
            dims[0] = ka_rows; dims[1] = pr.k; strides[0] = ka->ld; strides[1] = static_cast<uint64_t>(ka->ld) * pr.k;
            box[0] = 128; box[1] = slab;
        }
        // Two-slab stages of plain K-major byte operands: the operand is described as (128 bytes, rows, K slabs, groups) so that one
        // load brings both slabs of a stage (half as many TMA instructions per stage).  K must be whole slabs for that (a partial
        // last slab would read into the next row), otherwise the 3-D maps and one load per slab stay.
        const char* wide_env = getenv("DG_WIDE_K");
        // (not where the loads carry the evict-first hint: dense problems of a single row block, see below)
        const bool hinted = !swap && pr.type == DG_GEMM_NORMAL && pr.m <= 128 * plan.ctas;
        wide_k = plan.halves == 2 && !mxf4 && ka->bits == 8 && kb->bits == 8 && pr.k % 128 == 0 && !(!pr.bf16 && (ka->major_mn || kb->major_mn)) &&
                 !hinted && !(wide_env && strcmp(wide_env, "0") == 0);
        if (wide_k) {
            uint64_t d4[4] = {128, ka_rows, pr.k / 128, ka_groups};
            uint64_t s4[3] = {a_pitch, 128, a_pitch * ka_rows};
            uint32_t b4[4] = {128, dg::kBlockM, 2, 1};
            rc = encode_map(&maps[0], CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, ka->data, d4, s4, b4, CU_TENSOR_MAP_SWIZZLE_128B, "A");
            if (rc) return rc;
            uint64_t e4[4] = {128, kb_rows, pr.k / 128, kb_groups};
            uint64_t t4[3] = {b_pitch, 128, b_pitch * kb_rows};
            uint32_t c4[4] = {128, swap ? dg::swap_main_rows(plan.umma_n, plan.ctas) : plan.umma_n / plan.ctas, 2, 1};
            rc = encode_map(&maps[1], CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, kb->data, e4, t4, c4, CU_TENSOR_MAP_SWIZZLE_128B, "B");
            if (rc) return rc;
        } else {
        rc = encode_map(&maps[0], map_dtype(ka->bits), 3, ka->data, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B, "A");
        if (rc) return rc;
        uint64_t bdims[3] = {pr.k, kb_rows, kb_groups};
        uint64_t bstrides[2] = {b_pitch, b_pitch * kb_rows};
        uint32_t bbox[3] = {slab, swap ? dg::swap_main_rows(plan.umma_n, plan.ctas) : plan.umma_n / plan.ctas, 1};
        if (!pr.bf16 && kb->major_mn) {
            bdims[0] = kb_rows; bdims[1] = pr.k; bstrides[0] = kb->ld; bstrides[1] = static_cast<uint64_t>(kb->ld) * pr.k;
            bbox[0] = 128; bbox[1] = slab;
        }
        rc = encode_map(&maps[1], map_dtype(kb->bits), 3, kb->data, bdims, bstrides, bbox, CU_TENSOR_MAP_SWIZZLE_128B, "B");
        if (rc) return rc;
        }
        if (swap) {
            // smaller boxes of the activations: for tiles with few rows, and for the rows of a tile beyond 256
            uint64_t pdims[3] = {pr.k, kb_rows, kb_groups};
            uint64_t pstrides[2] = {b_pitch, b_pitch * kb_rows};
            uint32_t pbox[3] = {slab, dg::swap_part_rows(dg::swap_main_rows(plan.umma_n, plan.ctas)), 1};
            rc = encode_map(&maps[5], map_dtype(kb->bits), 3, kb->data, pdims, pstrides, pbox, CU_TENSOR_MAP_SWIZZLE_128B, "B part");
            if (rc) return rc;
            pbox[1] = dg::kSwapTailRows;
            rc = encode_map(&maps[6], map_dtype(kb->bits), 3, kb->data, pdims, pstrides, pbox, CU_TENSOR_MAP_SWIZZLE_128B, "B tail");
            if (rc) return rc;
        }
    }
    const uint32_t sfa_cols = dg_sf_packed_cols(pr.k, ka->gran_k), sfb_cols = dg_sf_packed_cols(pr.k, kb->gran_k);
    {
        // bf16 operands carry no scales: the kernel never issues these loads, the maps only have to be well-formed
        uint64_t dims[2] = {align4(ka_rows), static_cast<uint64_t>(sfa_cols) * ka_groups};
        uint64_t strides[1] = {static_cast<uint64_t>(align4(ka_rows)) * 4};
        uint32_t box[2] = {128, sfa_words};
        rc = encode_map(&maps[2], CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, pr.bf16 ? ka->data : ka->sf, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_NONE, "SFA");
        if (rc) return rc;
        uint64_t bdims[2] = {align4(kb_rows), static_cast<uint64_t>(sfb_cols) * kb_groups};
        uint64_t bstrides[1] = {static_cast<uint64_t>(align4(kb_rows)) * 4};
        uint32_t bbox[2] = {swiglu ? plan.umma_n / 2 : sf_block_n, sfb_words};   // fused activation: gate rows and up rows as two boxes
        if (swap) { bbox[0] = 128; bbox[1] = 1; }
        rc = encode_map(&maps[3], CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, pr.bf16 ? kb->data : kb->sf, bdims, bstrides, bbox, CU_TENSOR_MAP_SWIZZLE_NONE, "SFB");
        if (rc) return rc;
    }
    {
        // 32 rows per store; 32 columns of bf16 (64-byte rows) or f32, 128 columns of e4m3 (128-byte rows)
        if (swap) {
            // the swapped family writes the output itself, without a map, in 16-byte pieces
            if (reinterpret_cast<uintptr_t>(out->buf) % 16 != 0) return fail(DG_ERR_SHAPE, "D: base address must be 16-byte aligned");
        } else if (splits > 1) {
            // K ranges write f32 partial tiles into the workspace, one plane per range
            uint64_t dims[3] = {pr.n, pr.m, splits};
            uint64_t strides[2] = {static_cast<uint64_t>(ws_pitch) * 4, static_cast<uint64_t>(ws_pitch) * 4 * pr.m};
            uint32_t box[3] = {32, 32, 1};
            rc = encode_map(&maps[4], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, splitk_ws, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B, "D partials");
        } else {
            const CUtensorMapDataType dt = out->kind == DG_OUT_F32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32
                                           : (fp8_out ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16);
            const uint64_t pitch = static_cast<uint64_t>(out->ld) * d_elem;
            uint64_t dims[3] = {n_out, pr.m, a_groups};
            uint64_t strides[2] = {pitch, pitch * pr.m};
            uint32_t box[3] = {out->kind == DG_OUT_FP8 ? 128u : 32u, 32, 1};   // the fused activation stores 32 x 32 bytes, unswizzled
            rc = encode_map(&maps[4], dt, 3, out->buf, dims, strides, box,
                            swiglu ? CU_TENSOR_MAP_SWIZZLE_NONE : (out->kind == DG_OUT_BF16 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B), "D");
        }
        if (rc) return rc;
    }

    dg::GemmParams p;
    memset(&p, 0, sizeof(p));
    p.m = swap ? pr.n : pr.m;     // rows of the kernel's operand A per group (swapped family: weight rows)
    p.n = swap ? pr.m : n_out;
    p.k = pr.k;
    p.tile_n = swiglu ? plan.umma_n / 2 : plan.umma_n + plan.block_n2;
    p.block_n2 = plan.block_n2;
    p.num_groups = pr.groups;
    p.gemm_type = pr.type;
    p.block_n = plan.umma_n;
    p.block_k_elems = block_k;
    p.num_splits = splits;
    const uint32_t split_unit = 4 / plan.halves;
    p.kb_per_split = splits > 1 ? ceil_div(ceil_div(ceil_div(pr.k, block_k), splits), split_unit) * split_unit : ceil_div(pr.k, block_k);
    if (swap) {
        p.acc_stride = dg::gemm_swap_acc_stride(plan.umma_n, sfa_words, sfb_words);
        p.acc_edge_chunks = ceil_div(plan.umma_n, 32) - p.acc_stride / 32;
        if (p.acc_stride == plan.umma_n) p.acc_edge_chunks = 0;
        p.table_groups = plan.table_groups;
        p.splitk_ws = splitk_ws;
        p.splitk_counters = static_cast<uint32_t*>(ctx->scratch->splitk_counters.ptr);
    }
    p.num_stages = plan.stages;
    p.epi_bufs = swap ? 2 : plan.epi_bufs;
    p.num_accum_stages = plan.accum;
    p.gran_a = ka->gran_k;
    p.gran_b = kb->gran_k;
    // measured on B200: a 16U4_ALIGN16B load (e2m1 expanded to one code per byte) fills 128 bytes of shared memory per
    // 128 elements but signals only the 64 packed bytes it read on its barrier
    p.tx_shift_a = (!mxf4 && ka->bits == 4) ? 1 : 0;
    p.tx_shift_b = (!mxf4 && kb->bits == 4) ? 1 : 0;
    p.fmt_a = ka->bits == 8 ? 0u : 5u;
    p.fmt_b = kb->bits == 8 ? 0u : 5u;
    p.sf_a_cols = sfa_cols;
    p.sf_b_cols = sfb_cols;
    p.mk_alignment = align;
    // groups start at multiples of `align` rows; tiles stay 128 (or 256) rows tall and simply run into the next group's rows,
    // which are computed and not stored.  Stores go out in 32-row boxes, so only an alignment of 16 needs row-exact stores.
    // Both tile families write the same rows: a group's own and its padding up to the next multiple of 32.
    p.mask_rows = (contiguous && align % 32 != 0) ? 1 : 0;
    p.out_ptr = out->buf;
    p.out_ld = out->ld;
    {
        // dense problems of a single row block read every weight byte exactly once: those loads carry the L2 evict-first hint
        // (+9 % on 128 x 7168 x 16384).  Grouped problems with small groups were measured 4 % slower with it (a group's second row
        // block, running on a neighbouring CTA pair, finds its weight tile gone) and keep plain loads.  DG_STREAM_HINT=0 turns it off.
        const uint32_t row_block = swap ? plan.umma_n : 128 * plan.ctas;
        const char* v = getenv("DG_STREAM_HINT");
        const bool once = pr.type == DG_GEMM_NORMAL && pr.m <= row_block && !(v && strcmp(v, "0") == 0);
        p.stream_a = (once && swap) ? 1 : 0;
        p.stream_b = (once && !swap) ? 1 : 0;
    }
    p.wide_k = wide_k ? 1 : 0;
    p.mn_a = (!pr.bf16 && ka->major_mn) ? 1 : 0;
    p.mn_b = (!pr.bf16 && kb->major_mn) ? 1 : 0;
    p.accumulate = e.accumulate ? 1 : 0;
    p.tc_util = tc_util;
    p.has_alpha = (e.has_alpha && (swap || splits == 1)) ? 1 : 0;   // with K ranges summed by the second kernel alpha is applied there
    p.alpha = e.alpha;
    p.sfd = out->sfd;
    p.sfd_stride = align4(pr.m);
    p.grouped_layout = pr.layout;
    p.status = ctx->status;
#ifdef DG_PROFILE
    {   // debug builds: DG_PROF_PTR carries a device buffer address (8 x int64 per CTA)
        const char* pp = getenv("DG_PROF_PTR");
        p.prof = pp ? reinterpret_cast<long long*>(strtoull(pp, nullptr, 0)) : nullptr;
        const char* df = getenv("DG_DEBUG_FLAGS");
        p.debug_flags = df ? static_cast<uint32_t>(atoi(df)) : 0;
    }
#endif

    const uint32_t ctas = plan.ctas;
    uint32_t grid = static_cast<uint32_t>(ctx->num_sms) / ctas * ctas;
    if (pr.type == DG_GEMM_NORMAL || pr.type == DG_GEMM_BATCHED)
    {
        const uint32_t units = plan.tiles * splits;
        if (plan.block_n2 != 0) p.whole_tiles = wide_waves(pr.m, pr.n, plan.umma_n, grid / 2).whole;
        grid = units * ctas < grid ? units * ctas : grid;
    }
    const int kernel_out = splits > 1 && !swap ? DG_OUT_F32 : out->kind;
    const uint32_t smem = plan.smem;
    if (!swap && plan.block_n2 == 0 && (pr.type == DG_GEMM_NORMAL || pr.type == DG_GEMM_BATCHED) && kernel_out == DG_OUT_F32 &&
        static_cast<uint64_t>(plan.tiles) * splits <= static_cast<uint32_t>(ctx->num_sms) / ctas) {
        // one tile per CTA (pair): does the operand ring hold the CTA's 128 rows of it?
        const uint32_t ring = plan.stages * plan.halves * (dg::kBlockM + plan.umma_n / ctas) * dg::kBlockKBytes;
        p.stage_in_ring = dg::kBlockM * plan.umma_n * 4 <= ring ? 1 : 0;
    }
    DG_CUDA(cudaSetDevice(ctx->ordinal));
    cudaError_t ce;
    if (swap) {
        if (pr.bf16) ce = launch_swapped<dg::kFmtBf16>(plan, kernel_out, p, grid, ctx->stream, maps);
        else if (mxf4) ce = launch_swapped<dg::kFmtMxf4>(plan, kernel_out, p, grid, ctx->stream, maps);
        else ce = launch_swapped<dg::kFmtMxf8f6f4>(plan, kernel_out, p, grid, ctx->stream, maps);
    } else if (plan.block_n2 != 0) {
        if (mxf4) ce = launch_wide<dg::kFmtMxf4>(kernel_out, p, grid, smem, ctx->stream, maps);
        else ce = launch_wide<dg::kFmtMxf8f6f4>(kernel_out, p, grid, smem, ctx->stream, maps);
    } else if (pr.bf16) ce = ctas == 2 ? launch_by_out<dg::kFmtBf16, 2>(kernel_out, p, grid, smem, ctx->stream, maps)
                                : launch_by_out<dg::kFmtBf16, 1>(kernel_out, p, grid, smem, ctx->stream, maps);
    else if (mxf4) ce = ctas == 2 ? launch_by_out<dg::kFmtMxf4, 2>(kernel_out, p, grid, smem, ctx->stream, maps)
                                  : launch_by_out<dg::kFmtMxf4, 1>(kernel_out, p, grid, smem, ctx->stream, maps);
    else ce = ctas == 2 ? launch_by_out<dg::kFmtMxf8f6f4, 2>(kernel_out, p, grid, smem, ctx->stream, maps)
                        : launch_by_out<dg::kFmtMxf8f6f4, 1>(kernel_out, p, grid, smem, ctx->stream, maps);
    if (ce == cudaSuccess && splits > 1 && !swap) {
        const uint64_t threads = static_cast<uint64_t>(pr.m) * ceil_div(pr.n, 4);
        const uint32_t blocks = static_cast<uint32_t>((threads + 255) / 256);
        const float alpha = e.has_alpha ? e.alpha : 1.0f;
        ce = launch(out->kind == DG_OUT_BF16 ? dg::dg_splitk_reduce_kernel<true> : dg::dg_splitk_reduce_kernel<false>, blocks, 256, 0, ctx->stream,
                    splitk_ws, splits, pr.m, pr.n, ws_pitch, alpha, out->buf, out->ld);
    }
    if (ce != cudaSuccess) return fail(DG_ERR_DRIVER, "kernel launch failed: %s", cudaGetErrorString(ce));
    return DG_OK;
}

struct F32Plan {
    uint32_t ctas, block_n;          // a pair of CTAs with 256 x 256 tiles, or single CTAs with 128 x 128 tiles
    uint32_t splits, kb_per_split;   // K ranges (dense problems with few tiles), in k-blocks of 128
};
// Costs in microseconds.  A K block takes 0.36 of a 128 x 128 tile; that, and the 3.5 that K ranges pay for the second launch beside their planes, were
// fitted on B200 over 22 dense problems (m 68-6900, n 560-8096, k 1152-8064).  K ranges never make more than one wave.  A 256 x 256 tile (a quarter
// as many tiles, half the SM pairs) counts with
//   0.45 in dense problems: the pair wins wherever its waves are fewer than 0.8 of the others.  It took 0.56 before its loop became shorter; over 25
//     problems between the two lines (m 1046-7787, n 736-4976, k 1024-5760) it takes 0.94 of the single tiles' time, 0.88 to 1.01;
//   0.56 in contiguous groups, of which an arena says only how many rows they may have: over 50 problems between the two lines (2-96 groups) the pair takes 0.93
//     of the time where more than three quarters of the arena are live, 1.04 with 0.4 and 1.27 with 0.1 of it (16 groups of 75 rows in 8192, 1120 x 2816:
//     20.5 -> 35.3 us), 1.09 on average.
F32Plan choose_f32scale(uint32_t type, uint32_t m, uint32_t n, uint32_t k, uint32_t groups, uint32_t sms) {
    const uint32_t kbs = k / 128;
    const bool dense = type == DG_GEMM_NORMAL;
    // row blocks: a contiguous group ends inside a tile, half a tile is lost on average.  Its padding makes no tiles: counted as rows it
    // made three waves of 128-row tiles out of what is one or two, and small groups got tiles of 256 rows, half of them empty
    // (12 groups of 87 rows, 1152 x 3456: 22.6 us with 128-row tiles, 28.7 with 256).
    auto row_blocks = [&](uint32_t tile_m) {
        if (type == DG_GEMM_M_GROUPED_CONTIGUOUS) return groups * (contiguous_rows(m, groups) / tile_m + 0.5);
        return static_cast<double>(dense ? 1u : groups) * ceil_div(m, tile_m);
    };
    const double tiles = row_blocks(128) * ceil_div(n, 128), pair_tiles = row_blocks(256) * ceil_div(n, 256);
    auto waves = [](double t, uint32_t workers) { return static_cast<double>(static_cast<uint64_t>(t / workers + 0.999)); };
    F32Plan best = {1, 128, 1, kbs};
    double best_cost = waves(tiles, sms) * (kbs * 0.36 + 0.6);
    const double pair_cost = sms >= 2 ? waves(pair_tiles, sms / 2) * (kbs * (dense ? 0.45 : 0.56) + 1.2) : best_cost;
    // (a masked group's rows are known to the device only and usually fewer than its slot: small tiles)
    if (type != DG_GEMM_M_GROUPED_MASKED && pair_cost < best_cost) {
        best = {2, 256, 1, kbs};
        best_cost = pair_cost;
    }
    for (uint32_t splits = 2; dense && n % 4 == 0 && splits <= 8; ++splits) {
        const uint32_t per = ceil_div(kbs, splits);
        if (per < 4 || per * (splits - 1) >= kbs || tiles * splits > sms) continue;
        const double cost = per * 0.36 + 0.6 + 3.5 + static_cast<double>(splits) * m * n * 4.0 / 4e6;
        if (cost < best_cost) {
            best = {1, 128, splits, per};
            best_cost = cost;
        }
    }
    return best;
}

template <uint32_t kCtas, uint32_t kBlockN, bool kPartial>
cudaError_t launch_f32scale_kernel(const dg::F32ScaleParams& q, uint32_t grid, uint32_t smem, dg_ctx* ctx, const CUtensorMap* maps) {
    auto kernel = dg::dg_gemm_f32scale_kernel<kCtas, kBlockN, kPartial>;
    static std::atomic<uint64_t> configured{0};
    if (ctx->ordinal >= 64 || !(configured.load() & (1ull << ctx->ordinal))) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSmemCapacity));
        if (e != cudaSuccess) return e;
        if (ctx->ordinal < 64) configured.fetch_or(1ull << ctx->ordinal);
    }
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(grid, 1, 1);
    cfg.blockDim = dim3(dg::kF32Threads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kCtas;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, q, maps[0], maps[1], maps[2]);
}

int ensure_group_ends(dg_ctx* ctx, uint32_t groups, uint32_t** ends) {
    const int rc = reserve(ctx, &ctx->scratch->group_ends, sizeof(uint32_t) * (groups < 1024 ? 1024 : groups));
    *ends = static_cast<uint32_t*>(ctx->scratch->group_ends.ptr);
    return rc;
}

int run_group_ends(dg_ctx* ctx, const int32_t* m_indices, uint32_t m, uint32_t groups, uint32_t* ends) {
    DG_CUDA(cudaMemsetAsync(ends, 0, static_cast<size_t>(groups) * 4, ctx->stream));
    if (m > 0) DG_CUDA(launch(dg::dg_group_ends_kernel, ceil_div(m, 256), 256, 0, ctx->stream, m_indices, ends, groups, m));
    DG_CUDA(launch(dg::dg_group_ends_scan_kernel, 1, 1024, 0, ctx->stream, ends, groups));
    return DG_OK;
}

}  // namespace

extern "C" {

int dg_fp8_fp4_gemm(dg_ctx* ctx, const dg_lp_operand* a, const dg_lp_operand* b, const dg_out* out, const dg_epilogue* epi) {
    if (!ctx || !a || !b || !out) return fail(DG_ERR_SHAPE, "null argument");
    if (out->kind == DG_OUT_FP8) return fail(DG_ERR_SHAPE, "the dynamic FP8 output is only supported by the batched and masked APIs");
    Problem pr = {DG_GEMM_NORMAL, a->rows, b->rows, a->k, 1, a->rows, nullptr};
    return launch_gemm(ctx, a, b, out, epi, pr);
}

int dg_bf16_gemm(dg_ctx* ctx, const uint16_t* a, uint32_t a_ld, uint32_t m, const uint16_t* b, uint32_t b_ld, uint32_t n, uint32_t k,
                 const dg_out* out, const dg_epilogue* epi) {
    if (!ctx || !a || !b || !out) return fail(DG_ERR_SHAPE, "null argument");
    if (out->kind == DG_OUT_FP8) return fail(DG_ERR_UNSUPPORTED, "the bf16 GEMM writes bf16 or f32 outputs");
    if (k == 0 || k % 8 != 0) return fail(DG_ERR_SHAPE, "bf16 k (%u) must be a positive multiple of 8", k);
    if (a_ld < k || b_ld < k || a_ld % 8 != 0 || b_ld % 8 != 0) return fail(DG_ERR_SHAPE, "leading dimensions must be >= k and multiples of 8 elements");
    // the kernel sees K-major rows of 2k bytes: same tiles, same TMA boxes, same 32-byte UMMA steps as the 8-bit formats
    dg_lp_operand a8 = {a, nullptr, m, 2 * k, 2 * a_ld, 8, 128, 0, static_cast<size_t>(m) * 2 * a_ld, 0};
    dg_lp_operand b8 = {b, nullptr, n, 2 * k, 2 * b_ld, 8, 128, 0, static_cast<size_t>(n) * 2 * b_ld, 0};
    Problem pr = {DG_GEMM_NORMAL, m, n, 2 * k, 1, m, nullptr, true};
    return launch_gemm(ctx, &a8, &b8, out, epi, pr);
}

int dg_m_grouped_fp8_fp4_gemm_contiguous_ends(dg_ctx* ctx, const dg_lp_operand* a, const uint32_t* group_ends, const dg_lp_operand* b,
                                              const dg_out* out, uint32_t num_groups, const dg_epilogue* epi) {
    if (!ctx || !a || !b || !out || !group_ends) return fail(DG_ERR_SHAPE, "null argument");
    if (num_groups == 0 || b->rows % num_groups != 0) return fail(DG_ERR_SHAPE, "b.rows (%u) must be num_groups (%u) x n", b->rows, num_groups);
    if (out->kind == DG_OUT_FP8) return fail(DG_ERR_SHAPE, "the dynamic FP8 output is only supported by the batched and masked APIs");
    if (epi && epi->accumulate) return fail(DG_ERR_SHAPE, "accumulation is not supported by the grouped contiguous layout");
    Problem pr = {DG_GEMM_M_GROUPED_CONTIGUOUS, a->rows, b->rows / num_groups, a->k, num_groups, a->rows, group_ends};
    return launch_gemm(ctx, a, b, out, epi, pr);
}

int dg_m_grouped_fp8_fp4_gemm_contiguous(dg_ctx* ctx, const dg_lp_operand* a, const int32_t* m_indices, const dg_lp_operand* b,
                                         const dg_out* out, uint32_t num_groups, const dg_epilogue* epi) {
    if (!ctx || !a || !b || !out || !m_indices) return fail(DG_ERR_SHAPE, "null argument");
    if (num_groups == 0) return fail(DG_ERR_SHAPE, "num_groups must be positive");
    DG_CUDA(cudaSetDevice(ctx->ordinal));
    uint32_t* ends = nullptr;
    int rc = ensure_group_ends(ctx, num_groups, &ends);
    if (rc) return rc;
    rc = run_group_ends(ctx, m_indices, a->rows, num_groups, ends);
    if (rc) return rc;
    return dg_m_grouped_fp8_fp4_gemm_contiguous_ends(ctx, a, ends, b, out, num_groups, epi);
}

int dg_m_grouped_fp8_fp4_gemm_masked(dg_ctx* ctx, const dg_lp_operand* a, const int32_t* masked_m, const dg_lp_operand* b,
                                     const dg_out* out, uint32_t num_groups, uint32_t expected_m, const dg_epilogue* epi) {
    if (!ctx || !a || !b || !out || !masked_m) return fail(DG_ERR_SHAPE, "null argument");
    if (num_groups == 0 || b->rows % num_groups != 0) return fail(DG_ERR_SHAPE, "b.rows (%u) must be num_groups (%u) x n", b->rows, num_groups);
    Problem pr = {DG_GEMM_M_GROUPED_MASKED, a->rows, b->rows / num_groups, a->k, num_groups, expected_m ? expected_m : 1,
                  reinterpret_cast<const uint32_t*>(masked_m)};
    return launch_gemm(ctx, a, b, out, epi, pr);
}

int dg_fp8_fp4_bmm(dg_ctx* ctx, const dg_lp_operand* a, const dg_lp_operand* b, const dg_out* out, uint32_t num_groups,
                   const dg_epilogue* epi) {
    if (!ctx || !a || !b || !out) return fail(DG_ERR_SHAPE, "null argument");
    if (num_groups == 0) return fail(DG_ERR_SHAPE, "num_groups must be positive");
    Problem pr = {DG_GEMM_BATCHED, a->rows, b->rows, a->k, num_groups, a->rows, nullptr};
    return launch_gemm(ctx, a, b, out, epi, pr);
}

// ------------------------------------------------------------ f32-scale entry points
// The reference's older API hands scales over as f32 (activations transposed by transform_sf, weights one per
// 128x128 tile).  By default they are applied exactly, K block by K block, as the reference's CPU definition does
// (reference.rs:85-208): dg_gemm_f32scale_kernel.  With DG_F32_SCALES=exponent the calls do what the reference itself does on
// Blackwell (ops_sm100.rs:1414-1605): pack the exponents into UE8M0 words (mantissas are dropped, so the scales must be powers
// of two to be exact) and run the block-scaled kernel, which is about three times faster.
static int launch_f32scale(dg_ctx* ctx, uint32_t type, const uint8_t* a, uint32_t a_ld, const float* a_sf_t, const uint8_t* b, uint32_t b_ld,
                           const float* sfb, uint32_t m, uint32_t n, uint32_t k, uint32_t groups, const uint32_t* layout, uint16_t* out,
                           uint32_t out_ld) {
    if (m == 0 || n == 0) return DG_OK;
    const bool contiguous = type == DG_GEMM_M_GROUPED_CONTIGUOUS;
    const uint32_t a_groups = (type == DG_GEMM_NORMAL || contiguous) ? 1 : groups;
    const uint32_t b_groups = type == DG_GEMM_NORMAL ? 1 : groups;
    const uint32_t align = g_mk_alignment.load();
    if (contiguous && align % 32 != 0) return fail(DG_ERR_UNSUPPORTED, "the exact f32-scale path needs an mk alignment of at least 32");
    if (a_ld < k || b_ld < k || a_ld % 16 != 0 || b_ld % 16 != 0) return fail(DG_ERR_SHAPE, "leading dimensions must be >= k and multiples of 16 bytes");
    if (out_ld < n || (static_cast<size_t>(out_ld) * 2) % 16 != 0) return fail(DG_ERR_SHAPE, "output ld (%u) must be >= n and a multiple of 8 elements", out_ld);
    const F32Plan plan = choose_f32scale(type, m, n, k, groups, static_cast<uint32_t>(ctx->num_sms));
    if (print_configs())
        fprintf(stderr, "[dgb200] f32 scales: type=%u m=%u n=%u k=%u groups=%u -> block=%ux%u ctas=%u splits=%u\n", type, m, n, k, groups, 128 * plan.ctas,
                plan.block_n, plan.ctas, plan.splits);
    const uint32_t ws_pitch = align4(n);
    CUtensorMap maps[3];
    int rc;
    if (plan.splits > 1) {
        rc = reserve(ctx, &ctx->scratch->splitk_ws, sizeof(float) * plan.splits * m * ws_pitch);
        if (rc) return rc;
    }
    float* const splitk_ws = static_cast<float*>(ctx->scratch->splitk_ws.ptr);
    {
        uint64_t dims[3] = {k, m, a_groups};
        uint64_t strides[2] = {a_ld, static_cast<uint64_t>(a_ld) * m};
        uint32_t box[3] = {128, dg::kBlockM, 1};
        rc = encode_map(&maps[0], CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, a, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B, "A");
        if (rc) return rc;
        uint64_t bdims[3] = {k, n, b_groups};
        uint64_t bstrides[2] = {b_ld, static_cast<uint64_t>(b_ld) * n};
        uint32_t bbox[3] = {128, plan.block_n / plan.ctas, 1};
        rc = encode_map(&maps[1], CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, b, bdims, bstrides, bbox, CU_TENSOR_MAP_SWIZZLE_128B, "B");
        if (rc) return rc;
        const bool partial = plan.splits > 1;      // one f32 plane per K range, summed afterwards
        const uint64_t pitch = partial ? static_cast<uint64_t>(ws_pitch) * 4 : static_cast<uint64_t>(out_ld) * 2;
        uint64_t ddims[3] = {n, m, partial ? plan.splits : a_groups};
        uint64_t dstrides[2] = {pitch, pitch * m};
        uint32_t dbox[3] = {32, 32, 1};
        if (partial)
            rc = encode_map(&maps[2], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, splitk_ws, ddims, dstrides, dbox, CU_TENSOR_MAP_SWIZZLE_128B, "D partials");
        else
            rc = encode_map(&maps[2], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, out, ddims, dstrides, dbox, CU_TENSOR_MAP_SWIZZLE_64B, "D");
        if (rc) return rc;
    }
    dg::F32ScaleParams q;
    memset(&q, 0, sizeof(q));
    dg::GemmParams& p = q.g;
    p.m = m; p.n = n; p.k = k;
    p.num_groups = groups;
    p.gemm_type = type;
    p.block_n = p.tile_n = plan.block_n;
    p.block_k_elems = 128;
    p.num_splits = plan.splits;
    p.kb_per_split = plan.kb_per_split;
    p.num_accum_stages = 2;
    p.mk_alignment = align;
    p.grouped_layout = layout;
    p.status = ctx->status;
    uint32_t stages = dg::kMaxStages;
    while (stages > 1 && dg::f32scale_smem_bytes(plan.ctas, plan.block_n, plan.splits > 1, stages) > kSmemCapacity) --stages;
    p.num_stages = stages;
    q.sfa_t = a_sf_t;
    q.sfb = sfb;
    q.sfa_stride = align4(m);
    q.k_blocks = k / 128;
    q.n_blocks128 = ceil_div(n, 128);
    const uint32_t smem = dg::f32scale_smem_bytes(plan.ctas, plan.block_n, plan.splits > 1, stages);
    DG_CUDA(cudaSetDevice(ctx->ordinal));
    uint32_t grid = static_cast<uint32_t>(ctx->num_sms) / plan.ctas * plan.ctas;
    if (type == DG_GEMM_NORMAL || type == DG_GEMM_BATCHED) {
        const uint64_t ctas = static_cast<uint64_t>(ceil_div(m, dg::kBlockM * plan.ctas)) * ceil_div(n, plan.block_n) * (type == DG_GEMM_BATCHED ? groups : 1) *
                              plan.splits * plan.ctas;
        if (ctas < grid) grid = static_cast<uint32_t>(ctas);
    }
    cudaError_t ce;
    if (plan.ctas == 2) ce = launch_f32scale_kernel<2, 256, false>(q, grid, smem, ctx, maps);
    else if (plan.splits > 1) ce = launch_f32scale_kernel<1, 128, true>(q, grid, smem, ctx, maps);
    else ce = launch_f32scale_kernel<1, 128, false>(q, grid, smem, ctx, maps);
    if (ce == cudaSuccess && plan.splits > 1) {
        const uint64_t threads = static_cast<uint64_t>(m) * ceil_div(n, 4);
        ce = launch(dg::dg_splitk_reduce_kernel<true>, static_cast<uint32_t>((threads + 255) / 256), 256, 0, ctx->stream, splitk_ws, plan.splits, m, n,
                    ws_pitch, 1.0f, out, out_ld);
    }
    if (ce != cudaSuccess) return fail(DG_ERR_DRIVER, "kernel launch failed: %s", cudaGetErrorString(ce));
    return DG_OK;
}

static int bridge_common(dg_ctx* ctx, uint32_t type, const uint8_t* a, uint32_t a_ld, const float* a_sf_t, const uint8_t* b, uint32_t b_ld,
                         const float* sfb, uint32_t m, uint32_t n, uint32_t k, uint32_t groups, const uint32_t* layout, uint32_t expected_m,
                         uint16_t* out, uint32_t out_ld) {
    if (!ctx || !a || !a_sf_t || !b || !sfb || !out) return fail(DG_ERR_SHAPE, "null argument");
    if (k == 0 || k % 128 != 0) return fail(DG_ERR_SHAPE, "k (%u) must be a multiple of 128 (per-128-channel scaling)", k);
    if (n % 8 != 0) return fail(DG_ERR_SHAPE, "n (%u) must be a multiple of 8", n);
    if (groups == 0) return fail(DG_ERR_SHAPE, "num_groups must be positive");
    const bool contiguous = type == DG_GEMM_M_GROUPED_CONTIGUOUS;
    const uint32_t a_groups = (type == DG_GEMM_NORMAL || contiguous) ? 1 : groups;
    const uint32_t b_groups = type == DG_GEMM_NORMAL ? 1 : groups;
    {
        const char* mode = getenv("DG_F32_SCALES");
        if (!(mode && strcmp(mode, "exponent") == 0)) {
            const uint32_t* table = layout;
            if (contiguous) {
                // the group-end table the scheduler walks, built from m_indices in the context's scratch
                uint32_t* ends = nullptr;
                int rc = ensure_group_ends(ctx, groups, &ends);
                if (rc) return rc;
                DG_CUDA(cudaSetDevice(ctx->ordinal));
                rc = run_group_ends(ctx, reinterpret_cast<const int32_t*>(layout), m, groups, ends);
                if (rc) return rc;
                table = ends;
            }
            return launch_f32scale(ctx, type, a, a_ld, a_sf_t, b, b_ld, sfb, m, n, k, groups, table, out, out_ld);
        }
    }
    const size_t need[2] = {dg_sf_words(m * a_groups, k, 128, a_groups), dg_sf_words(n * b_groups, k, 128, b_groups)};
    DG_CUDA(cudaSetDevice(ctx->ordinal));
    int rc = reserve(ctx, &ctx->scratch->bridge_sf[0], need[0] * 4);
    if (rc == DG_OK) rc = reserve(ctx, &ctx->scratch->bridge_sf[1], need[1] * 4);
    if (rc) return rc;
    uint32_t *const sfa_words = static_cast<uint32_t*>(ctx->scratch->bridge_sf[0].ptr), *const sfb_words = static_cast<uint32_t*>(ctx->scratch->bridge_sf[1].ptr);
    // padding rows of the packed layouts must read as a valid exponent
    DG_CUDA(cudaMemsetAsync(sfa_words, 0, need[0] * 4, ctx->stream));
    DG_CUDA(cudaMemsetAsync(sfb_words, 0, need[1] * 4, ctx->stream));
    rc = dg_transform_sf_t_packed_ue8m0(ctx, a_sf_t, m * a_groups, k, 128, a_groups, sfa_words);
    if (rc) return rc;
    rc = dg_transform_sf2d_packed_ue8m0(ctx, sfb, k / 128, n * b_groups, k, b_groups, sfb_words);
    if (rc) return rc;
    dg_lp_operand a_op = {a, sfa_words, m, k, a_ld, 8, 128, 0, static_cast<size_t>(m) * a_groups * a_ld, need[0]};
    dg_lp_operand b_op = {b, sfb_words, type == DG_GEMM_BATCHED || type == DG_GEMM_NORMAL ? n : n * groups, k, b_ld, 8, 128, 0,
                          static_cast<size_t>(n) * b_groups * b_ld, need[1]};
    dg_out o = {DG_OUT_BF16, out, out_ld, nullptr, static_cast<size_t>(m) * a_groups * out_ld, 0};
    switch (type) {
        case DG_GEMM_NORMAL: return dg_fp8_fp4_gemm(ctx, &a_op, &b_op, &o, nullptr);
        case DG_GEMM_M_GROUPED_CONTIGUOUS:
            return dg_m_grouped_fp8_fp4_gemm_contiguous(ctx, &a_op, reinterpret_cast<const int32_t*>(layout), &b_op, &o, groups, nullptr);
        case DG_GEMM_M_GROUPED_MASKED:
            return dg_m_grouped_fp8_fp4_gemm_masked(ctx, &a_op, reinterpret_cast<const int32_t*>(layout), &b_op, &o, groups, expected_m, nullptr);
        default: return dg_fp8_fp4_bmm(ctx, &a_op, &b_op, &o, groups, nullptr);
    }
}

int dg_fp8_gemm_nt(dg_ctx* ctx, const uint8_t* a, uint32_t a_ld, const float* a_sf_t, const uint8_t* b, uint32_t b_ld, const float* sfb, uint32_t m,
                   uint32_t n, uint32_t k, uint16_t* out, uint32_t out_ld) {
    return bridge_common(ctx, DG_GEMM_NORMAL, a, a_ld, a_sf_t, b, b_ld, sfb, m, n, k, 1, nullptr, m, out, out_ld);
}
int dg_m_grouped_fp8_gemm_nt_contiguous(dg_ctx* ctx, const uint8_t* a, uint32_t a_ld, const float* a_sf_t, const uint8_t* b, uint32_t b_ld,
                                        const float* sfb, uint32_t m_total, uint32_t n, uint32_t k, uint16_t* out, uint32_t out_ld,
                                        const int32_t* m_indices, uint32_t num_groups) {
    if (!m_indices) return fail(DG_ERR_SHAPE, "null argument");
    return bridge_common(ctx, DG_GEMM_M_GROUPED_CONTIGUOUS, a, a_ld, a_sf_t, b, b_ld, sfb, m_total, n, k, num_groups,
                         reinterpret_cast<const uint32_t*>(m_indices), m_total, out, out_ld);
}
int dg_m_grouped_fp8_gemm_nt_masked(dg_ctx* ctx, const uint8_t* a, uint32_t a_ld, const float* a_sf_t, const uint8_t* b, uint32_t b_ld,
                                    const float* sfb, uint32_t m_max, uint32_t n, uint32_t k, uint16_t* out, uint32_t out_ld,
                                    const int32_t* masked_m, uint32_t num_groups, uint32_t expected_m) {
    if (!masked_m) return fail(DG_ERR_SHAPE, "null argument");
    return bridge_common(ctx, DG_GEMM_M_GROUPED_MASKED, a, a_ld, a_sf_t, b, b_ld, sfb, m_max, n, k, num_groups,
                         reinterpret_cast<const uint32_t*>(masked_m), expected_m, out, out_ld);
}
int dg_fp8_bmm_nt(dg_ctx* ctx, const uint8_t* a, uint32_t a_ld, const float* a_sf_t, const uint8_t* b, uint32_t b_ld, const float* sfb, uint32_t m,
                  uint32_t n, uint32_t k, uint16_t* out, uint32_t out_ld, uint32_t num_groups) {
    return bridge_common(ctx, DG_GEMM_BATCHED, a, a_ld, a_sf_t, b, b_ld, sfb, m, n, k, num_groups, nullptr, m, out, out_ld);
}

// ------------------------------------------------------- entry point that allocates nothing
// Scratch for dg_m_grouped_fp8_fp4_gemm_contiguous_static: words [0, 4) are the record a kernel
// writes when one of its bounded waits runs out, words [64, 64 + kStaticMaxGroups) hold the
// group-end table.  One copy per GPU that loads the library, kept until the process exits.
constexpr uint32_t kStaticMaxGroups = DG_STATIC_MAX_GROUPS;
constexpr uint32_t kStaticEndsOffset = 64;
static __device__ __align__(256) uint32_t g_static_scratch[kStaticEndsOffset + kStaticMaxGroups];

namespace {
struct StaticDevice {
    bool ready = false;
    uint32_t* scratch = nullptr;   // device address of g_static_scratch on this device
    int num_sms = 0;
};
StaticDevice g_static_devices[64];
std::mutex g_static_mutex;

// Once per device, with that device current: ask the runtime for the device address of the array.
// In host code the array's name is only a handle for this lookup, never a pointer a kernel can use.
int static_device_setup(int device, StaticDevice** out) {
    if (device < 0 || device >= 64) return fail(DG_ERR_SHAPE, "device ordinal %d out of range", device);
    std::lock_guard<std::mutex> lock(g_static_mutex);
    StaticDevice& d = g_static_devices[device];
    if (!d.ready) {
        DG_CUDA(cudaSetDevice(device));
        int major = 0;
        DG_CUDA(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device));
        if (major != 10) return fail(DG_ERR_UNSUPPORTED, "device %d is not sm_100; these kernels are built for sm_100a only", device);
        if (encode_tiled_fn() == nullptr) return fail(DG_ERR_DRIVER, "cuTensorMapEncodeTiled not found in the driver");
        DG_CUDA(cudaDeviceGetAttribute(&d.num_sms, cudaDevAttrMultiProcessorCount, device));
        uint32_t* ptr = nullptr;
        DG_CUDA(cudaGetSymbolAddress(reinterpret_cast<void**>(&ptr), g_static_scratch));
        d.scratch = ptr;
        // every kernel the contiguous path can reach gets its shared-memory opt-in (and its image loaded) now, so that later
        // calls with another output kind, operand format or tile choice do no set-up work
        DG_CUDA(configure_contiguous_kernels());
        d.ready = true;
    }
    *out = &d;
    return DG_OK;
}
}  // namespace

int dg_m_grouped_fp8_fp4_gemm_contiguous_static(int device, void* cuda_stream, const dg_lp_operand* a, const int32_t* m_indices,
                                                const dg_lp_operand* b, const dg_out* out, uint32_t num_groups, const dg_epilogue* epi) {
    if (!a || !b || !out || !m_indices) return fail(DG_ERR_SHAPE, "null argument");
    if (num_groups == 0) return fail(DG_ERR_SHAPE, "num_groups must be positive");
    if (num_groups > kStaticMaxGroups)
        return fail(DG_ERR_SHAPE, "num_groups (%u) exceeds the %u groups the built-in scratch holds; use dg_m_grouped_fp8_fp4_gemm_contiguous",
                    num_groups, kStaticMaxGroups);
    StaticDevice* dev = nullptr;
    int rc = static_device_setup(device, &dev);
    if (rc) return rc;
    DG_CUDA(cudaSetDevice(device));
    // a context view on the stack: nothing is created, nothing has to be destroyed
    dg_ctx view;
    view.ordinal = device;
    view.stream = static_cast<cudaStream_t>(cuda_stream);
    view.num_sms = dev->num_sms;
    view.status = reinterpret_cast<dg::Status*>(dev->scratch);
    uint32_t* ends = dev->scratch + kStaticEndsOffset;
    // the table keeps the previous call's contents: run_group_ends clears the entries it is about to fill
    rc = run_group_ends(&view, m_indices, a->rows, num_groups, ends);
    if (rc) return rc;
    return dg_m_grouped_fp8_fp4_gemm_contiguous_ends(&view, a, ends, b, out, num_groups, epi);
}

int dg_static_check_status(int device, void* cuda_stream) {
    StaticDevice* dev = nullptr;
    int rc = static_device_setup(device, &dev);
    if (rc) return rc;
    DG_CUDA(cudaSetDevice(device));
    cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
    dg::Status st;
    // a stack destination and 16 bytes: the copy allocates nothing; it is ordered after the GEMMs enqueued on `stream`
    DG_CUDA(cudaMemcpyAsync(&st, dev->scratch, sizeof(st), cudaMemcpyDeviceToHost, stream));
    DG_CUDA(cudaStreamSynchronize(stream));
    if (st.code != 0) {
        DG_CUDA(cudaMemsetAsync(dev->scratch, 0, sizeof(st), stream));
        DG_CUDA(cudaStreamSynchronize(stream));
        return fail(DG_ERR_TIMEOUT, "a device-side wait ran out: block %u, site 0x%x, parity %u", st.block, st.site, st.extra);
    }
    return DG_OK;
}

// ------------------------------------------------------------------ quantise / re-layout
static int cast_common(dg_ctx* ctx, const uint16_t* src, uint32_t src_ld, uint32_t rows, uint32_t k, uint32_t gran, uint32_t groups, int rule,
                       bool fp4, uint8_t* dst, uint32_t* sf, bool silu_mul = false, const uint32_t* live_rows = nullptr) {
    if (!ctx || !src || !dst || !sf) return fail(DG_ERR_SHAPE, "null argument");
    if (groups == 0) groups = 1;
    if (rows % groups != 0) return fail(DG_ERR_SHAPE, "rows (%u) must be a multiple of num_groups (%u)", rows, groups);
    if (src_ld < (silu_mul ? 2 * k : k) || src_ld % 8 != 0)
        return fail(DG_ERR_SHAPE, "src_ld (%u) must cover the %u source columns and be a multiple of 8 elements", src_ld, silu_mul ? 2 * k : k);
    if (reinterpret_cast<uintptr_t>(src) % 16 != 0 || reinterpret_cast<uintptr_t>(dst) % 16 != 0)
        return fail(DG_ERR_SHAPE, "src and dst must be 16-byte aligned");
    if (rows == 0) return DG_OK;
    dg::CastParams p;
    p.src = src; p.dst = dst; p.sf = sf;
    p.src_ld = src_ld; p.rows = rows; p.k = k; p.group_rows = rows / groups;
    p.sf_cols = dg_sf_packed_cols(k, gran);
    p.sf_stride = align4(rows / groups);
    p.rule = rule;
    p.live_rows = live_rows;
    // one block per 8 consecutive rows x one 1024-element segment (one warp per row)
    const uint64_t units = static_cast<uint64_t>(ceil_div(rows, 8)) * ceil_div(k, 1024);
    if (units > 0x7FFFFFFFull) return fail(DG_ERR_SHAPE, "matrix too large for one launch");
    const uint32_t blocks = static_cast<uint32_t>(units);
    DG_CUDA(cudaSetDevice(ctx->ordinal));
    if (silu_mul && gran == 32) DG_CUDA(launch(dg::dg_cast_kernel<32, false, true>, blocks, 256, 0, ctx->stream, p));
    else if (silu_mul) DG_CUDA(launch(dg::dg_cast_kernel<128, false, true>, blocks, 256, 0, ctx->stream, p));
    else if (fp4) DG_CUDA(launch(dg::dg_cast_kernel<32, true>, blocks, 256, 0, ctx->stream, p));
    else if (gran == 32) DG_CUDA(launch(dg::dg_cast_kernel<32, false>, blocks, 256, 0, ctx->stream, p));
    else DG_CUDA(launch(dg::dg_cast_kernel<128, false>, blocks, 256, 0, ctx->stream, p));
    return DG_OK;
}

int dg_cast_bf16_to_fp8_sf(dg_ctx* ctx, const uint16_t* src, uint32_t src_ld, uint32_t rows, uint32_t k, uint32_t gran_k,
                           uint32_t num_groups, uint8_t* dst, uint32_t* sf) {
    if (gran_k != 32 && gran_k != 128) return fail(DG_ERR_SHAPE, "gran_k must be 32 or 128");
    if (k == 0 || k % (gran_k * 4) != 0) return fail(DG_ERR_SHAPE, "k must be a multiple of %u for gran %u", gran_k * 4, gran_k);
    return cast_common(ctx, src, src_ld, rows, k, gran_k, num_groups, 0, false, dst, sf);
}

int dg_silu_mul_cast_fp8_sf(dg_ctx* ctx, const uint16_t* gate_up, uint32_t src_ld, uint32_t rows, uint32_t n, uint32_t gran_k,
                            uint32_t num_groups, uint8_t* dst, uint32_t* sf, const uint32_t* live_rows) {
    if (gran_k != 32 && gran_k != 128) return fail(DG_ERR_SHAPE, "gran_k must be 32 or 128");
    if (n == 0 || n % (gran_k * 4) != 0) return fail(DG_ERR_SHAPE, "n must be a multiple of %u for gran %u", gran_k * 4, gran_k);
    return cast_common(ctx, gate_up, src_ld, rows, n, gran_k, num_groups, 0, false, dst, sf, true, live_rows);
}

int dg_cast_bf16_to_fp4_packed_sf(dg_ctx* ctx, const uint16_t* src, uint32_t src_ld, uint32_t rows, uint32_t k, uint32_t num_groups,
                                  int sf_rule, uint8_t* dst, uint32_t* sf) {
    if (k == 0 || k % 128 != 0) return fail(DG_ERR_SHAPE, "fp4 k must be a multiple of 128");
    if (sf_rule != DG_SF_RULE_REFERENCE_CPU && sf_rule != DG_SF_RULE_RANGE_FIT) return fail(DG_ERR_SHAPE, "unknown sf_rule %d", sf_rule);
    return cast_common(ctx, src, src_ld, rows, k, 32, num_groups, sf_rule, true, dst, sf);
}

int dg_transform_sf(dg_ctx* ctx, const float* sf, uint32_t mn, uint32_t sf_k, uint32_t num_batches, float* dst) {
    if (!ctx || !sf || !dst) return fail(DG_ERR_SHAPE, "null argument");
    if (mn == 0 || sf_k == 0 || num_batches == 0) return DG_OK;
    DG_CUDA(cudaSetDevice(ctx->ordinal));
    dim3 grid(ceil_div(align4(mn), 32), ceil_div(sf_k, 32), num_batches);
    DG_CUDA(launch(dg::dg_transpose_sf_kernel, grid, 256, 0, ctx->stream, sf, dst, mn, sf_k, align4(mn)));
    return DG_OK;
}

static int sf_pack_common(dg_ctx* ctx, const float* src, uint32_t src_ld, uint32_t rows, uint32_t k, uint32_t gran, uint32_t groups,
                          uint32_t mode, uint32_t* dst) {
    if (!ctx || !src || !dst) return fail(DG_ERR_SHAPE, "null argument");
    if (gran != 32 && gran != 128) return fail(DG_ERR_SHAPE, "gran_k must be 32 or 128");
    if (groups == 0) groups = 1;
    if (rows % groups != 0) return fail(DG_ERR_SHAPE, "rows (%u) must be a multiple of num_groups (%u)", rows, groups);
    if (rows == 0 || k == 0) return DG_OK;
    dg::SfPackParams p;
    p.src = src; p.dst = dst; p.src_ld = src_ld; p.rows = rows; p.group_rows = rows / groups;
    p.k_blocks = ceil_div(k, gran);
    p.cols = ceil_div(p.k_blocks, 4);
    p.dst_stride = align4(rows / groups);
    p.mode = mode;
    const uint64_t total = static_cast<uint64_t>(rows) * p.cols;
    DG_CUDA(cudaSetDevice(ctx->ordinal));
    DG_CUDA(launch(dg::dg_sf_pack_kernel, static_cast<uint32_t>((total + 255) / 256), 256, 0, ctx->stream, p));
    return DG_OK;
}

int dg_transform_sf1d_packed_ue8m0(dg_ctx* ctx, const float* src, uint32_t src_ld, uint32_t rows, uint32_t k, uint32_t gran_k,
                                   uint32_t num_groups, uint32_t* dst) {
    return sf_pack_common(ctx, src, src_ld, rows, k, gran_k, num_groups, 0, dst);
}
int dg_transform_sf2d_packed_ue8m0(dg_ctx* ctx, const float* src, uint32_t src_ld, uint32_t rows, uint32_t k, uint32_t num_groups,
                                   uint32_t* dst) {
    const uint32_t g = num_groups ? num_groups : 1;
    if (g > 1 && (rows / g) % 128 != 0) return fail(DG_ERR_SHAPE, "2-D SF groups must own whole 128-row tiles (group rows %u)", rows / g);
    return sf_pack_common(ctx, src, src_ld, rows, k, 128, num_groups, 1, dst);
}
int dg_transform_sf_t_packed_ue8m0(dg_ctx* ctx, const float* src, uint32_t rows, uint32_t k, uint32_t gran_k, uint32_t num_groups,
                                   uint32_t* dst) {
    const uint32_t g = num_groups ? num_groups : 1;
    return sf_pack_common(ctx, src, align4(rows / g), rows, k, gran_k, num_groups, 2, dst);
}

int dg_group_ends_from_m_indices(dg_ctx* ctx, const int32_t* m_indices, uint32_t m, uint32_t num_groups, uint32_t* group_ends) {
    if (!ctx || !m_indices || !group_ends) return fail(DG_ERR_SHAPE, "null argument");
    if (num_groups == 0) return DG_OK;
    DG_CUDA(cudaSetDevice(ctx->ordinal));
    return run_group_ends(ctx, m_indices, m, num_groups, group_ends);
}

int dg_unpack_fp4_raw(dg_ctx* ctx, const uint8_t* src, size_t packed_len, uint8_t* dst) {
    if (!ctx || !src || !dst) return fail(DG_ERR_SHAPE, "null argument");
    if (packed_len == 0) return DG_OK;
    if (reinterpret_cast<uintptr_t>(src) % 16 != 0 || reinterpret_cast<uintptr_t>(dst) % 16 != 0)
        return fail(DG_ERR_SHAPE, "src and dst must be 16-byte aligned");
    DG_CUDA(cudaSetDevice(ctx->ordinal));
    const uint64_t threads = (packed_len + 15) / 16;
    DG_CUDA(launch(dg::dg_unpack_fp4_kernel, static_cast<uint32_t>((threads + 255) / 256), 256, 0, ctx->stream, src, dst, packed_len));
    return DG_OK;
}

int dg_debug_expire_wait(dg_ctx* ctx, uint32_t limit_us) {
    if (!ctx) return fail(DG_ERR_SHAPE, "null context");
    if (limit_us == 0 || limit_us > 1000000) return fail(DG_ERR_SHAPE, "limit must be between 1 us and 1 s");
    DG_CUDA(cudaSetDevice(ctx->ordinal));
    dg::dg_expire_wait_kernel<<<1, 32, 0, ctx->stream>>>(ctx->status, static_cast<uint64_t>(limit_us) * 1000ull);
    DG_CUDA(cudaGetLastError());
    return DG_OK;
}

// ------------------------------------------------------------------ MoE row movers
static bool aligned16(const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }

int dg_gather_rows(dg_ctx* ctx, const void* src, size_t src_pitch, const int32_t* idx, uint32_t n_dst, uint32_t row_bytes, void* dst,
                   size_t dst_pitch) {
    if (!ctx || !src || !idx || !dst) return fail(DG_ERR_SHAPE, "null argument");
    if (row_bytes % 16 || src_pitch % 16 || dst_pitch % 16 || !aligned16(src) || !aligned16(dst))
        return fail(DG_ERR_SHAPE, "rows, pitches and base addresses must be multiples of 16 bytes");
    if (n_dst == 0) return DG_OK;
    DG_CUDA(cudaSetDevice(ctx->ordinal));
    DG_CUDA(launch(dg::dg_gather_rows_kernel, ceil_div(n_dst, 8), 256, 0, ctx->stream, static_cast<const uint8_t*>(src), src_pitch, idx, n_dst, row_bytes, static_cast<uint8_t*>(dst), dst_pitch));
    return DG_OK;
}

int dg_moe_pack_rows(dg_ctx* ctx, const uint8_t* data, uint32_t k, const uint32_t* sf, uint32_t sf_stride, uint32_t sf_cols, const int32_t* idx,
                     uint32_t n, uint8_t* out, size_t out_pitch) {
    if (!ctx || !data || !sf || !idx || !out) return fail(DG_ERR_SHAPE, "null argument");
    if (k % 16 || out_pitch % 16 || out_pitch < static_cast<size_t>(k) + 4 * sf_cols || !aligned16(data) || !aligned16(out))
        return fail(DG_ERR_SHAPE, "k and out_pitch must be multiples of 16 and out_pitch >= k + 4 * sf_cols");
    if (n == 0) return DG_OK;
    DG_CUDA(cudaSetDevice(ctx->ordinal));
    DG_CUDA(launch(dg::dg_moe_pack_rows_kernel, ceil_div(n, 8), 256, 0, ctx->stream, data, k, sf, sf_stride, sf_cols, idx, n, out, out_pitch));
    return DG_OK;
}

int dg_moe_unpack_rows(dg_ctx* ctx, const uint8_t* in, size_t in_pitch, uint32_t k, uint32_t sf_cols, const int32_t* idx, uint32_t n_dst,
                       uint8_t* dst_data, uint32_t* dst_sf, uint32_t dst_sf_stride) {
    if (!ctx || !in || !idx || !dst_data || !dst_sf) return fail(DG_ERR_SHAPE, "null argument");
    if (k % 16 || in_pitch % 16 || in_pitch < static_cast<size_t>(k) + 4 * sf_cols || !aligned16(in) || !aligned16(dst_data))
        return fail(DG_ERR_SHAPE, "k and in_pitch must be multiples of 16 and in_pitch >= k + 4 * sf_cols");
    if (dst_sf_stride < n_dst) return fail(DG_ERR_SHAPE, "scale stride smaller than the row count");
    if (n_dst == 0) return DG_OK;
    DG_CUDA(cudaSetDevice(ctx->ordinal));
    DG_CUDA(launch(dg::dg_moe_unpack_rows_kernel, ceil_div(n_dst, 8), 256, 0, ctx->stream, in, in_pitch, k, sf_cols, idx, n_dst, dst_data, dst_sf, dst_sf_stride));
    return DG_OK;
}

int dg_moe_combine(dg_ctx* ctx, const uint16_t* rows, size_t pitch, const int32_t* pos, const float* weights, uint32_t tokens, uint32_t topk,
                   uint32_t n, uint16_t* out, size_t out_pitch) {
    if (!ctx || !rows || !pos || !weights || !out) return fail(DG_ERR_SHAPE, "null argument");
    if (n % 8 || pitch % 8 || out_pitch % 8 || !aligned16(rows) || !aligned16(out)) return fail(DG_ERR_SHAPE, "n and pitches must be multiples of 8 elements");
    if (tokens == 0 || n == 0) return DG_OK;
    DG_CUDA(cudaSetDevice(ctx->ordinal));
    const uint64_t threads = static_cast<uint64_t>(tokens) * (n / 8);
    DG_CUDA(launch(dg::dg_moe_combine_kernel, static_cast<uint32_t>((threads + 255) / 256), 256, 0, ctx->stream, rows, pitch, pos, weights, tokens, topk, n, out, out_pitch));
    return DG_OK;
}

// ------------------------------------------------------------------------------------------------
// Buffers other processes' GPUs can map, and the expert-parallel exchange over them
// ------------------------------------------------------------------------------------------------
int dg_peer_alloc(dg_ctx* ctx, size_t bytes, void** ptr, unsigned char* handle64) {
    if (!ctx || !ptr || bytes == 0) return fail(DG_ERR_SHAPE, "null argument or zero size");
    static_assert(sizeof(cudaIpcMemHandle_t) == DG_PEER_HANDLE_BYTES, "handle size");
    DG_CUDA(cudaSetDevice(ctx->ordinal));
    void* p = nullptr;
    DG_CUDA(cudaMalloc(&p, bytes));
    if (handle64 != nullptr) {
        cudaIpcMemHandle_t h;
        const cudaError_t e = cudaIpcGetMemHandle(&h, p);
        if (e != cudaSuccess) {
            cudaFree(p);
            return fail(DG_ERR_DRIVER, "cudaIpcGetMemHandle: %s", cudaGetErrorString(e));
        }
        memcpy(handle64, &h, sizeof(h));
    }
    *ptr = p;
    return DG_OK;
}

int dg_peer_open(dg_ctx* ctx, const unsigned char* handle64, void** ptr) {
    if (!ctx || !ptr || !handle64) return fail(DG_ERR_SHAPE, "null argument");
    DG_CUDA(cudaSetDevice(ctx->ordinal));
    cudaIpcMemHandle_t h;
    memcpy(&h, handle64, sizeof(h));
    DG_CUDA(cudaIpcOpenMemHandle(ptr, h, cudaIpcMemLazyEnablePeerAccess));
    return DG_OK;
}

int dg_peer_close(dg_ctx* ctx, void* ptr) {
    if (!ctx || !ptr) return fail(DG_ERR_SHAPE, "null argument");
    DG_CUDA(cudaSetDevice(ctx->ordinal));
    DG_CUDA(cudaIpcCloseMemHandle(ptr));
    return DG_OK;
}

int dg_peer_free(dg_ctx* ctx, void* ptr) {
    if (!ctx || !ptr) return fail(DG_ERR_SHAPE, "null argument");
    DG_CUDA(cudaSetDevice(ctx->ordinal));
    DG_CUDA(cudaFree(ptr));
    return DG_OK;
}

size_t dg_ep_block_hist_words(uint32_t pairs, uint32_t num_experts) {
    return static_cast<size_t>(ceil_div(pairs, dg::kEpChunk)) * num_experts;
}

int dg_ep_count(dg_ctx* ctx, const int32_t* expert_of_pair, uint32_t pairs, uint32_t num_experts, int32_t* local_rank, uint32_t* block_hist,
                uint32_t* counts) {
    if (!ctx || !expert_of_pair || !local_rank || !block_hist || !counts) return fail(DG_ERR_SHAPE, "null argument");
    if (num_experts == 0 || num_experts > 8192) return fail(DG_ERR_SHAPE, "num_experts must be in [1, 8192]");
    DG_CUDA(cudaSetDevice(ctx->ordinal));
    const uint32_t chunks = ceil_div(pairs, dg::kEpChunk);
    // Up to four chunks (a decode step of 128 tokens, top-8) one block is as fast as the two launches or 2 us faster; eight take it 2 us longer.
    if (chunks <= 4) {
        DG_CUDA(launch(dg::dg_ep_rank_pairs_kernel<true>, 1, dg::kEpChunk, num_experts * sizeof(uint32_t), ctx->stream, expert_of_pair, pairs, num_experts, local_rank,
                       block_hist, counts));
        return DG_OK;
    }
    DG_CUDA(launch(dg::dg_ep_rank_pairs_kernel<false>, chunks, dg::kEpChunk, num_experts * sizeof(uint32_t), ctx->stream, expert_of_pair, pairs, num_experts, local_rank,
                   block_hist, counts));
    DG_CUDA(launch(dg::dg_ep_block_scan_kernel, ceil_div(num_experts, 8), 256, 0, ctx->stream, block_hist, chunks, num_experts, counts));
    return DG_OK;
}

int dg_ep_layout(dg_ctx* ctx, const uint32_t* all_counts, uint32_t world, uint32_t rank, uint32_t num_experts, uint32_t alignment,
                 uint32_t capacity, uint32_t slot_rows, uint32_t* pair_base, uint32_t* group_ends, uint32_t* totals) {
    if (!ctx || !all_counts || !pair_base || !group_ends || !totals) return fail(DG_ERR_SHAPE, "null argument");
    if (world == 0 || world > 1024 || rank >= world || num_experts == 0 || num_experts > 4096 || num_experts % world != 0)
        return fail(DG_ERR_SHAPE, "need 1 <= world <= 1024, rank < world, num_experts <= 4096 and a multiple of world");
    if (alignment == 0) return fail(DG_ERR_SHAPE, "alignment must be positive");
    DG_CUDA(cudaSetDevice(ctx->ordinal));
    DG_CUDA(launch(dg::dg_ep_layout_kernel, 1, 1024, 3 * num_experts * sizeof(uint32_t), ctx->stream, all_counts, world, rank, num_experts, alignment, capacity, slot_rows, pair_base, group_ends, totals));
    return DG_OK;
}

// Pieces a row of `steps` warp loads is cut into, one warp each: of seven loads where that gives enough warps, of fewer down to one
// where it does not.
static uint32_t row_segments(uint32_t rows, uint32_t steps, uint64_t enough) {
    if (steps == 0) return 1;
    uint32_t per = dg::kEpPieceLoads;
    while (per > 1 && static_cast<uint64_t>(rows) * ceil_div(steps, per) < enough) --per;
    return ceil_div(steps, per);
}
// Eight pieces per block, those of a row next to each other; max_blocks (0: no bound) bounds the grid.
static uint32_t piece_blocks(uint64_t pieces, uint32_t max_blocks) {
    const uint32_t blocks = static_cast<uint32_t>((pieces + 7) / 8);
    return max_blocks != 0 && blocks > max_blocks ? max_blocks : blocks;
}

int dg_ep_dispatch(dg_ctx* ctx, const int32_t* expert_of_pair, const int32_t* local_rank, const uint32_t* block_base, const uint32_t* pair_base,
                   uint32_t pairs, uint32_t topk, uint32_t num_experts, uint32_t world, const uint8_t* data, uint32_t k, const uint32_t* sf,
                   uint32_t sf_stride, uint32_t sf_cols, void* const* peer_data, void* const* peer_sf, uint32_t peer_sf_stride,
                   uint32_t capacity, uint32_t slot_rows, int32_t* pos_of_pair, uint32_t max_blocks) {
    if (!ctx || !expert_of_pair || !local_rank || !block_base || !pair_base || !data || !sf || !peer_data || !peer_sf || !pos_of_pair)
        return fail(DG_ERR_SHAPE, "null argument");
    if (k % 16 || !aligned16(data)) return fail(DG_ERR_SHAPE, "k and the token rows must be multiples of 16 bytes");
    if (topk == 0 || pairs % topk != 0) return fail(DG_ERR_SHAPE, "pairs (%u) must be tokens x topk (%u)", pairs, topk);
    if (world == 0 || num_experts % world != 0) return fail(DG_ERR_SHAPE, "num_experts (%u) must be a multiple of world (%u)", num_experts, world);
    if (peer_sf_stride < (slot_rows ? slot_rows : capacity)) return fail(DG_ERR_SHAPE, "arena scale stride smaller than the rows it indexes");
    if (pairs == 0) return DG_OK;
    dg::EpDispatchParams p;
    p.expert_of_pair = expert_of_pair; p.local_rank = local_rank; p.block_base = block_base; p.pair_base = pair_base;
    p.data = data; p.sf = sf;
    p.peer_data = reinterpret_cast<uint8_t* const*>(peer_data); p.peer_sf = reinterpret_cast<uint32_t* const*>(peer_sf);
    p.pos_of_pair = pos_of_pair;
    p.pairs = pairs; p.topk = topk; p.k = k; p.sf_cols = sf_cols; p.sf_stride = sf_stride; p.peer_sf_stride = peer_sf_stride;
    p.num_experts = num_experts; p.experts_per_rank = num_experts / world; p.capacity = capacity; p.slot_rows = slot_rows;
    DG_CUDA(cudaSetDevice(ctx->ordinal));
    // A warp per pair and piece while that makes at most 14 warps per SM, pieces as short as 7 warps per SM allow (top-8, both ways of work
    // side by side: 128 tokens of 2048 / 4096 / 5120 / 7168 bytes 2.56 / 2.96 / 3.15 / 3.47 us against 3.13 / 3.20 / 3.38 / 3.41 with a
    // warp per token and piece; 256 tokens of 4096 / 5120 / 7168 bytes 3.73 / 4.06 / 4.86 against 3.57 / 3.89 / 4.59; with top-1 and
    // top-2 within 4 % of each other).  Beyond, pieces of seven loads where they make six warps per SM, else shorter ones (256 tokens of
    // 7168 bytes: four pieces 4.59 us, three 5.23, two 6.66; 512 of 2048 bytes: two 3.53, one 4.61).
    const uint32_t loads = k == 0 ? 1 : ceil_div(k, 512), tokens = pairs / topk, sms = static_cast<uint32_t>(ctx->num_sms);
    if (static_cast<uint64_t>(pairs) * ceil_div(loads, dg::kEpPieceLoads) <= 14ull * sms) {
        p.piece_loads = dg::kEpPieceLoads;
        while (p.piece_loads > 1 && static_cast<uint64_t>(pairs) * ceil_div(loads, p.piece_loads - 1) <= 7ull * sms) --p.piece_loads;
        p.pieces = ceil_div(loads, p.piece_loads);
        p.piece_loads = ceil_div(loads, p.pieces);
        dim3 grid(ceil_div(pairs, 8), p.pieces, 1);
        if (max_blocks != 0) {
            if (grid.y > max_blocks) grid.y = max_blocks;
            if (grid.x > max_blocks / grid.y) grid.x = max_blocks / grid.y;
        }
        DG_CUDA(launch(dg::dg_ep_dispatch_pairs_kernel, grid, 256, 0, ctx->stream, p));
        return DG_OK;
    }
    p.pieces = row_segments(tokens, loads, 6ull * sms);
    p.piece_loads = ceil_div(loads, p.pieces);
    const uint64_t units = static_cast<uint64_t>(tokens) * ceil_div(topk, 32) * p.pieces;
    if (units > 0xFFFFFFFFull) return fail(DG_ERR_SHAPE, "tokens x pieces of a row must fit 32 bits");
    DG_CUDA(launch(dg::dg_ep_dispatch_tokens_kernel, piece_blocks(units, max_blocks), 256, 0, ctx->stream, p));
    return DG_OK;
}

int dg_ep_combine(dg_ctx* ctx, const int32_t* expert_of_pair, const int32_t* pos_of_pair, const float* weights, uint32_t tokens, uint32_t topk,
                  uint32_t num_experts, uint32_t world, const void* const* peer_rows, size_t pitch, uint32_t n, uint16_t* out, size_t out_pitch,
                  uint32_t max_blocks) {
    if (!ctx || !expert_of_pair || !pos_of_pair || !weights || !peer_rows || !out) return fail(DG_ERR_SHAPE, "null argument");
    if (n % 8 || pitch % 8 || out_pitch % 8 || !aligned16(out)) return fail(DG_ERR_SHAPE, "n and pitches must be multiples of 8 elements");
    if (world == 0 || num_experts % world != 0) return fail(DG_ERR_SHAPE, "num_experts (%u) must be a multiple of world (%u)", num_experts, world);
    if (tokens == 0 || n == 0) return DG_OK;
    dg::EpCombineParams p;
    p.expert_of_pair = expert_of_pair; p.pos_of_pair = pos_of_pair; p.weights = weights;
    p.peer_rows = reinterpret_cast<const uint16_t* const*>(peer_rows);
    p.out = out; p.pitch = pitch; p.out_pitch = out_pitch;
    p.tokens = tokens; p.topk = topk; p.n = n; p.experts_per_rank = num_experts / world;
    DG_CUDA(cudaSetDevice(ctx->ordinal));
    if (static_cast<uint64_t>(tokens) * (n / 8) > 0xFFFFFF00ull) return fail(DG_ERR_SHAPE, "tokens x n / 8 must fit 32 bits");
    // Pieces as short as one wave allows (32 warps per SM), of seven steps at most.  A wave and a bit costs two: 1024 tokens x 7168 (28
    // steps), top-8: pieces of 7 steps 24.4 us (one wave), 6: 31.2, 5: 28.1, 4: 25.8, 2: 26.0, 1: 28.2; 512 tokens 4: 10.7, 3: 12.8; x 5120 3:
    // 8.0, 4: 10.2; 256 tokens x 7168 2: 6.1, 1: 6.4.  Beyond one wave seven is within 3 % of the best where it divides the row (8192 x
    // 7168: 166.8, 4: 165.5, 14: 169.8) and within 15 % elsewhere (2048 x 4096, 16 steps: 33.0, 4: 29.1).
    uint32_t steps = 1;
    while (steps < 7 && static_cast<uint64_t>(tokens) * ceil_div(ceil_div(n, 256), steps) > 32ull * ctx->num_sms) ++steps;
    p.segments = ceil_div(ceil_div(n, 256), steps);
    DG_CUDA(launch(dg::dg_ep_combine_kernel, piece_blocks(static_cast<uint64_t>(tokens) * p.segments, max_blocks), 256, 0, ctx->stream, p));
    return DG_OK;
}

}  // extern "C"
