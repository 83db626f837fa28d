// extern "C" entry points of libglorcq_b200: argument checks, launch geometry, launches.
// No torch types, no allocation: the caller owns every buffer.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "aux_kernels.cuh"
#include "skinny_mm.cuh"
#include "stream_mm.cuh"
#include "tc_mm.cuh"
#include "tc_ps.cuh"
#include "xu_mm.cuh"

using namespace glq;

static thread_local int g_last_cuda_error = 0;

#define GLQ_CUDA(call)                                   \
    do {                                                 \
        cudaError_t e__ = (call);                        \
        if (e__ != cudaSuccess) {                        \
            g_last_cuda_error = (int)e__;                \
            return GLQ_ERR_CUDA;                         \
        }                                                \
    } while (0)

static inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
static inline bool aligned_to(const void* p, uintptr_t a) { return (reinterpret_cast<uintptr_t>(p) & (a - 1)) == 0; }
static inline int cdiv(int a, int b) { return (a + b - 1) / b; }
static inline int pow2ceil(int v) {
    int p = 1;
    while (p < v) p <<= 1;
    return p;
}

extern "C" int glq_version(void) { return 100; }

extern "C" const char* glq_status_string(int status) {
    switch (status) {
        case GLQ_OK: return "ok";
        case GLQ_ERR_ARG: return "invalid argument (null pointer or inconsistent size)";
        case GLQ_ERR_ALIGN: return "pointer or leading dimension not aligned to 16 bytes";
        case GLQ_ERR_UNSUPPORTED: return "shape, group size or rank not supported by the sm_100a kernels";
        case GLQ_ERR_CUDA: return "CUDA call failed (see glq_last_cuda_error)";
        case GLQ_ERR_WORKSPACE: return "workspace too small (or, for the *_static entry point, the problem needs more scratch than the fixed array holds)";
        default: return "unknown status";
    }
}

extern "C" int glq_last_cuda_error(void) { return g_last_cuda_error; }

// ---------------------------------------------------------------------------------------------
// tiled layout sizes
// ---------------------------------------------------------------------------------------------
static inline int tile_fmt(int fmt) { return fmt == GLQ_FMT_Q3 ? GLQ_FMT_Q4 : fmt; }
static inline int fmt_kb(int fmt) { return (fmt == GLQ_FMT_Q2 || fmt == GLQ_FMT_T2) ? 128 : 64; }
static inline int dest_pairs(int n_rows, int count) { return (cdiv(n_rows, 16) * count + 1) / 2; }

extern "C" size_t glq_tiled_bytes(int fmt, int n_rows, int K, int count) {
    fmt = tile_fmt(fmt);
    if (fmt < 0 || fmt > 2 || n_rows <= 0 || K <= 0 || count < 1 || count > 2) return 0;
    return (size_t)dest_pairs(n_rows, count) * cdiv(K, fmt_kb(fmt)) * 2 * block_bytes_of(fmt);
}
extern "C" size_t glq_sv_bytes(int n_rows, int rank, int count) {
    if (n_rows <= 0 || rank <= 0 || count < 1 || count > 2) return 0;
    return (size_t)dest_pairs(n_rows, count) * cdiv(rank, 64) * 4096;
}
extern "C" size_t glq_rows_f32_count(int n_rows, int count) {
    if (n_rows <= 0 || count < 1 || count > 2) return 0;
    return (size_t)dest_pairs(n_rows, count) * 32;
}
extern "C" size_t glq_tiled_f16_bytes(int N, int K) {
    if (N <= 0 || K <= 0) return 0;
    return (size_t)cdiv(N, 16) * cdiv(K, 64) * 4 * 512;
}

// ---------------------------------------------------------------------------------------------
// launch geometry of the skinny kernel (shared by the workspace query and the launcher)
// ---------------------------------------------------------------------------------------------
struct Geometry {
    int nw, ntt, ntc, nkb, group_blocks, tile_groups, tgn, sk, kb_per_split, kb_chunk, max_passes;
    size_t smem, n_counters, scratch_bytes;
};

// SM count of the current device (cached per device: the planned splits follow the GPU the call runs on)
static int num_sms() {
    static int sms[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    if (sms[dev] == 0) {
        int v = 0;
        if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) v = 148;
        sms[dev] = v;
    }
    return sms[dev];
}

static int plan_geometry(int fmt, int epilogue, int N, int K, int group_size, int n_problems, int max_rows,
                         bool allow_split, Geometry* out) {
    fmt = tile_fmt(fmt);
    if (fmt < 0 || fmt > 3 || N <= 0 || K <= 0 || n_problems <= 0 || max_rows <= 0) return GLQ_ERR_ARG;
    Geometry g{};
    g.nw = (epilogue == GLQ_EPI_SWIGLU) ? 2 : 1;
    if (g.nw == 2 && fmt == GLQ_FMT_F16) return GLQ_ERR_UNSUPPORTED;
    const int kb = fmt_kb(fmt);
    g.nkb = cdiv(K, kb);
    g.group_blocks = 1;
    if (fmt == GLQ_FMT_Q2 || fmt == GLQ_FMT_Q4) {
        if (group_size <= 0 || group_size % kb != 0) return GLQ_ERR_UNSUPPORTED;
        g.group_blocks = group_size / kb;
    }
    if (max_rows <= 8) g.ntt = 1;
    else if (max_rows <= 16 || g.nw == 2) g.ntt = 2;
    else g.ntt = 4;
    g.ntc = g.ntt == 1 ? std::max(2, pow2ceil(max_rows)) : 8 * g.ntt;
    g.max_passes = cdiv(max_rows, 8 * g.ntt);
    g.tile_groups = cdiv(cdiv(N, kRowTile), kRW);

    // CTA-level k split: fill the machine about twice over while every warp keeps >= 1 k block
    const long ctas = (long)n_problems * g.tile_groups;
    const int units = cdiv(g.nkb, g.group_blocks);  // split granularity = one scale group
    int sk = 1;
    if (allow_split) {
        const long want = 2L * num_sms();
        if (ctas < want) sk = (int)std::min<long>((want + ctas - 1) / ctas, std::max(1, units / kKW));
    }
    g.kb_per_split = cdiv(units, sk) * g.group_blocks;
    g.sk = cdiv(g.nkb, g.kb_per_split);
    // shared memory holds kb_chunk blocks of staged activations at a time (two CTAs per SM)
    const size_t per_kb = skinny_smem_bytes(fmt, 1, g.ntc, g.nw, g.ntt) - skinny_smem_bytes(fmt, 0, g.ntc, g.nw, g.ntt);
    const size_t fixed = skinny_smem_bytes(fmt, 0, g.ntc, g.nw, g.ntt);
    const size_t smem_cap = 100 * 1024;
    g.kb_chunk = (int)std::max<size_t>(1, std::min<size_t>((size_t)std::min(g.kb_per_split, g.nkb),
                                                             (smem_cap - fixed) / per_kb));
    g.smem = skinny_smem_bytes(fmt, g.kb_chunk, g.ntc, g.nw, g.ntt);
    // rows too long to stage at once are staged again by every CTA: four tile groups share a staging when that still leaves
    // a CTA for every slot
    g.tgn = ((fmt == GLQ_FMT_Q2 || fmt == GLQ_FMT_Q4) && g.nw == 1 && g.ntt == 1 && g.sk == 1 && g.kb_chunk < g.nkb &&
             (long)n_problems * g.tile_groups >= 4L * 2 * num_sms()) ? 4 : 1;
    const size_t tiles = (size_t)n_problems * g.tile_groups * g.max_passes;
    g.n_counters = g.sk > 1 ? tiles : 0;
    g.scratch_bytes = g.sk > 1 ? tiles * g.sk * (size_t)(kRW * g.nw * g.ntt * 32) * sizeof(float4) : 0;
    *out = g;
    return GLQ_OK;
}

static thread_local bool t_dependent_launch = false;
static thread_local bool t_share_sm = false;
template <int FMT, int NW, int NTT, bool RM, int TGN = 1>
static int launch_one(const SkinnyParams& p, int grid, size_t smem, cudaStream_t st) {
    auto kern = skinny_kernel<FMT, NW, NTT, RM, TGN>;
    if (smem > 48 * 1024) {
        static SmemLimit limit;
        GLQ_CUDA(reserve_smem(reinterpret_cast<const void*>(kern), limit, smem));
    }
    GLQ_CUDA(launch_kernel(t_dependent_launch, kern, dim3(grid), dim3(kThreads), smem, st, p));
    return GLQ_OK;
}

template <int FMT, bool RM>
static int launch_fmt(const SkinnyParams& p, const Geometry& g, int grid, cudaStream_t st) {
    if (g.nw == 2) {
        if constexpr (FMT == GLQ_FMT_F16 || RM) {
            return GLQ_ERR_UNSUPPORTED;
        } else {
            if (g.ntt == 1) return launch_one<FMT, 2, 1, false>(p, grid, g.smem, st);
            return launch_one<FMT, 2, 2, false>(p, grid, g.smem, st);
        }
    }
    if constexpr (!RM && (FMT == GLQ_FMT_Q2 || FMT == GLQ_FMT_Q4))
        if (g.tgn == 4) return launch_one<FMT, 1, 1, false, 4>(p, grid, g.smem, st);
    if (g.ntt == 1) return launch_one<FMT, 1, 1, RM>(p, grid, g.smem, st);
    if (g.ntt == 2) return launch_one<FMT, 1, 2, RM>(p, grid, g.smem, st);
    return launch_one<FMT, 1, 4, RM>(p, grid, g.smem, st);
}

static int launch_skinny(int fmt, bool rowmajor, const SkinnyParams& p, const Geometry& g, int n_problems,
                         cudaStream_t st) {
    const long grid = (long)n_problems * cdiv(g.tile_groups, g.tgn) * g.sk;
    if (grid <= 0 || grid > 0x7fffffffL) return GLQ_ERR_UNSUPPORTED;
    if (rowmajor) {
        if (fmt != GLQ_FMT_T2) return GLQ_ERR_UNSUPPORTED;
        return launch_fmt<GLQ_FMT_T2, true>(p, g, (int)grid, st);
    }
    switch (tile_fmt(fmt)) {
        case GLQ_FMT_Q2: return launch_fmt<GLQ_FMT_Q2, false>(p, g, (int)grid, st);
        case GLQ_FMT_Q4: return launch_fmt<GLQ_FMT_Q4, false>(p, g, (int)grid, st);
        case GLQ_FMT_T2: return launch_fmt<GLQ_FMT_T2, false>(p, g, (int)grid, st);
        case GLQ_FMT_F16: return launch_fmt<GLQ_FMT_F16, false>(p, g, (int)grid, st);
    }
    return GLQ_ERR_ARG;
}

static void fill_geometry(SkinnyParams& p, const Geometry& g) {
    p.tile_groups = g.tile_groups;
    p.sk = g.sk;
    p.kb_per_split = g.kb_per_split;
    p.kb_chunk = g.kb_chunk;
    p.group_blocks = g.group_blocks;
    p.nkb = g.nkb;
    p.ntc = g.ntc;
    p.max_passes = g.max_passes;
}

// ---------------------------------------------------------------------------------------------
// streaming kernel: eligibility, geometry, launch
// ---------------------------------------------------------------------------------------------
struct StreamGeom {
    int i8, nt, ntc, nkb, nw, cb, chunks, sk, kb_per_split, npairs, ips, stages, stage_bytes, swiglu;
    int off_xs, off_ox, off_as, off_ring, off_red;
    size_t smem;
    int grid;
};

static bool stream_disabled() {
    static int v = -1;
    if (v < 0) {
        const char* e = getenv("GLQ_NO_STREAM");
        v = (e && e[0] == '1') ? 1 : 0;
    }
    return v == 1;
}
static bool i8_disabled() {
    static int v = -1;
    if (v < 0) {
        const char* e = getenv("GLQ_NO_I8");
        v = (e && e[0] == '1') ? 1 : 0;
    }
    return v == 1;
}

// k splits of a pair, -1 when the call is not the streaming kernel's.  The splits fix the order of the sums, which deep models
// amplify, so they follow the problem and the memory of CTAs of eight warps alone, whatever form of CTA then runs it:
// enough iterations to give every CTA slot one, as few as fit beside the staged activations (`base` bytes up to the ring) with
// two ring stages and four floats per lane, tile and split for their sums.
static int stream_splits(size_t base, size_t stage, int nt, int npairs, int units, int n_problems) {
    int sk = 1;
    const long want = (long)kStreamCtasPerSm * num_sms();
    while (sk < 8 && (long)n_problems * cdiv(npairs * sk, kWarpsPerCta) < want && units >= 2 * sk) sk *= 2;
    const size_t half = (size_t)110 * 1024, full = (size_t)220 * 1024, ring = 2 * kWarpsPerCta * stage;
    const auto sums = [&](int k) { return k > 1 ? (size_t)2 * kWarpsPerCta * 2 * nt * 32 * 16 : 0; };
    while (sk > 1 && base + sums(sk) + ring > full) sk /= 2;
    if (base + sums(sk) + ring > full) return -1;
    // (fewer splits with two CTAs per SM stream better, as long as every SM still gets work)
    if (sk > 1 && base + sums(sk) + ring > half && base + ring <= half && (long)n_problems * cdiv(npairs, kWarpsPerCta) >= num_sms()) sk = 1;
    return sk;
}

// returns true when the streaming kernel covers this call
// chunks: slots that a problem's rows are cut into
static bool plan_stream(int fmt, int epilogue, int N, int K, int rank, int group_size, int n_problems, int max_rows,
                        StreamGeom* out, int chunks = 1) {
    if (stream_disabled()) return false;
    const bool exact = fmt == GLQ_FMT_Q3;
    fmt = tile_fmt(fmt);
    if (fmt != GLQ_FMT_Q2 && fmt != GLQ_FMT_Q4 && fmt != GLQ_FMT_T2) return false;
    if (N <= 0 || K <= 0 || n_problems <= 0 || max_rows <= 0 || rank < 0 || rank % 16 != 0) return false;
    StreamGeom g{};
    g.swiglu = (epilogue == GLQ_EPI_SWIGLU) ? 1 : 0;
    const int kb = fmt_kb(fmt);
    g.nkb = cdiv(K, kb);
    int group_blocks = 1;
    if (fmt != GLQ_FMT_T2) {
        if (group_size <= 0 || group_size % kb != 0) return false;
        group_blocks = group_size / kb;
    }
    int rows;
    if (max_rows <= 8 && !exact && !i8_disabled()) {
        g.i8 = 1;
        g.nt = max_rows <= 4 ? 1 : 2;
        rows = 4 * g.nt;
        g.ntc = 8 * g.nt;
    } else {
        g.i8 = 0;
        if (max_rows <= 8) g.nt = 1;
        else if (max_rows <= 16) g.nt = 2;
        else if (max_rows <= 32) g.nt = 4;
        else return false;
        rows = 8 * g.nt;
        g.ntc = g.nt == 1 ? std::max(2, pow2ceil(max_rows)) : 8 * g.nt;
    }
    const int ntiles = cdiv(N, kRowTile);
    g.npairs = g.swiglu ? ntiles : cdiv(ntiles, 2);
    const int units = cdiv(g.nkb, group_blocks);      // splits lie on group boundaries
    // shared memory up to the ring, for CTAs of nw warps
    auto base_bytes = [&](int nw) {
        size_t off = (size_t)nw * kMaxStages * 8;
        off = (off + 127) / 128 * 128;
        g.off_xs = (int)off;
        if (g.i8) {
            const int p8 = fmt == GLQ_FMT_Q4 ? 1 : 2;
            off += (size_t)g.nkb * p8 * (2 * rows) * 4 * 16;
            g.off_ox = (int)off;
            off += (size_t)g.nkb * rows * 8;
        } else {
            const int xs_u4 = (fmt == GLQ_FMT_Q4) ? 8 : 16;
            off += (size_t)g.nkb * xs_u4 * g.ntc * 16;
            g.off_ox = (int)off;
            off += (size_t)g.nkb * g.ntc * 8;
        }
        off = (off + 15) / 16 * 16;
        g.off_as = (int)off;
        off += (size_t)(g.swiglu ? 2 : 1) * rows * std::max(rank, 16) * 2;
        return (off + 127) / 128 * 128;
    };
    const size_t stage4 = std::max<size_t>(4 * 2 * block_bytes_of(fmt), 4096);
    g.sk = stream_splits(base_bytes(kWarpsPerCta), stage4, g.nt, g.npairs, units, n_problems);
    if (g.sk < 0) return false;
    g.kb_per_split = cdiv(units, g.sk) * group_blocks;
    // Form of the CTAs: of those that fit beside the staged activations, the one with the fewest rounds of iterations over its
    // slots.  Two CTAs of eight warps per SM are the rule; one of eight leaves room for the sums of many splits; one of
    // sixteen shares its activations among all warps of an SM.  Stages hold four k blocks, two when that is what it takes.
    const int sms = num_sms();
    g.chunks = chunks;
    StreamGeom best{};
    long best_rounds = -1;
    auto consider = [&](int nw, int cb, size_t cap, int slots) {
        const size_t off = base_bytes(nw), stage = (size_t)nw * std::max(cb * 2 * block_bytes_of(fmt), 4096);
        const size_t red = g.sk > 1 ? (size_t)2 * nw * 2 * g.nt * 32 * (g.i8 ? 8 : 16) : 0;
        if (off + red + 2 * stage > cap) return;
        g.nw = nw;
        g.cb = cb;
        g.ips = cdiv(g.npairs * g.sk, nw);
        const long iters = (long)n_problems * chunks * g.ips, rounds = (iters + slots - 1) / slots;      // (ties: the form named first)
        if (best_rounds >= 0 && rounds >= best_rounds) return;
        g.stage_bytes = (int)(stage / nw);
        g.off_ring = (int)off;
        g.stages = std::min((int)((cap - off - red) / stage), kMaxStages);
        g.off_red = (int)(off + g.stages * stage);
        g.smem = g.off_red + red;
        g.grid = (int)std::min<long>(iters, slots);
        best_rounds = rounds;
        best = g;
    };
    const size_t half = (size_t)110 * 1024, full = (size_t)225 * 1024;
    consider(8, 4, half, kStreamCtasPerSm * sms);
    if (g.i8) {
        consider(16, 4, full, sms);
        consider(16, 2, full, sms);
    }
    consider(8, 4, full, sms);
    if (best_rounds < 0) return false;
    *out = best;
    return best.grid > 0;
}

template <int FMT, bool I8, int NT, int NW = 8>
static int launch_stream_one(const StreamParams& sp, const StreamGeom& g, cudaStream_t st) {
    auto kern = stream_kernel<FMT, I8, NT, NW>;
    static SmemLimit limit;
    GLQ_CUDA(reserve_smem(reinterpret_cast<const void*>(kern), limit, g.smem));
    GLQ_CUDA(launch_kernel(sp.a_late || sp.dependent, kern, dim3(g.grid), dim3(NW * 32), g.smem, st, sp));
    return GLQ_OK;
}

template <int FMT>
static int launch_stream_fmt(const StreamParams& sp, const StreamGeom& g, cudaStream_t st) {
    if (g.i8 && g.nw == 16)
        return g.nt == 1 ? launch_stream_one<FMT, true, 1, 16>(sp, g, st) : launch_stream_one<FMT, true, 2, 16>(sp, g, st);
    if (g.i8) {
        if (g.nt == 1) return launch_stream_one<FMT, true, 1>(sp, g, st);
        return launch_stream_one<FMT, true, 2>(sp, g, st);
    }
    if (g.nt == 1) return launch_stream_one<FMT, false, 1>(sp, g, st);
    if (g.nt == 2) return launch_stream_one<FMT, false, 2>(sp, g, st);
    return launch_stream_one<FMT, false, 4>(sp, g, st);
}

template <int FMT, bool I8, int NT, int NW = 8>
static int launch_stream_pair_t(const StreamParams& sp, const StreamGeom& g, const SkinnyParams& xu, int n_xu, cudaStream_t st) {
    auto kern = stream_pair_kernel<FMT, I8, NT, NW>;
    static SmemLimit limit;
    GLQ_CUDA(reserve_smem(reinterpret_cast<const void*>(kern), limit, g.smem));
    GLQ_CUDA(launch_kernel(true, kern, dim3(g.grid + n_xu), dim3(NW * 32), g.smem, st, sp, xu, n_xu));
    return GLQ_OK;
}
template <int FMT>
static int launch_stream_pair_fmt(const StreamParams& sp, const StreamGeom& g, const SkinnyParams& xu, int n_xu, cudaStream_t st) {
    if (!g.i8) {
        if constexpr (FMT == GLQ_FMT_Q4) return launch_stream_pair_t<FMT, false, 1>(sp, g, xu, n_xu, st);
        return GLQ_ERR_UNSUPPORTED;
    }
    if (g.nw == 16)
        return g.nt == 1 ? launch_stream_pair_t<FMT, true, 1, 16>(sp, g, xu, n_xu, st) : launch_stream_pair_t<FMT, true, 2, 16>(sp, g, xu, n_xu, st);
    return g.nt == 1 ? launch_stream_pair_t<FMT, true, 1>(sp, g, xu, n_xu, st) : launch_stream_pair_t<FMT, true, 2>(sp, g, xu, n_xu, st);
}
static int launch_stream_pair(int fmt, const StreamParams& sp, const StreamGeom& g, const SkinnyParams& xu, int n_xu, cudaStream_t st) {
    switch (fmt) {
        case GLQ_FMT_Q2: return launch_stream_pair_fmt<GLQ_FMT_Q2>(sp, g, xu, n_xu, st);
        case GLQ_FMT_Q4: return launch_stream_pair_fmt<GLQ_FMT_Q4>(sp, g, xu, n_xu, st);
        case GLQ_FMT_T2: return launch_stream_pair_fmt<GLQ_FMT_T2>(sp, g, xu, n_xu, st);
    }
    return GLQ_ERR_ARG;
}

// Rows of a chunk when a product with host-known counts is cut into chunks of its rows, the slots of ONE launch of the
// streaming kernel; 0 when it is not.
// 9..32 rows: the integer path stages at most 8 rows (4 when the staged activations of a long reduction leave no room for 8)
// and streams at a multiple of the fp16 path's rate for many rows (a launch per chunk took 17.7 us for each 8 of 16 rows of a
// 4-bit 4096 x 4096); the chunks read the weights at about the same time, once from memory and then from L2.
// (Codebook rows: the fp16 path rounds the levels to fp16.  Error against 64 bits, 9..32 tokens of a 60-expert block behind its
// Hadamard rotation: 0.82-0.83e-3, fp16 path 0.86-0.94e-3; with 1 in 200 input values 50 times larger 0.75-0.80, 0.79-0.84.)
// GLQ_FMT_Q3: any number of rows, on the fp16 path.  8 rows take the integer path's time (4096 x 4096: 16.8 us both), 32 rows of
// 2048 x 2048 21 us instead of 13, 512 rows 111 instead of 210 in launches of 32; error against 64 bits 2.07e-4, the rounding
// of the result, where block fixed point gives 2.12e-4 and 3.3e-4 with 1 in 200 activations 50 times larger.
static int plan_chunks(const glq_mm_args_t* a, StreamGeom* sg) {
    const bool exact = a->fmt == GLQ_FMT_Q3;
    if (a->slot_count || a->slot_offset || a->slot_index || a->max_rows <= 8 || a->fmt == GLQ_FMT_F16 ||
        (!exact && (a->max_rows > 32 || i8_disabled())))
        return 0;
    for (int c : {8, 4})
        if (plan_stream(a->fmt, a->epilogue, a->N, a->K, a->rank, a->group_size, a->n_problems, c, sg, cdiv(a->max_rows, c)) &&
            (exact || sg->i8))
            return c;
    return 0;
}

static void fill_operands(const glq_mm_args_t* a, SkinnyParams& p) {
    p.w = a->w;
    p.table = a->w_table;
    p.sv_slices = cdiv(std::max(a->rank, 1), 64);
    p.slot_index = a->slot_index;
    p.n_slots = a->n_slots;
    p.slot_count = a->slot_count;
    p.slot_offset = a->slot_offset;
    p.entry_row = a->entry_row;
    p.entry_scale = reinterpret_cast<const __half*>(a->entry_scale);
    p.x = reinterpret_cast<const __half*>(a->x);
    p.ldx = a->ldx;
    p.a[0] = reinterpret_cast<const __half*>(a->a0);
    p.a[1] = reinterpret_cast<const __half*>(a->a1);
    p.lda = a->lda;
    p.y = reinterpret_cast<__half*>(a->y);
    p.ldy = a->ldy;
    p.counters = a->counters;
    p.scratch = reinterpret_cast<float4*>(a->workspace);
    p.max_rows = a->max_rows;
    p.rows_stride = a->rows_stride > 0 ? a->rows_stride : a->max_rows;
    p.epilogue = a->epilogue;
    p.x_vec = (aligned16(a->x) && a->ldx % 8 == 0) ? 1 : 0;
}

// xu, n_xu, pair: x.U in the grid's first n_xu blocks and the two counters it meets the product at (stream_pair_kernel)
static int launch_stream(const glq_mm_args_t* a, SkinnyParams& p, const StreamGeom& g, cudaStream_t st, bool a_late = false, bool dependent = false, int cnt_lo = 0,
                         int cnt_hi = 0x7fffffff, const SkinnyParams* xu = nullptr, int n_xu = 0, int* pair = nullptr, int pair_target = 0) {
    const int fmt = a->fmt, N = a->N, K = a->K, rank = a->rank, n_problems = a->n_problems;
    StreamParams sp{};
    sp.cnt_lo = cnt_lo;
    sp.cnt_hi = cnt_hi;
    sp.a_late = (a_late && rank > 0 && p.a[0] != nullptr && !pdl_disabled()) ? 1 : 0;
    sp.dependent = ((dependent || a_late) && !pdl_disabled()) ? 1 : 0;
    p.nkb = g.nkb;
    p.ntc = g.ntc;
    p.kb_chunk = g.nkb;
    p.kb_per_split = g.nkb;
    p.sk = 1;
    sp.b = p;
    sp.N = N;
    sp.K = K;
    sp.rank = rank;
    sp.n_problems = n_problems * g.chunks;
    sp.chunks = g.chunks;
    sp.chunk_rows = p.max_rows;
    sp.prob_rows = a->max_rows;
    sp.swiglu = g.swiglu;
    sp.sk = g.sk;
    sp.sk_log2 = g.sk == 1 ? 0 : (g.sk == 2 ? 1 : (g.sk == 4 ? 2 : 3));
    sp.kb_per_split = g.kb_per_split;
    sp.cb = g.cb;
    sp.npairs = g.npairs;
    sp.ips = g.ips;
    sp.stages = g.stages;
    sp.stage_bytes = g.stage_bytes;
    sp.off_xs = g.off_xs;
    sp.off_ox = g.off_ox;
    sp.off_as = g.off_as;
    sp.off_ring = g.off_ring;
    sp.off_red = g.off_red;
    if (xu) {
        sp.a_late = 1;
        sp.settled = (a->flags & GLQ_MM_WEIGHTS_SETTLED) != 0 ? 1 : 0;
        sp.pair = pair;
        sp.pair_target = pair_target;
        return launch_stream_pair(tile_fmt(fmt), sp, g, *xu, n_xu, st);
    }
    StreamGeom gl = g;
    // a concurrent stream runs grouped products too: two thirds of the CTA slots, so that its kernels find room
    // (measured on the MoE block: the shared expert's branch beside the routed experts')
    if (t_share_sm && gl.grid > 4 * num_sms() / 3) gl.grid = 4 * num_sms() / 3;
    switch (tile_fmt(fmt)) {
        case GLQ_FMT_Q2: return launch_stream_fmt<GLQ_FMT_Q2>(sp, gl, st);
        case GLQ_FMT_Q4: return launch_stream_fmt<GLQ_FMT_Q4>(sp, gl, st);
        case GLQ_FMT_T2: return launch_stream_fmt<GLQ_FMT_T2>(sp, gl, st);
    }
    return GLQ_ERR_ARG;
}

// ---------------------------------------------------------------------------------------------
// tensor-core path (tc_mm.cuh): many rows per problem
// ---------------------------------------------------------------------------------------------
struct TcGeom {
    int tn, nm, nkb, ns, na, tiles_max;    // nm: accumulators of an item of the tensor-memory kernel
    bool hybrid;
    long long tile_bytes;
    size_t xp_bytes;
};
static bool hybrid_disabled() {
    static const bool v = std::getenv("GLQ_NO_HYBRID") != nullptr;
    return v;
}
static bool tc_disabled() {
    static const bool v = std::getenv("GLQ_NO_TC") != nullptr;
    return v;
}
// entries of all problems together: the upper bound that sizes grids and the token operand
static long long total_entries(const glq_mm_args_t* a) {
    const long long stride = a->rows_stride > 0 ? a->rows_stride : a->max_rows;
    const long long total = a->total_rows > 0 ? a->total_rows : (long long)a->n_problems * (a->slot_offset ? a->max_rows : stride);
    return a->slot_offset ? total : std::max(total, (long long)(a->n_problems - 1) * stride + a->max_rows);
}

// Token tile (and, for a plain product, one or two 128-feature tiles per item) of the tcgen05 kernels: the least time of the
// fullest SM, rounds of items x (stages x time of a stage + time around an item), in units of 0.4 us.  Stages measured on
// B200 with packed codes: one accumulator 1 / 1.1 / 1.5 at 64 / 128 / 256 tokens (unpack-bound up to 128), two 1.8 / 2.0;
// around an item five, and two for every 64 tokens of results.  A problem's rows fill ceil(rows / tile) tiles; with device-side
// counts half a tile more than their mean.
static void choose_tile(const glq_mm_args_t* a, long long total, int stages, TcGeom* g) {
    const double rows = (double)total / a->n_problems;
    if (a->fmt == GLQ_FMT_F16) {
        g->tn = rows > 64 ? 128 : 64;
        g->nm = 1;
        return;
    }
    const bool sw = a->epilogue == GLQ_EPI_SWIGLU;
    struct Form { int tn, nm; double stage; };
    static const Form plain[] = {{64, 1, 1.0}, {64, 2, 1.8}, {128, 1, 1.1}, {256, 1, 1.5}}, fused[] = {{64, 2, 1.8}, {128, 2, 2.0}};
    double best = -1;
    for (const Form* f = sw ? fused : plain; f != (sw ? fused + 2 : plain + 4); ++f) {
        const double tiles = a->slot_count ? (rows <= 0.75 * f->tn ? 1.0 : rows / f->tn + 0.5) : std::ceil(rows / f->tn);
        const double items = a->n_problems * tiles * cdiv(a->N, kTcFeat * (sw ? 1 : f->nm));
        const double t = std::ceil(items / num_sms()) * (stages * f->stage + 5 + 2 * (f->tn / 64) * (sw ? 1 : f->nm));
        if (best < 0 || t < best) best = t, g->tn = f->tn, g->nm = f->nm;
    }
}
// true when a tcgen05 kernel takes the call: more rows than the streaming kernel stages
static bool plan_tc(const glq_mm_args_t* a, TcGeom* out) {
    if (tc_disabled() || a->max_rows <= 32) return false;
    if (a->N <= 0 || a->K <= 0 || a->n_problems <= 0 || a->rank < 0 || a->rank % 16 != 0) return false;
    if (a->fmt == GLQ_FMT_Q2 || a->fmt == GLQ_FMT_Q4) {
        if (a->group_size <= 0 || a->group_size % fmt_kb(a->fmt) != 0) return false;
    } else if (a->fmt == GLQ_FMT_F16) {
        if (a->epilogue != GLQ_EPI_LINEAR) return false;
    } else if (a->fmt != GLQ_FMT_T2) {
        return false;
    }
    TcGeom g{};
    const long long total = total_entries(a);
    g.nkb = cdiv(a->K, 128);
    g.ns = a->rank > 0 && a->fmt != GLQ_FMT_F16 ? cdiv(a->rank, 64) : 0;      // (dense weights have no low-rank term)
    g.na = a->epilogue == GLQ_EPI_SWIGLU ? 2 : 1;
    choose_tile(a, total, g.nkb + g.ns, &g);
    const long long tiles = total / g.tn + a->n_problems + 1;
    if (tiles > 65535) return false;
    g.tiles_max = (int)tiles;
    g.tile_bytes = (long long)g.nkb * g.tn * 256 + (long long)g.ns * g.na * g.tn * 128;
    g.xp_bytes = (size_t)g.tiles_max * (size_t)g.tile_bytes + 256;   // + the work-item counter of the persistent kernel
    // device-side row counts with few rows per problem on average: the streaming kernels take the
    // problems with up to 32 rows (one launch for <= 8 rows on the integer path, one for 9..32), this
    // kernel only the larger ones
    g.hybrid = a->slot_count != nullptr && a->fmt != GLQ_FMT_F16 && total / a->n_problems <= 24 && !hybrid_disabled();
    *out = g;
    return true;
}

// dense fp16 weights
template <int TN>
static int launch_tc_t(const TcParams& p, cudaStream_t st) {
    using C = TcCfg<TN>;
    static SmemLimit limit;
    GLQ_CUDA(reserve_smem(reinterpret_cast<const void*>(tc_kernel<TN>), limit, C::SMEM));
    tc_pack_b_kernel<TN><<<dim3(p.tiles_max, p.nkb + p.ns), 256, 0, st>>>(p);
    GLQ_CUDA(cudaGetLastError());
    tc_kernel<TN><<<dim3(p.n_ft, p.tiles_max), kTcThreads, C::SMEM, st>>>(p);
    GLQ_CUDA(cudaGetLastError());
    return GLQ_OK;
}

// packed codes: one CTA per SM over all (token tile, feature tile) items
template <int FMT, int TN, int NM, bool SW>
static int launch_tc_ps_t(TcParams& p, cudaStream_t st) {
    using C = TcPsCfg<FMT, TN, NM, SW>;
    static SmemLimit limit;
    GLQ_CUDA(reserve_smem(reinterpret_cast<const void*>(tc_ps_kernel<FMT, TN, NM, SW>), limit, C::SMEM));
    p.n_ft = cdiv(p.N, kTcFeat * C::NOUT);
    GLQ_CUDA(launch_kernel(p.a_late != 0, tc_pack_b_kernel<TN>, dim3(p.tiles_max, p.nkb + p.ns), dim3(256), 0, st, p));
    const long work = (long)p.n_ft * p.tiles_max;
    // A CTA of this kernel fills its SM.  Where another stream has launches at the same time, no more of them than the rounds of
    // items need: the shared expert's gate|up for 512 tokens has 176 items, two rounds on 148 SMs and on 88, and on the other 60 the
    // routing plan and the routed x.U now run beside it (24-layer prompt 8840 -> 8485 us).
    const long rounds = (work + num_sms() - 1) / num_sms(), grid = t_share_sm ? (work + rounds - 1) / rounds : std::min<long>(work, num_sms());
    GLQ_CUDA(launch_kernel(true, tc_ps_kernel<FMT, TN, NM, SW>, dim3((int)grid), dim3(kPsThreads), C::SMEM, st, p));
    return GLQ_OK;
}
template <int FMT>
static int launch_tc_ps(TcParams& p, const TcGeom& g, bool sw, cudaStream_t st) {
    if (sw) return g.tn == 128 ? launch_tc_ps_t<FMT, 128, 2, true>(p, st) : launch_tc_ps_t<FMT, 64, 2, true>(p, st);
    if (g.tn == 256) return launch_tc_ps_t<FMT, 256, 1, false>(p, st);
    if (g.tn == 128) return launch_tc_ps_t<FMT, 128, 1, false>(p, st);
    return g.nm == 2 ? launch_tc_ps_t<FMT, 64, 2, false>(p, st) : launch_tc_ps_t<FMT, 64, 1, false>(p, st);
}

// operands and alignment facts of the many-row kernels; the geometry is filled in by the launchers
static void fill_tc_operands(const glq_mm_args_t* a, TcParams& p) {
    p.w = a->w;
    p.table = a->w_table;
    p.slot_index = a->slot_index;
    p.n_slots = a->n_slots;
    p.slot_count = a->slot_count;
    p.slot_offset = a->slot_offset;
    p.entry_row = a->entry_row;
    p.entry_scale = reinterpret_cast<const __half*>(a->entry_scale);
    p.x = reinterpret_cast<const __half*>(a->x);
    p.ldx = a->ldx;
    p.a[0] = reinterpret_cast<const __half*>(a->a0);
    p.a[1] = reinterpret_cast<const __half*>(a->a1);
    p.lda = a->lda;
    p.y = reinterpret_cast<__half*>(a->y);
    p.ldy = a->ldy;
    p.n_problems = a->n_problems;
    p.max_rows = a->max_rows;
    p.rows_stride = a->rows_stride > 0 ? a->rows_stride : a->max_rows;
    p.K = a->K;
    p.N = a->N;
    p.rank = (a->a0 != nullptr) ? a->rank : 0;
    p.fmt = a->fmt;
    p.x_vec16 = ((reinterpret_cast<uintptr_t>(a->x) & 15u) == 0 && a->ldx % 8 == 0) ? 1 : 0;
    p.y_vec = ((reinterpret_cast<uintptr_t>(a->y) & 15u) == 0 && a->ldy % 8 == 0 && a->N % 8 == 0) ? 1 : 0;
}

// Dense products with few columns (xu_mm.cuh).  Above 32 rows, where the order of the sums is the tcgen05 kernel's.  Up to 512
// columns: every 64-column slice reads x again (from L2), and a wide W fills the tcgen05 kernel's tiles.  Nothing of x itself
// decides, so that the workspace query, which may come before there is an x, gives the answer of the call.
static bool xu_takes(const glq_mm_args_t* a) {
    return a->fmt == GLQ_FMT_F16 && a->max_rows > 32 && a->N > 0 && a->N <= 512 && a->K > 0 && a->K % 8 == 0 && a->n_problems > 0 &&
           a->epilogue == GLQ_EPI_LINEAR && !a->entry_scale && !(a->rank > 0 && a->a0);
}

template <int NT, bool VEC>
static int launch_xu_t(TcParams& p, const glq_mm_args_t* a, cudaStream_t st) {
    using C = XuCfg<NT>;
    static SmemLimit limit;
    GLQ_CUDA(reserve_smem(reinterpret_cast<const void*>(xu_kernel<NT, VEC>), limit, C::SMEM));
    const bool one = a->n_problems == 1 && !a->slot_offset && !a->n_slots;
    p.tiles_max = one ? cdiv(a->max_rows, C::ROWS) : (int)(total_entries(a) / C::ROWS + a->n_problems + 1);
    // (not beside a launch that left SMs to another stream: CTAs that wait there would take that stream's places, and a routing plan
    // that starts 90 us later costs a 2000-token block 490 us instead of 470)
    // (nor h.U behind the GEMM of many experts: its few CTAs lay two to an SM in the first places that came free; 300 tokens through eight
    // Mixtral-shaped experts, codebook: 691 us against 663)
    const bool beside = !t_share_sm && (!a->n_slots || (a->flags & GLQ_MM_AFTER_KERNEL) != 0);
    GLQ_CUDA(launch_kernel(beside, xu_kernel<NT, VEC>, dim3(p.tiles_max, cdiv(a->N, kXuCols)), dim3(kXuThreads), C::SMEM, st, p));
    return GLQ_OK;
}
static int launch_xu(const glq_mm_args_t* a, cudaStream_t st) {
    if (!a->w_table && !a->w.codes) return GLQ_ERR_ARG;
    TcParams p{};
    fill_tc_operands(a, p);
    p.nkb = cdiv(a->K, 64);
    // 64 rows per CTA read W half as often; 32 where the smaller tiles still leave CTA slots free
    const long long total = total_entries(a), tiles = std::max(total / 32, std::min<long long>(a->n_problems, total));
    if (tiles * cdiv(a->N, kXuCols) > 3 * num_sms()) return p.x_vec16 ? launch_xu_t<8, true>(p, a, st) : launch_xu_t<8, false>(p, a, st);
    return p.x_vec16 ? launch_xu_t<4, true>(p, a, st) : launch_xu_t<4, false>(p, a, st);
}

// output of the x.U product that this thread launched last, if xu_kernel took it and no other product has come since
static thread_local const void* t_xu_out = nullptr;

static int launch_tc(const glq_mm_args_t* a, const TcGeom& g, cudaStream_t st, const void* xu_out, int min_rows = 0) {
    if (!a->workspace || a->workspace_bytes < g.xp_bytes) return GLQ_ERR_WORKSPACE;
    if ((reinterpret_cast<uintptr_t>(a->workspace) & 127u) != 0) return GLQ_ERR_ALIGN;
    TcParams p{};
    fill_tc_operands(a, p);
    p.xp = reinterpret_cast<unsigned char*>(a->workspace);
    p.tile_bytes = g.tile_bytes;
    p.nkb = g.nkb;
    p.ns = p.rank > 0 ? g.ns : 0;
    p.na = g.na;
    p.tiles_max = g.tiles_max;
    p.min_rows = min_rows;
    const bool sw = a->epilogue == GLQ_EPI_SWIGLU;
    p.n_ft = cdiv(a->N, kTcFeat);
    // The pre-pass may run beside x.U only when that is xu_kernel: it uses no workspace, and the caller's workspace is often the
    // same memory for both products.
    p.a_late = (a->flags & GLQ_MM_A_FROM_PREVIOUS_LAUNCH) != 0 && xu_out != nullptr && xu_out == a->a0 && p.ns > 0 && min_rows == 0 &&
                       a->fmt != GLQ_FMT_F16 && !pdl_disabled()
                   ? 1 : 0;
    if (a->fmt == GLQ_FMT_F16) return g.tn == 128 ? launch_tc_t<128>(p, st) : launch_tc_t<64>(p, st);
    p.ts = 1;
    p.tile_ctr = reinterpret_cast<int*>(p.xp + (g.xp_bytes - 256));
    switch (a->fmt) {
        case GLQ_FMT_Q2: return launch_tc_ps<GLQ_FMT_Q2>(p, g, sw, st);
        case GLQ_FMT_Q4: return launch_tc_ps<GLQ_FMT_Q4>(p, g, sw, st);
        case GLQ_FMT_T2: return launch_tc_ps<GLQ_FMT_T2>(p, g, sw, st);
    }
    return GLQ_ERR_UNSUPPORTED;
}

// workspace bytes and arrival counters of a call: one planning for both
struct MmNeeds {
    size_t bytes = 0, counters = 0;
};
static MmNeeds mm_needs(const glq_mm_args_t* a) {
    MmNeeds n;
    TcGeom tg;
    StreamGeom sg;
    Geometry g;
    if (!a || xu_takes(a)) return n;
    if (plan_tc(a, &tg)) {
        n.bytes = tg.xp_bytes;
    } else if (!plan_chunks(a, &sg) &&
               !plan_stream(a->fmt, a->epilogue, a->N, a->K, a->rank, a->group_size, a->n_problems, a->max_rows, &sg) &&
               plan_geometry(a->fmt, a->epilogue, a->N, a->K, a->group_size, a->n_problems, a->max_rows, true, &g) == GLQ_OK) {
        n.bytes = g.scratch_bytes;
        n.counters = g.n_counters;
    }
    return n;
}
extern "C" size_t glq_mm_workspace_bytes(const glq_mm_args_t* a) { return mm_needs(a).bytes; }
extern "C" size_t glq_mm_counters(const glq_mm_args_t* a) { return mm_needs(a).counters; }

extern "C" int glq_grouped_matmul(const glq_mm_args_t* a, void* stream) {
    if (!a || !a->x || !a->y) return GLQ_ERR_ARG;
    if (a->n_problems == 0 || a->max_rows == 0) return GLQ_OK;
    if (a->epilogue != GLQ_EPI_LINEAR && a->epilogue != GLQ_EPI_SWIGLU) return GLQ_ERR_ARG;
    if (a->rank < 0 || a->rank % 16 != 0) return GLQ_ERR_UNSUPPORTED;
    if (a->rank > 0 && (a->a0 || a->a1) && (a->lda % 8 != 0 || !aligned16(a->a0) || !aligned16(a->a1)))
        return GLQ_ERR_ALIGN;
    t_share_sm = (a->flags & GLQ_MM_SHARE_SM) != 0;
    const void* const xu_out = t_xu_out;
    t_xu_out = nullptr;
    if (xu_takes(a)) {
        const int r = launch_xu(a, reinterpret_cast<cudaStream_t>(stream));
        if (r == GLQ_OK) t_xu_out = a->y;
        return r;
    }
    TcGeom tg;
    const bool use_tc = plan_tc(a, &tg);
    if (use_tc && !tg.hybrid) {
        if (!a->w_table && !a->w.codes) return GLQ_ERR_ARG;
        return launch_tc(a, tg, reinterpret_cast<cudaStream_t>(stream), xu_out);
    }
    StreamGeom sg;
    // Row-count classes (device-side counts): slots with <= 8 rows go to the integer path, 9..16 to the
    // fp16 path with two activation tiles, and above that to the tcgen05 kernel when the call may have
    // more than 32 rows per slot, else to the fp16 path with four tiles.  Each class is one launch that
    // skips the slots of the others.
    StreamGeom sg8, sg16;
    const int chunk = use_tc ? 0 : plan_chunks(a, &sg);
    const int cap = chunk ? chunk : use_tc ? 16 : std::min(a->max_rows, 32);
    // (more rows than a slot of the streaming kernel holds, and no other kernel for them: the general one)
    const bool use_stream = chunk || ((use_tc || a->max_rows <= cap) &&
                                      plan_stream(a->fmt, a->epilogue, a->N, a->K, a->rank, a->group_size, a->n_problems, cap, &sg));
    const bool classes = use_stream && a->slot_count != nullptr && a->max_rows > 8 && !hybrid_disabled();
    const bool split8 = classes && plan_stream(a->fmt, a->epilogue, a->N, a->K, a->rank, a->group_size, a->n_problems, 8, &sg8) &&
                        sg8.i8;
    const bool split16 = classes && cap > 16 &&
                         plan_stream(a->fmt, a->epilogue, a->N, a->K, a->rank, a->group_size, a->n_problems, 16, &sg16);
    if (use_tc && !use_stream) {
        if (!a->w_table && !a->w.codes) return GLQ_ERR_ARG;
        return launch_tc(a, tg, reinterpret_cast<cudaStream_t>(stream), nullptr);
    }
    Geometry g{};
    int rc = use_stream ? GLQ_OK
                        : plan_geometry(a->fmt, a->epilogue, a->N, a->K, a->group_size, a->n_problems, a->max_rows,
                                        true, &g);
    if (rc != GLQ_OK) return rc;
    if (!use_stream && g.sk > 1) {
        if (!a->workspace || a->workspace_bytes < g.scratch_bytes) return GLQ_ERR_WORKSPACE;
        if (!a->counters || a->n_counters < g.n_counters) return GLQ_ERR_WORKSPACE;
        if (!aligned16(a->workspace)) return GLQ_ERR_ALIGN;
    }
    if (!a->w_table && !a->w.codes) return GLQ_ERR_ARG;

    SkinnyParams p{};
    fill_operands(a, p);
    if (chunk) p.max_rows = chunk;
    if (use_stream) {
        cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
        const bool a_late = (a->flags & GLQ_MM_A_FROM_PREVIOUS_LAUNCH) != 0, dep = (a->flags & GLQ_MM_AFTER_KERNEL) != 0;
        if (!split8 && !split16 && !use_tc) return launch_stream(a, p, sg, st, a_late, dep);
        // one launch per class; only the first may depend programmatically on the producer of x.U (the
        // later ones start after it has finished)
        int lo = 0;
        bool first = true;
        auto one = [&](const StreamGeom& gg, int rows, int hi) {
            SkinnyParams pp = p;
            pp.max_rows = rows;
            const int r2 = launch_stream(a, pp, gg, st, first && a_late, first && dep, lo, hi);
            first = false;
            lo = hi;
            return r2;
        };
        if (split8 && (rc = one(sg8, 8, 8)) != GLQ_OK) return rc;
        if (split16 && (rc = one(sg16, 16, 16)) != GLQ_OK) return rc;
        if ((rc = one(sg, cap, cap)) != GLQ_OK) return rc;
        if (use_tc) return launch_tc(a, tg, st, nullptr, cap);
        return GLQ_OK;
    }
    fill_geometry(p, g);
    t_dependent_launch = (a->flags & (GLQ_MM_AFTER_KERNEL | GLQ_MM_A_FROM_PREVIOUS_LAUNCH)) != 0;
    rc = launch_skinny(a->fmt, false, p, g, a->n_problems, reinterpret_cast<cudaStream_t>(stream));
    t_dependent_launch = false;
    return rc;
}

// x.U (u) and the product that adds its low-rank term (m): one launch where both are small enough to be resident together, two
// otherwise.  One launch: at most 8 rows with counts that the host knows, the streaming kernel for m, the general kernel without
// tile groups for u, a CTA slot for every block of both (where the product fills the slots, blocks behind x.U's would start late
// and the launch that is saved is a small part), and two counters more than u needs.  It reads weights before it has waited
// for the launch ahead only on the caller's word that none writes them there: one row of 4-bit 4096 x 4096, back to back, 7.7 us a
// call, 8.9 without; 8 rows of 2-bit 5632 x 2048 8.8 and 10.1; a token of 24 layers 1434 and 1475.
constexpr size_t kPairCounters = 2;
static int matmul_pair(const glq_mm_args_t* u, const glq_mm_args_t* m, void* stream) {
    StreamGeom sg;
    Geometry g;
    const bool known = !m->slot_index && !m->n_slots && !m->slot_count && !m->slot_offset && !u->slot_index && !u->n_slots && !u->slot_count &&
                       !u->slot_offset;
    if (known && !pdl_disabled() && m->max_rows <= 8 && u->max_rows == m->max_rows && u->n_problems == m->n_problems && m->n_problems > 0 && u->fmt == GLQ_FMT_F16 &&
        u->epilogue == GLQ_EPI_LINEAR && m->epilogue == GLQ_EPI_LINEAR && u->rank == 0 && u->K == m->K && u->y == m->a0 && m->a0 && m->rank > 0 &&
        m->rank % 16 == 0 && m->lda % 8 == 0 && aligned16(m->a0) && u->x && m->x && m->y && (u->w_table || u->w.codes) && (m->w_table || m->w.codes) &&
        !u->entry_scale &&
        plan_stream(m->fmt, m->epilogue, m->N, m->K, m->rank, m->group_size, m->n_problems, m->max_rows, &sg) &&
        (sg.i8 || (m->fmt == GLQ_FMT_Q3 && sg.nt == 1 && sg.nw == 8)) &&
        plan_geometry(GLQ_FMT_F16, GLQ_EPI_LINEAR, u->N, u->K, 0, u->n_problems, u->max_rows, true, &g) == GLQ_OK && g.ntt == 1 && g.smem <= sg.smem) {
        const long n_xu = (long)u->n_problems * g.tile_groups * g.sk;
        const long slots = (long)num_sms() * (sg.nw == 8 && sg.smem <= 110 * 1024 ? kStreamCtasPerSm : 1);
        const bool scratch = (g.scratch_bytes == 0 || (u->workspace && u->workspace_bytes >= g.scratch_bytes && aligned16(u->workspace))) && u->counters &&
                             u->n_counters >= g.n_counters + kPairCounters;
        if (n_xu + sg.grid <= slots && scratch) {
            SkinnyParams xp{}, p{};
            fill_operands(u, xp);
            fill_geometry(xp, g);
            fill_operands(m, p);
            t_xu_out = nullptr;
            return launch_stream(m, p, sg, reinterpret_cast<cudaStream_t>(stream), false, false, 0, 0x7fffffff, &xp, (int)n_xu,
                                 u->counters + g.n_counters, u->n_problems * cdiv(u->N, kRowTile));
        }
    }
    const int rc = glq_grouped_matmul(u, stream);
    return rc != GLQ_OK ? rc : glq_grouped_matmul(m, stream);
}
extern "C" int glq_grouped_matmul_pair(const glq_mm_args_t* xu, const glq_mm_args_t* mm, void* stream) {
    if (!xu || !mm) return GLQ_ERR_ARG;
    return matmul_pair(xu, mm, stream);
}

// ---------------------------------------------------------------------------------------------
// glq_linear_forward
// ---------------------------------------------------------------------------------------------
static void linear_args(int fmt, int group_size, const glq_weight_t* w, int B, glq_mm_args_t* m) {
    std::memset(m, 0, sizeof(*m));
    m->fmt = fmt;
    m->group_size = group_size;
    m->epilogue = GLQ_EPI_LINEAR;
    m->n_problems = 1;
    m->max_rows = B;
    m->rows_stride = B;
    m->N = w->N;
    m->K = w->K;
    m->rank = w->rank;
    m->w = *w;
}
static void xu_args(const glq_weight_t* w, const void* ut, int B, glq_mm_args_t* m) {
    std::memset(m, 0, sizeof(*m));
    m->fmt = GLQ_FMT_F16;
    m->epilogue = GLQ_EPI_LINEAR;
    m->n_problems = 1;
    m->max_rows = B;
    m->rows_stride = B;
    m->N = w->rank;
    m->K = w->K;
    m->w.codes = ut;
    m->w.N = w->rank;
    m->w.K = w->K;
}
static inline size_t up256(size_t v) { return (v + 255) / 256 * 256; }

extern "C" size_t glq_linear_workspace_bytes(int fmt, int group_size, const glq_weight_t* w, int B) {
    if (!w || B <= 0) return 0;
    glq_mm_args_t m;
    linear_args(fmt, group_size, w, B, &m);
    size_t total = up256(glq_mm_workspace_bytes(&m));
    if (w->rank > 0) {
        glq_mm_args_t u;
        xu_args(w, w->codes, B, &u);
        total += up256((size_t)B * w->rank * sizeof(__half)) + up256(glq_mm_workspace_bytes(&u));
    }
    return total;
}

extern "C" size_t glq_linear_counters(int fmt, int group_size, const glq_weight_t* w, int B) {
    if (!w || B <= 0) return 0;
    glq_mm_args_t m;
    linear_args(fmt, group_size, w, B, &m);
    size_t total = glq_mm_counters(&m);
    if (w->rank > 0) {
        glq_mm_args_t u;
        xu_args(w, w->codes, B, &u);
        total += glq_mm_counters(&u) + (B <= 8 ? kPairCounters : 0);
    }
    return total;
}

// x: rows of the low-rank term, xq: rows of the quantized product; settled: GLQ_WEIGHT_SETTLED holds
static int linear_forward(bool settled, int fmt, int group_size, const glq_weight_t* w, const void* ut, const void* x, int64_t ldx,
                          const void* xq, int64_t ldxq, const void* a, void* y, int64_t ldy, int B, void* workspace,
                          size_t workspace_bytes, int32_t* counters, size_t n_counters, void* stream) {
    if (!w || !x || !y || B < 0) return GLQ_ERR_ARG;
    if (B == 0 || w->N == 0) return GLQ_OK;
    glq_mm_args_t m;
    linear_args(fmt, group_size, w, B, &m);
    char* ws = reinterpret_cast<char*>(workspace);
    const MmNeeds main = mm_needs(&m);
    const size_t main_ws = up256(main.bytes), main_ctr = main.counters;
    const void* a_use = a;
    glq_mm_args_t u;
    const bool own_xu = !a && ut && w->rank > 0 && w->sv;
    if (own_xu) {
        xu_args(w, ut, B, &u);
        const size_t a_bytes = up256((size_t)B * w->rank * sizeof(__half));
        const MmNeeds un = mm_needs(&u);
        const size_t u_ws = up256(un.bytes), u_ctr = un.counters;
        if (!ws || workspace_bytes < main_ws + a_bytes + u_ws) return GLQ_ERR_WORKSPACE;
        if (u_ctr > 0 && (!counters || n_counters < main_ctr + u_ctr)) return GLQ_ERR_WORKSPACE;
        u.x = x;
        u.ldx = ldx;
        u.y = ws + main_ws;
        u.ldy = w->rank;
        u.workspace = ws + main_ws + a_bytes;
        u.workspace_bytes = u_ws;
        u.counters = counters ? counters + main_ctr : nullptr;
        u.n_counters = counters ? n_counters - main_ctr : 0;
        a_use = ws + main_ws;
    }
    if (main_ws > 0 && (!ws || workspace_bytes < main_ws)) return GLQ_ERR_WORKSPACE;
    if (main_ctr > 0 && (!counters || n_counters < main_ctr)) return GLQ_ERR_WORKSPACE;
    m.x = xq;
    m.ldx = ldxq;
    m.a0 = a_use;
    m.lda = w->rank;
    m.y = y;
    m.ldy = ldy;
    m.workspace = ws;
    m.workspace_bytes = main_ws;
    m.counters = counters;
    m.n_counters = main_ctr;
    if (!a_use) m.w.rank = 0, m.rank = 0;
    if (!own_xu) return glq_grouped_matmul(&m, stream);
    // (as two launches: x.U is the launch before and is needed only in the epilogue; x itself is older)
    m.flags = GLQ_MM_A_FROM_PREVIOUS_LAUNCH | (settled ? GLQ_MM_WEIGHTS_SETTLED : 0);
    return matmul_pair(&u, &m, stream);
}

extern "C" int glq_linear_forward(int fmt, int group_size, const glq_weight_t* w, const void* ut, const void* x,
                                  int64_t ldx, const void* a, void* y, int64_t ldy, int B, void* workspace,
                                  size_t workspace_bytes, int32_t* counters, size_t n_counters, void* stream) {
    return linear_forward(w && w->reserved == GLQ_WEIGHT_SETTLED, fmt, group_size, w, ut, x, ldx, x, ldx, a, y, ldy, B, workspace, workspace_bytes,
                          counters, n_counters, stream);
}

// the quantized product sees the rotated rows, the low-rank term the rows as given: rotation, x.U, product.  The
// rotation goes first: the product may then start while x.U still runs (it needs x.U only in its epilogue)
extern "C" size_t glq_linear_rht_workspace_bytes(int fmt, int group_size, const glq_weight_t* w, int B) {
    if (!w || B <= 0) return 0;
    return glq_linear_workspace_bytes(fmt, group_size, w, B) + up256((size_t)B * w->K * sizeof(__half));
}

extern "C" int glq_linear_rht_forward(int fmt, int group_size, const glq_weight_t* w, const void* ut, const float* signs,
                                      const void* x, int64_t ldx, const void* a, void* y, int64_t ldy, int B, void* workspace,
                                      size_t workspace_bytes, int32_t* counters, size_t n_counters, void* stream) {
    if (!w || !x || !y || !signs || B < 0) return GLQ_ERR_ARG;
    if (B == 0 || w->N == 0) return GLQ_OK;
    const size_t rot = up256((size_t)B * w->K * sizeof(__half));
    if (!workspace || workspace_bytes < rot) return GLQ_ERR_WORKSPACE;
    int rc = glq_rht_forward(x, 0, ldx, signs, B, w->K, 1.0f / sqrtf((float)w->K), workspace, 0, w->K, stream);
    if (rc != GLQ_OK) return rc;
    // (the launch ahead is the rotation, which waits for all before it and writes no weights)
    return linear_forward(true, fmt, group_size, w, ut, x, ldx, workspace, w->K, a, y, ldy, B, static_cast<char*>(workspace) + rot,
                          workspace_bytes - rot, counters, n_counters, stream);
}

// ---------------------------------------------------------------------------------------------
// Drop-ins for the reference's native modules
// ---------------------------------------------------------------------------------------------
static int turbo_rowmajor(const void* x, const uint8_t* packed, const float* norms, const float* centroids, void* y,
                          int n_problems, int rows, int N, int K, int slot_rows, void* stream) {
    if (!x || !packed || !norms || !centroids || !y) return GLQ_ERR_ARG;
    if (K <= 0 || K % 4 != 0) return GLQ_ERR_UNSUPPORTED;
    if (!aligned_to(x, 2) || !aligned_to(y, 2) || !aligned_to(norms, 4) || !aligned_to(centroids, 4)) return GLQ_ERR_ALIGN;
    Geometry g;
    int rc = plan_geometry(GLQ_FMT_T2, GLQ_EPI_LINEAR, N, K, 0, n_problems, rows, false, &g);
    if (rc != GLQ_OK) return rc;
    SkinnyParams p{};
    p.w.codes = packed;
    p.w.reserved = aligned_to(packed, 8) ? 1 : 0;   // 8-byte loads of the codes only from an 8-byte aligned base
    p.w.norms = norms;
    p.w.centroids = centroids;
    p.w.N = N;
    p.w.K = K;
    p.sv_slices = 1;
    p.x = reinterpret_cast<const __half*>(x);
    p.ldx = K;
    p.y = reinterpret_cast<__half*>(y);
    p.ldy = N;
    p.max_rows = rows;
    p.rows_stride = rows;
    p.x_vec = (aligned16(x) && K % 8 == 0) ? 1 : 0;
    p.slot_rows = slot_rows;
    p.x_extent = (long long)n_problems * rows * K;
    p.y_extent = (long long)n_problems * rows * N;
    fill_geometry(p, g);
    return launch_skinny(GLQ_FMT_T2, true, p, g, n_problems, reinterpret_cast<cudaStream_t>(stream));
}

extern "C" int glq_turbo_dequant_matmul(const void* x_rot, const uint8_t* packed, const float* norms,
                                        const float* centroids, void* y, int B, int N, int K, void* stream) {
    if (B < 0 || N < 0) return GLQ_ERR_ARG;
    if (B == 0 || N == 0) return GLQ_OK;
    return turbo_rowmajor(x_rot, packed, norms, centroids, y, 1, B, N, K, 0, stream);
}

extern "C" int glq_turbo_dequant_grouped_gemv(const void* x_grouped, const uint8_t* packed_cat, const float* norms_cat,
                                              const float* centroids, void* y, int E, int N_out, int K,
                                              void* stream) {
    if (E < 0 || N_out < 0) return GLQ_ERR_ARG;
    if (E == 0 || N_out == 0) return GLQ_OK;
    return turbo_rowmajor(x_grouped, packed_cat, norms_cat, centroids, y, E, 1, N_out, K, N_out, stream);
}

extern "C" int glq_gptq_dequant_matmul(const float* x, const int8_t* q, const void* scales, const void* zeros,
                                       const float* lora_out, float* y, int B, int N, int K, int groupsize,
                                       int n_groups, int sym, void* stream) {
    if (B < 0 || N < 0 || K < 0) return GLQ_ERR_ARG;
    if (B == 0 || N == 0) return GLQ_OK;
    if (!x || !q || !scales || !y || (!sym && !zeros)) return GLQ_ERR_ARG;
    if (groupsize <= 0 || n_groups <= 0 || (long)n_groups * groupsize < K) return GLQ_ERR_ARG;
    if (!aligned_to(x, 4) || !aligned_to(y, 4) || !aligned_to(lora_out, 4) || !aligned_to(scales, 2) || !aligned_to(zeros, 2))
        return GLQ_ERR_ALIGN;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const size_t smem = (size_t)K * sizeof(float);
    // activation rows per pass over the codes: up to 8, as many as the staged rows leave room for (one pass for a
    // decode batch; a long prompt re-reads the int8 matrix once per 8 rows)
    int per = 8;
    while (per > 1 && smem * per > 200 * 1024) per /= 2;
    if (smem > 200 * 1024) return GLQ_ERR_UNSUPPORTED;
    static SmemLimit limit[2];
    for (int b0 = 0; b0 < B; b0 += per) {
        const int nb = std::min(per, B - b0);
        const int wide = nb > 4 ? 1 : 0;
        const dim3 grid(cdiv(N, kWarpsPerCta));
        const size_t need = smem * nb;
        if (need > 48 * 1024)
            GLQ_CUDA(reserve_smem(wide ? reinterpret_cast<const void*>(gptq_i8_kernel<8>) : reinterpret_cast<const void*>(gptq_i8_kernel<4>),
                                  limit[wide], smem * (wide ? per : std::min(per, 4))));
        const float* xb = x + (size_t)b0 * K;
        const float* lb = lora_out ? lora_out + (size_t)b0 * N : nullptr;
        float* yb = y + (size_t)b0 * N;
        if (wide)
            gptq_i8_kernel<8><<<grid, kThreads, need, st>>>(xb, q, reinterpret_cast<const __half*>(scales),
                                                            reinterpret_cast<const __half*>(zeros), lb, yb, nb, N, K,
                                                            groupsize, n_groups, sym);
        else
            gptq_i8_kernel<4><<<grid, kThreads, need, st>>>(xb, q, reinterpret_cast<const __half*>(scales),
                                                            reinterpret_cast<const __half*>(zeros), lb, yb, nb, N, K,
                                                            groupsize, n_groups, sym);
        GLQ_CUDA(cudaGetLastError());
    }
    return GLQ_OK;
}

// ---------------------------------------------------------------------------------------------
// glq_turbo_dequant_matmul_static: the same product as glq_turbo_dequant_matmul, with k split over
// CTAs so that a single small matmul fills the machine, for callers that cannot hand over (or
// allocate) a workspace.  The partial sums and the arrival counters of the split live in a fixed
// array that is part of the library image.
// ---------------------------------------------------------------------------------------------
#define GLQ_STATIC_SCRATCH_BYTES (4u << 20)  /* partial sums */
#define GLQ_STATIC_COUNTERS 4096             /* arrival counters (ints), in front of the partial sums */
static __device__ __align__(256) unsigned char g_static_scratch[GLQ_STATIC_COUNTERS * 4 + GLQ_STATIC_SCRATCH_BYTES];

extern "C" size_t glq_static_scratch_bytes(void) { return GLQ_STATIC_SCRATCH_BYTES; }

extern "C" size_t glq_static_scratch_needed(int B, int N, int K) {
    Geometry g;
    if (B <= 0 || N <= 0 || K <= 0 || K % 4 != 0) return 0;
    if (plan_geometry(GLQ_FMT_T2, GLQ_EPI_LINEAR, N, K, 0, 1, B, true, &g) != GLQ_OK) return 0;
    return g.scratch_bytes;
}

extern "C" int glq_turbo_dequant_matmul_static(const void* x_rot, const uint8_t* packed, const float* norms,
                                               const float* centroids, void* y, int B, int N, int K, void* stream) {
    if (B < 0 || N < 0) return GLQ_ERR_ARG;
    if (B == 0 || N == 0) return GLQ_OK;
    if (!x_rot || !packed || !norms || !centroids || !y) return GLQ_ERR_ARG;
    if (K <= 0 || K % 4 != 0) return GLQ_ERR_UNSUPPORTED;
    if (!aligned_to(x_rot, 2) || !aligned_to(y, 2) || !aligned_to(norms, 4) || !aligned_to(centroids, 4)) return GLQ_ERR_ALIGN;
    // The array's name is only a host-side handle: its device address is looked up once per device,
    // with that device current, and it is that address the kernel gets.
    static unsigned char* dev_ptr[64] = {nullptr};
    int dev = 0;
    GLQ_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return GLQ_ERR_UNSUPPORTED;
    if (dev_ptr[dev] == nullptr) {
        void* ptr = nullptr;
        GLQ_CUDA(cudaGetSymbolAddress(&ptr, g_static_scratch));
        if (ptr == nullptr) return GLQ_ERR_CUDA;
        dev_ptr[dev] = reinterpret_cast<unsigned char*>(ptr);
    }
    Geometry g;
    int rc = plan_geometry(GLQ_FMT_T2, GLQ_EPI_LINEAR, N, K, 0, 1, B, true, &g);
    if (rc != GLQ_OK) return rc;
    // sizes the fixed array cannot hold are rejected, not truncated
    if (g.scratch_bytes > GLQ_STATIC_SCRATCH_BYTES || g.n_counters > GLQ_STATIC_COUNTERS) return GLQ_ERR_WORKSPACE;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    // every call shares the array and it keeps the previous call's contents: the counters must start at zero
    if (g.n_counters > 0) GLQ_CUDA(cudaMemsetAsync(dev_ptr[dev], 0, g.n_counters * sizeof(int), st));
    SkinnyParams p{};
    p.w.codes = packed;
    p.w.reserved = aligned_to(packed, 8) ? 1 : 0;
    p.w.norms = norms;
    p.w.centroids = centroids;
    p.w.N = N;
    p.w.K = K;
    p.sv_slices = 1;
    p.x = reinterpret_cast<const __half*>(x_rot);
    p.ldx = K;
    p.y = reinterpret_cast<__half*>(y);
    p.ldy = N;
    p.max_rows = B;
    p.rows_stride = B;
    p.x_vec = (aligned16(x_rot) && K % 8 == 0) ? 1 : 0;
    p.x_extent = (long long)B * K;
    p.y_extent = (long long)B * N;
    p.counters = reinterpret_cast<int*>(dev_ptr[dev]);
    p.scratch = reinterpret_cast<float4*>(dev_ptr[dev] + GLQ_STATIC_COUNTERS * 4);
    fill_geometry(p, g);
    return launch_skinny(GLQ_FMT_T2, true, p, g, 1, st);
}

// ---------------------------------------------------------------------------------------------
// Load-time re-tiling and the dequantised-tile check
// ---------------------------------------------------------------------------------------------
// Behind a packing kernel: a launch may start beside the one ahead of it and read weights (GLQ_WEIGHT_SETTLED), so the one ahead is
// never the kernel that writes them.  This one starts when that one is complete.
static int pack_end(void* stream) {
    GLQ_CUDA(cudaGetLastError());
    settle_kernel<<<1, 32, 0, reinterpret_cast<cudaStream_t>(stream)>>>();
    GLQ_CUDA(cudaGetLastError());
    return GLQ_OK;
}
static inline bool slot_ok(int slot, int count) { return count >= 1 && count <= 2 && slot >= 0 && slot < count; }

extern "C" int glq_pack_gptq(const int32_t* q, const void* scales, const void* zeros, int bits, int N, int K,
                             int group_size, void* tiled, int slot, int count, void* stream) {
    if (!q || !scales || !tiled || N <= 0 || K <= 0 || !slot_ok(slot, count)) return GLQ_ERR_ARG;
    if (bits != 2 && bits != 4) return GLQ_ERR_UNSUPPORTED;
    const int kb = bits == 2 ? 128 : 64;
    if (group_size <= 0 || group_size % kb != 0) return GLQ_ERR_UNSUPPORTED;
    const size_t words = (size_t)cdiv(N, 16) * cdiv(K, kb) * 144;
    pack_gptq_kernel<<<(unsigned)((words + 255) / 256), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
        q, reinterpret_cast<const __half*>(scales), reinterpret_cast<const __half*>(zeros), bits, N, K, group_size,
        reinterpret_cast<unsigned char*>(tiled), slot, count);
    return pack_end(stream);
}

extern "C" int glq_pack_turbo(const uint8_t* packed, int N, int K, void* tiled, int slot, int count, void* stream) {
    if (!packed || !tiled || N <= 0 || K <= 0 || !slot_ok(slot, count)) return GLQ_ERR_ARG;
    if (K % 4 != 0) return GLQ_ERR_UNSUPPORTED;
    const size_t words = (size_t)cdiv(N, 16) * cdiv(K, 128) * 128;
    pack_turbo_kernel<<<(unsigned)((words + 255) / 256), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
        packed, N, K, reinterpret_cast<unsigned char*>(tiled), slot, count);
    return pack_end(stream);
}

extern "C" int glq_pack_rows_f32(const float* v, int N, float* out, int slot, int count, void* stream) {
    if (!v || !out || N <= 0 || !slot_ok(slot, count)) return GLQ_ERR_ARG;
    const int n = cdiv(N, 16) * 16;
    pack_rows_f32_kernel<<<(n + 255) / 256, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(v, N, out, slot, count);
    return pack_end(stream);
}

extern "C" int glq_pack_sv(const void* sv, int N, int rank, void* out, int slot, int count, void* stream) {
    if (!sv || !out || N <= 0 || rank <= 0 || !slot_ok(slot, count)) return GLQ_ERR_ARG;
    if (rank % 16 != 0) return GLQ_ERR_UNSUPPORTED;
    const size_t total = (size_t)cdiv(N, 16) * cdiv(rank, 64) * 1024;
    pack_sv_kernel<<<(unsigned)((total + 255) / 256), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
        reinterpret_cast<const __half*>(sv), N, rank, reinterpret_cast<__half*>(out), slot, count);
    return pack_end(stream);
}

extern "C" int glq_pack_f16(const void* W, long stride_n, long stride_k, int N, int K, void* tiled, void* stream) {
    if (!W || !tiled || N <= 0 || K <= 0) return GLQ_ERR_ARG;
    const size_t elems = glq_tiled_f16_bytes(N, K) / 2;
    pack_f16_kernel<<<(unsigned)((elems + 255) / 256), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
        reinterpret_cast<const __half*>(W), stride_n, stride_k, N, K, reinterpret_cast<__half*>(tiled), elems);
    return pack_end(stream);
}

extern "C" int glq_dequant_tiled(int fmt, const void* tiled, const float* norms_tiled, const float* centroids, int N,
                                 int K, int slot, int count, void* out, void* stream) {
    if (!tiled || !out || N <= 0 || K <= 0 || !slot_ok(slot, count)) return GLQ_ERR_ARG;
    fmt = tile_fmt(fmt);
    const size_t elems = (size_t)N * K;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (fmt == GLQ_FMT_Q2 || fmt == GLQ_FMT_Q4) {
        dequant_tiled_q_kernel<<<(unsigned)((elems + 255) / 256), 256, 0, st>>>(
            fmt, reinterpret_cast<const unsigned char*>(tiled), N, K, slot, count, reinterpret_cast<__half*>(out));
    } else if (fmt == GLQ_FMT_T2) {
        if (!norms_tiled || !centroids) return GLQ_ERR_ARG;
        dequant_tiled_t2_kernel<<<(unsigned)((elems + 255) / 256), 256, 0, st>>>(
            reinterpret_cast<const unsigned char*>(tiled), norms_tiled, centroids, N, K, slot, count,
            reinterpret_cast<float*>(out));
    } else {
        return GLQ_ERR_UNSUPPORTED;
    }
    GLQ_CUDA(cudaGetLastError());
    return GLQ_OK;
}

// ---------------------------------------------------------------------------------------------
// randomized Hadamard rotation
// ---------------------------------------------------------------------------------------------
template <int E, typename TI, typename TO>
static int launch_rht_e(const void* x, int64_t ldx, const float* signs, int rows, int d, int n, float scale, void* y, int64_t ldy, cudaStream_t st) {
    const int threads = std::max(32, n >> E);
    const size_t smem = threads > 32 ? (size_t)n * sizeof(float) : 0;
    auto kern = rht_kernel<E, TI, TO>;
    if (smem > 48 * 1024) {
        static SmemLimit limit;
        GLQ_CUDA(reserve_smem(reinterpret_cast<const void*>(kern), limit, smem));
    }
    const int vec = aligned16(x) && ldx % 8 == 0 ? 1 : 0;
    // (more rows than SMs gain nothing from waiting beside the launch ahead)
    GLQ_CUDA(launch_kernel(rows <= num_sms(), kern, dim3(rows), dim3(threads), smem, st, reinterpret_cast<const TI*>(x), (long long)ldx, signs, d, n,
                           scale, reinterpret_cast<TO*>(y), (long long)ldy, vec));
    return GLQ_OK;
}
// values per thread: the smallest power whose exponent covers the stages between warps (log2(n) <= 2 E + 5)
template <typename TI, typename TO>
static int launch_rht(const void* x, int64_t ldx, const float* signs, int rows, int d, int n, float scale, void* y, int64_t ldy, cudaStream_t st) {
    if (n <= 32) return launch_rht_e<0, TI, TO>(x, ldx, signs, rows, d, n, scale, y, ldy, st);
    if (n <= 128) return launch_rht_e<1, TI, TO>(x, ldx, signs, rows, d, n, scale, y, ldy, st);
    if (n <= 512) return launch_rht_e<2, TI, TO>(x, ldx, signs, rows, d, n, scale, y, ldy, st);
    if (n <= 2048) return launch_rht_e<3, TI, TO>(x, ldx, signs, rows, d, n, scale, y, ldy, st);
    if (n <= 8192) return launch_rht_e<4, TI, TO>(x, ldx, signs, rows, d, n, scale, y, ldy, st);
    return launch_rht_e<5, TI, TO>(x, ldx, signs, rows, d, n, scale, y, ldy, st);
}

extern "C" int glq_rht_forward(const void* x, int x_is_f32, int64_t ldx, const float* signs, int rows, int d, float scale,
                               void* y, int y_is_f32, int64_t ldy, void* stream) {
    if (!x || !y || !signs || rows < 0 || d <= 0) return GLQ_ERR_ARG;
    if (rows == 0) return GLQ_OK;
    int n = 1;
    while (n < d) n <<= 1;
    if (n > 32768) return GLQ_ERR_UNSUPPORTED;       // n floats of shared memory per row
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (x_is_f32 && y_is_f32) return launch_rht<float, float>(x, ldx, signs, rows, d, n, scale, y, ldy, st);
    if (!x_is_f32 && !y_is_f32) return launch_rht<__half, __half>(x, ldx, signs, rows, d, n, scale, y, ldy, st);
    if (x_is_f32) return launch_rht<float, __half>(x, ldx, signs, rows, d, n, scale, y, ldy, st);
    return launch_rht<__half, float>(x, ldx, signs, rows, d, n, scale, y, ldy, st);
}

int glq_moe_error_words(unsigned long long* out4, int clear);   // moe.cu: the error word of that translation unit

// First bounds violation or timed-out wait recorded by a kernel: {code, index, limit, block<<32|thread};
// all zero when there was none.  Synchronises the device.
extern "C" int glq_debug_error(unsigned long long* out4, int clear) {
    if (!out4) return GLQ_ERR_ARG;
    GLQ_CUDA(cudaMemcpyFromSymbol(out4, g_glq_err, 4 * sizeof(unsigned long long)));
    if (clear) {
        unsigned long long z[4] = {0, 0, 0, 0};
        GLQ_CUDA(cudaMemcpyToSymbol(g_glq_err, z, sizeof(z)));
    }
    unsigned long long m[4] = {0, 0, 0, 0};
    const int rc = glq_moe_error_words(m, clear);
    if (rc != GLQ_OK) return rc;
    if (out4[0] == 0 && m[0] != 0)
        for (int i = 0; i < 4; ++i) out4[i] = m[i];
    return GLQ_OK;
}
