// SPDX-License-Identifier: Apache-2.0
//
// Grouped dequant-GEMM with the weight operand in tensor memory: 2-bit, 4-bit and codebook codes.
//
// An SS-operand MMA reads both operands from shared memory (8 KB per 128x128x16 instruction, the whole
// 128 B/clk port) while producers would store the unpacked weights and the bulk copy write the token
// operand through the same port.  Here the producers write the unpacked fp16 values straight into
// tensor memory (tcgen05.st, 16 lanes x 256 bit shape, which matches the (g, t) ownership of the code
// tiles: lane (g, t) holds rows g and g+8 and four consecutive K positions of every 16) and the MMA
// takes A from there; only the token operand uses shared memory.
//
// Tensor memory (512 columns): accumulators first (TN columns, twice for gate|up), then a ring of S
// stages of 64 columns (128 K positions x fp16) per matrix.
//
// One CTA per SM works through the list of (token tile, 128-feature tile) items; the warps keep their roles
// over all of a CTA's items, so barrier set-up, the TMEM allocation and the pipeline fill are paid once per
// CTA instead of once per tile.  16 producer warps unpack the codes of a 128-channel stage into the
// tensor-memory ring, one warp issues the MMAs, one bulk-copies the token operand.
//
//  * Work items are drawn from a grid-wide counter (zeroed by the pre-pass) by a warp of its own, up to kPsQueue ahead;
//    it looks the problem up and hands the operands' addresses to the other warps through a small queue in
//    shared memory, so an SM that runs faster takes more items and nobody else walks the dependent loads.
//  * The rings run on across item boundaries: the loader fetches the next item's token operand while the
//    producers still finish the current one, and the producers request the next item's first codes before
//    they turn to the finished accumulator.
//  * A finished accumulator is read into registers (epilogue arithmetic, fp16 pairs) and released at once;
//    the results go to y after the weight ring of the next item is full again, through a staging tile in
//    shared memory ([token][feature], two passes) with 16-byte row-contiguous stores.  With one accumulator the tensor
//    pipe waits for this: 128 experts x 256 rows, 2048 x 768, took 228 us with a bulk copy per row and the output scales read
//    by every lane, and 161 with plain stores and the scales requested before the wait.
//
// What bounds it: with few tokens per problem (an expert of a prompt sees some tens of rows) the producers' issue
// slots.  A first form spent 253 instructions per warp, matrix and stage (one shift per pair of codes, both
// roundings of the dequantisation computed and one selected, every warp looking up its item): 142 us for the gate|up
// product of 60 experts x 34 rows (1408 x 2048, 2-bit), scheduler slots 57 % used, DRAM 12 %.  Now 140 instructions
// and 99 us; 97 -> 60 us for the down product (2048 x 1408).  With one multiply-add per pair of 2-bit codes and one election
// per four MMAs 95 and 54 us; with the look-ups in a warp of their own, the accumulator released before the epilogue's arithmetic
// and that arithmetic left out for tokens that do not exist 86 and 55 (codebook codes: 105 -> 95; prompts of few large experts gain nothing
// by it: 600 tokens through 8 Mixtral-shaped experts 740 us a block before, 734 now).  No pipe is full (gate|up:
// integer 49 %, issue slots 53 %, tensor 23 %): what is left is the latency of a warp's own chain through a stage, of which four
// warps per scheduler cover only a part.
//
// Every wait is bounded (tc_wait); a wait that runs out marks the CTA dead, all roles leave their loops
// and the kernel ends.
#pragma once

#include "tc_mm.cuh"

namespace glq {

// Work items that may be handed out ahead of the slowest warp.  Two hide a look-up; with four a CTA held items back at the end that
// others had time for (8 Mixtral-shaped experts, codebook, 300 tokens 663 us a block against 607; 2-bit, 600 tokens 803 against 734; a
// 512-token prompt of 24 layers 8065 against 7905).
constexpr int kPsQueue = 2;

__device__ __forceinline__ void tc_st_x4(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void tc_st_x2(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.16x256b.x2.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]),
                 "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
__device__ __forceinline__ void tc_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// D (TMEM) += A (TMEM, 128 lanes x 8 columns = 16 fp16 per row) * B (shared memory descriptor), a run of four k steps: A
// advances by 8 columns, B by 32 bytes.  The whole warp comes here with the same operands and one elected lane issues: in code
// that one lane runs alone the issuing warp, not the tensor pipe, set the pace (113 to 117 cycles per MMA of any N up to
// 128).  One election serves the four (one for each still left 70
// to 90 cycles between MMAs of 64 columns, which the tensor pipe does in 32).
__device__ __forceinline__ void tc_mma4_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n .reg .pred p, o, e;\n .reg .b32 a1, a2, a3;\n .reg .b64 b1, b2, b3;\n"
        " setp.ne.b32 p, %4, 0;\n setp.eq.b32 o, 0, 0;\n"
        " add.u32 a1, %1, 8;\n add.u32 a2, %1, 16;\n add.u32 a3, %1, 24;\n"
        " add.u64 b1, %2, 2;\n add.u64 b2, %2, 4;\n add.u64 b3, %2, 6;\n"
        " elect.sync _|e, 0xffffffff;\n"
        " @e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
        " @e tcgen05.mma.cta_group::1.kind::f16 [%0], [a1], b1, %3, o;\n"
        " @e tcgen05.mma.cta_group::1.kind::f16 [%0], [a2], b2, %3, o;\n"
        " @e tcgen05.mma.cta_group::1.kind::f16 [%0], [a3], b3, %3, o;\n}\n" ::"r"(d_tmem),
        "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(acc)
        : "memory");
}
__device__ __forceinline__ void tc_commit_warp(uint32_t bar) {
    asm volatile(
        "{\n .reg .pred e;\n elect.sync _|e, 0xffffffff;\n"
        " @e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(bar)
        : "memory");
}

constexpr int kPsRows = 64;                                      // tokens of a result pass
constexpr int kPsOut = kPsRows * 256;                            // its staging tile [token][128 features] fp16, two of them
constexpr int kPsThreads = (kTcProducers + 4) * 32;              // and products, results, loader, items
// Registers of a thread: 96 at launch (640 threads).  With 4-bit codes of two matrices the producers' loop spills; there the
// warpgroup of the other roles hands some of its own over (gate|up of 60 experts x 34 rows 138 -> 130 us; 2-bit codes fit, and their
// down product takes 58 us instead of 56 with the others at 64).
constexpr int kPsRegsProducer = 104, kPsRegsOther = 64;
static_assert(kTcProducers * 32 * kPsRegsProducer + 4 * 32 * kPsRegsOther <= kPsThreads * 96, "registers");

template <int FMT, int TN, int NM, bool SW> struct TcPsCfg {
    static constexpr bool SHIFT_REGS = FMT == GLQ_FMT_Q4 && NM == 2;
    static constexpr int NOUT = SW ? 1 : NM;                     // 128-feature output tiles of an item
    static constexpr int ACC = NM * TN;                          // accumulator columns
    static constexpr int B_BYTES = TN * 256;
    static constexpr int NPASS = NOUT * (TN / kPsRows);          // passes in which an item's results leave
    // ring stages: what tensor memory and shared memory both hold, at most 6
    static constexpr int S_TMEM = (512 - ACC) / (NM * 64), S_SMEM = (225 * 1024 - 2 * kPsOut) / B_BYTES;
    static constexpr int S0 = S_TMEM < S_SMEM ? S_TMEM : S_SMEM, S = S0 < 6 ? S0 : 6;
    static constexpr size_t SMEM = (size_t)S * B_BYTES + 2 * kPsOut + 1024;
    static_assert(S >= 2 && SMEM <= 227 * 1024, "shared memory");
};

// tc_wait of a whole warp: the barrier is tried before anything else is looked at (the common case costs one instruction)
__device__ __forceinline__ bool ps_wait_warp(uint32_t bar, uint32_t parity, volatile int* dead, int code) {
    return __all_sync(0xffffffffu, mbar_try_wait(bar, parity) || tc_wait(bar, parity, dead, code));
}

// A work item as it is handed out; ft < 0 ends the list.
struct PsItem {
    const unsigned char *codes, *sv;
    const __half* bias;
    const float *norms, *centroids;
    int ft, lt, cnt, e0, gt;
};

// One row's 16 codes of a stage -> eight fp16 pairs in K position order (tc_ts_channel_of).
// Affine codes: the code bits are put into the mantissa of an fp16 number of a known offset, one subtraction of
// offset + z -- exact for every zero point that the sum keeps whole, which integer zero points, the quantizer's
// output, always are -- yields fp16(q - z), one product the same fp16(fp16(q - z) * s) as the reference's tiles.
// Three instructions per pair; another zero point takes (offset + code - offset) - z.
template <int FMT> struct PsUnpack;
template <> struct PsUnpack<GLQ_FMT_Q2> {
    static __device__ __forceinline__ constexpr float off(int c) { return c == 0 ? 64.f : (c == 1 ? 16.f : 4.f); }
    static constexpr float kTop = 64.f;        // the largest offset
    // offset class of pair j (see unpack_q2)
    static __device__ __forceinline__ constexpr int cls(int j) { return (j == 4 || j == 7) ? 2 : ((j == 1 || j == 3 || j == 6) ? 1 : 0); }
    static constexpr int WORDS = 1;             // 32-bit words that hold a row's 16 codes of a half
    static __device__ __forceinline__ void pairs(const uint32_t (&w)[1], int, uint32_t (&h)[8]) { unpack_q2(w[0], h); }
};
template <> struct PsUnpack<GLQ_FMT_Q4> {
    static __device__ __forceinline__ constexpr float off(int c) { return c == 0 ? 1024.f : 64.f; }
    static constexpr float kTop = 1024.f;
    static __device__ __forceinline__ constexpr int cls(int j) { return j & 1; }
    static constexpr int WORDS = 4;             // word t >> 1 of each of the block's four groups of 16 channels
    // codes (c, c + 4), (c + 1, c + 5) of every word, c = 2 (t & 1); sh = 8 (t & 1)
    static __device__ __forceinline__ void pairs(const uint32_t (&w)[4], int sh, uint32_t (&h)[8]) {
#pragma unroll
        for (int n = 0; n < 4; ++n) {
            const uint32_t v = w[n] >> sh;
            h[2 * n] = and_or(v, 0x000F000Fu, 0x64006400u);
            h[2 * n + 1] = and_or(v, 0x00F000F0u, 0x54005400u);
        }
    }
};
template <> struct PsUnpack<GLQ_FMT_T2> { static constexpr int WORDS = 1; };

// 2-bit codes, the usual case: a field masked out of its word, with nothing or-ed in, IS an fp16 number, the subnormal
// q 2^-18 (bits 6, 7) or q 2^-16 (bits 8, 9).  With s 2^18 / s 2^16 as the factor and -z s as the addend, one multiply-add
// yields fp16((q - z) s): the product is exact, and so is z s for z = 0, 1, 2 (z = 3: the codes are inverted, 3 - q, and the
// factor's sign with them), so that the one rounding is that of the reference's product.  Two instructions per pair and two
// of the half-precision pipe's slots fewer.  |s| < 1/4 keeps the factors finite.
struct PsQ2 {
    uint32_t f6, f8, c, flip;         // (row g, row g + 8): s 2^18, s 2^16, -z s; inversion mask
    bool fast;                        // the whole warp's rows allow this
};
__device__ __forceinline__ PsQ2 ps_q2_setup(const uint32_t (&sz)[2]) {
    auto h2 = [](uint32_t v) { return *reinterpret_cast<const __half2*>(&v); };
    auto u = [](__half2 v) { return *reinterpret_cast<const uint32_t*>(&v); };
    PsQ2 r;
    const uint32_t zb = __byte_perm(sz[0], sz[1], 0x7632), sb = __byte_perm(sz[0], sz[1], 0x5410);
    r.flip = __heq2_mask(h2(zb), __float2half2_rn(3.f));
    const __half2 z = h2(zb & ~r.flip), big = __float2half2_rn(1024.f);
    // z one of 0, 1, 2: 1024 + z keeps it, and it lies in the range
    const bool ok = __hbeq2(__hsub2(__hadd2(z, big), big), z) && __hbeq2(__hmax2(__hmin2(z, __float2half2_rn(2.f)), __float2half2_rn(0.f)), z) &&
                    __hblt2(__habs2(h2(sb)), __float2half2_rn(0.25f));
    r.fast = __all_sync(0xffffffffu, ok);
    const __half2 s = h2(sb ^ (r.flip & 0x80008000u));
    const __half2 f8 = __hmul2(__hmul2(s, __float2half2_rn(256.f)), __float2half2_rn(256.f));
    r.f8 = u(f8);
    r.f6 = u(__hmul2(f8, __float2half2_rn(4.f)));
    r.c = u(__hneg2(__hmul2(z, h2(sb))));
    return r;
}

// Both rows (g, g + 8) of a lane: words w[row][..], (scale, zero) pairs sz[row] -> the 16 registers of tc_st_x4.
template <int FMT>
__device__ __forceinline__ void ps_affine(const uint32_t (&w)[2][PsUnpack<FMT>::WORDS], const uint32_t (&sz)[2], int sh, uint32_t (&r)[16]) {
    using U = PsUnpack<FMT>;
    const uint32_t zb = __byte_perm(sz[0], sz[1], 0x7632);        // (z of row g, z of row g + 8)
    const __half2 z2 = *reinterpret_cast<const __half2*>(&zb);
    __half2 zo[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) zo[i] = __hadd2(z2, __float2half2_rn(U::off(i)));
    // the largest offset keeps every bit of both zero points (the smaller ones then do, for |z| <= 1024)
    const __half2 top = __hadd2(z2, __float2half2_rn(U::kTop));
    const bool whole = __hbeq2(__hsub2(top, __float2half2_rn(U::kTop)), z2) && __hble2(__habs2(z2), __float2half2_rn(1024.f));
    const bool fast = __all_sync(0xffffffffu, whole);
#pragma unroll
    for (int hrow = 0; hrow < 2; ++hrow) {
        uint32_t h[8];
        U::pairs(w[hrow], sh, h);
        const __half2 s2 = __half2half2(__ushort_as_half((unsigned short)(sz[hrow] & 0xffffu)));
        if (fast) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const __half2 zc = zo[U::cls(j)];
                const __half2 zr = hrow ? __high2half2(zc) : __low2half2(zc);
                const __half2 v = __hmul2(__hsub2(*reinterpret_cast<const __half2*>(&h[j]), zr), s2);
                r[4 * (j >> 1) + 2 * hrow + (j & 1)] = *reinterpret_cast<const uint32_t*>(&v);
            }
        } else {
            const __half2 zr = hrow ? __high2half2(z2) : __low2half2(z2);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const __half2 q = __hsub2(*reinterpret_cast<const __half2*>(&h[j]), __float2half2_rn(U::off(U::cls(j))));
                const __half2 v = __hmul2(__hsub2(q, zr), s2);
                r[4 * (j >> 1) + 2 * hrow + (j & 1)] = *reinterpret_cast<const uint32_t*>(&v);
            }
        }
    }
}

__device__ __forceinline__ void ps_q2_fast(const uint32_t (&w)[2][1], const PsQ2& q, uint32_t (&r)[16]) {
#pragma unroll
    for (int hrow = 0; hrow < 2; ++hrow) {
        auto sel = [&](uint32_t v) {
            const __half2 h = *reinterpret_cast<const __half2*>(&v);
            return hrow ? __high2half2(h) : __low2half2(h);
        };
        const __half2 f6 = sel(q.f6), f8 = sel(q.f8), c = sel(q.c);
        const uint32_t v = w[hrow][0] ^ __byte_perm(q.flip, 0, hrow ? 0x3232 : 0x1010);
        // fields 0..7 of either half of the word, moved to bits 6 or 8
        const uint32_t h[8] = {(v << 6) & 0x00C000C0u, (v << 6) & 0x03000300u, (v << 4) & 0x03000300u, v & 0x00C000C0u,
                               v & 0x03000300u, (v >> 4) & 0x00C000C0u, (v >> 4) & 0x03000300u, (v >> 6) & 0x03000300u};
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const bool low = j == 0 || j == 3 || j == 5;
            const __half2 y = __hfma2(*reinterpret_cast<const __half2*>(&h[j]), low ? f6 : f8, c);
            r[4 * (j >> 1) + 2 * hrow + (j & 1)] = *reinterpret_cast<const uint32_t*>(&y);
        }
    }
}

// NM = 2: an item is 128 features of gate and of up (SW), or two adjacent 128-feature tiles of a plain product; a producer
// warp then unpacks all 128 channels of its 16-row tile of one matrix.  NM = 1 (few items, or token tiles so wide that one
// accumulator fills half of tensor memory): two warps share a tile, one per half of the lanes' channels.
template <int FMT, int TN, int NM, bool SW>
__global__ void __launch_bounds__(kPsThreads, 1) tc_ps_kernel(const TcParams p) {
    using C = TcPsCfg<FMT, TN, NM, SW>;
    constexpr int S = C::S;
    static_assert(!SW || NM == 2, "gate|up items hold two matrices");
    constexpr bool AFFINE = FMT != GLQ_FMT_T2;
    constexpr int BB = FMT == GLQ_FMT_T2 ? 512 : 576;       // bytes of a (tile, k block)
    constexpr int HALVES = NM;                              // halves of the lanes' channels that a warp unpacks
    extern __shared__ unsigned char tc_smem_raw[];
    __shared__ __align__(8) unsigned long long bars[2 * S + 6 + 2 * kPsQueue];
    __shared__ uint32_t s_tmem;
    __shared__ int s_dead;
    __shared__ PsItem s_item[kPsQueue];       // work items in the order they were drawn

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t sbase = (smem_u32(tc_smem_raw) + 1023u) & ~1023u;
    const uint32_t obase = sbase + (uint32_t)S * C::B_BYTES;      // two staging tiles of the results
    const uint32_t bar_full = smem_u32(bars), bar_empty = bar_full + 8 * S;
    const uint32_t bar_acc = bar_full + 16 * S, bar_acc_free = bar_acc + 8;
    const uint32_t bar_staged = bar_acc + 16, bar_stored = bar_acc + 32;   // per staging tile: written by the producers / read
    const uint32_t bar_tq_full = bar_acc + 48, bar_tq_empty = bar_tq_full + 8 * kPsQueue;
    volatile int* dead = &s_dead;

    if (threadIdx.x == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(bar_full + 8 * s, kTcProducers + 1);
            mbar_init(bar_empty + 8 * s, 1);
        }
        mbar_init(bar_acc, 1);
        mbar_init(bar_acc_free, kTcProducers);
        for (int i = 0; i < 2; ++i) {
            mbar_init(bar_staged + 8 * i, kTcProducers);
            mbar_init(bar_stored + 8 * i, 1);
        }
        for (int i = 0; i < kPsQueue; ++i) {
            mbar_init(bar_tq_full + 8 * i, 1);
            mbar_init(bar_tq_empty + 8 * i, kTcProducers + 3);
        }
        s_dead = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kTcProducers) tc_alloc(smem_u32(&s_tmem), 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    const uint32_t ring = tmem + C::ACC;      // first column of the weight ring

    const int N = p.N;
    const bool has_lr = p.rank > 0 && p.a[0] != nullptr;
    const int nst = p.nkb + (has_lr ? p.ns : 0);
    const int n_work = p.n_ft * p.tiles_max;
    // Work item n of this CTA (all lanes of a consumer warp call it): false when there is none left, or the CTA is dead.
    // Its slot is the caller's until release_item.
    auto have_item = [&](int n) -> bool {
        const int qi = n % kPsQueue;
        const bool got = __all_sync(0xffffffffu, tc_wait(bar_tq_full + 8 * qi, (uint32_t)((n / kPsQueue) & 1), dead, 108));
        return got && s_item[qi].ft >= 0;
    };
    auto release_item = [&](int n) {
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_tq_empty + 8 * (n % kPsQueue));
    };

    if (warp < kTcProducers) {
        if constexpr (C::SHIFT_REGS) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kPsRegsProducer));
        // ================= producers: unpack into tensor memory, then the tile's epilogue =================
        const int g = lane >> 2, t = lane & 3;
        const int q = warp & 3, sub = warp >> 2;                   // a warp reaches the tensor-memory lanes of its quarter q
        const int tl = 2 * q + (sub & 1);                          // its 16-row tile of the 128
        const int mx = NM == 2 ? sub >> 1 : 0, wh0 = NM == 2 ? 0 : sub >> 1;   // its matrix / its half of the channels
        const uint32_t lane_base = (uint32_t)(16 * tl) << 16;
        const int nblk = FMT == GLQ_FMT_Q4 ? (p.K + 63) / 64 : p.nkb;
        int s = 0;
        uint32_t ph = 0;
        // ---- results of item n: accumulator -> epilogue arithmetic -> staging tile [token][feature], 64 tokens per pass;
        // the store warp takes the tiles from there.  Done while the ring of item n + 1 is already full, so that neither the
        // producers wait for the last products of item n nor the tensor pipe for the producers.
        const int part = warp >> 2;                                // this warp's 16 tokens of a pass
        const uint32_t trow = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(part * 16);
        const uint32_t orow = obase + (uint32_t)(part * 16) * 256u + (uint32_t)(q * 32 + lane) * 2u;
        int pass = 0;
        auto results = [&](int n) -> bool {
            const volatile PsItem& im = s_item[n % kPsQueue];
            // the tokens' output scales, lane j that of token j, all requested before the wait
            const bool scaled = !SW && p.entry_scale;
            __half sc_h[TN / kPsRows];
#pragma unroll
            for (int i = 0; i < TN / kPsRows; ++i) {
                const int r = im.lt * TN + i * kPsRows + part * 16 + (lane & 15);
                sc_h[i] = scaled && r < im.cnt ? __ldg(p.entry_scale + im.e0 + r) : __float2half(0.f);
            }
            bool ok = ps_wait_warp(bar_acc, (uint32_t)(n & 1), dead, 101);
            tc_fence_after();
#pragma unroll
            for (int h = 0; h < C::NPASS; ++h) {
                const int o = h / (TN / kPsRows), c0 = (h % (TN / kPsRows)) * kPsRows;
                const int f = (im.ft * C::NOUT + o) * kTcFeat + q * 32 + lane;
                uint32_t vg[16], vu[16];
                tc_ld16(trow + (uint32_t)(o * TN + c0), vg);
                if (SW) tc_ld16(trow + (uint32_t)(TN + c0), vu);
                const __half* bias = im.bias;
                const float bv = (!SW && bias && f < N) ? __half2float(__ldg(bias + f)) : 0.f;
                float nrm_g = 1.f, nrm_u = 1.f;     // codebook format: per-row norms, in tile order
                if constexpr (!AFFINE) {
                    if (f < N) {
                        const int t16 = f >> 4, r16 = f & 15;
                        nrm_g = __ldg(im.norms + (size_t)(SW ? 2 * t16 : t16) * 16 + r16);
                        if (SW) nrm_u = __ldg(im.norms + (size_t)(2 * t16 + 1) * 16 + r16);
                    }
                }
                const int b = pass & 1;
                if (pass > 1) ok = ps_wait_warp(bar_stored + 8 * b, (uint32_t)((pass >> 1) & 1) ^ 1u, dead, 106) && ok;
                tc_ld_wait();
                if (h == C::NPASS - 1) {            // the accumulator is in registers: the next item's products may start
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar_acc_free);
                }
                const uint32_t dst = orow + (uint32_t)(b * kPsOut);
                const int live = im.cnt - (im.lt * TN + c0 + part * 16);       // tokens of this warp's 16 that exist
                const float scv = __half2float(sc_h[h % (TN / kPsRows)]);
                if (ok && live > 0) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        if (j >= live) break;
                        float v = __uint_as_float(vg[j]);
                        if constexpr (!AFFINE) v *= nrm_g;
                        if constexpr (SW) {
                            float u = __uint_as_float(vu[j]);
                            if constexpr (!AFFINE) u *= nrm_u;
                            v = silu16(round16(v)) * round16(u);
                        } else {
                            if (bias) v = round16(v) + bv;
                            if (scaled) v = __shfl_sync(0xffffffffu, scv, j) * round16(v);
                        }
                        const unsigned short hv = __half_as_ushort(__float2half_rn(v));
                        asm volatile("st.shared.u16 [%0], %1;" ::"r"(dst + (uint32_t)j * 256u), "h"(hv) : "memory");
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_staged + 8 * b);
                ++pass;
            }
            release_item(n);
            return ok;
        };

        // ---- codes: requested D stages ahead (the first ones of an item before the previous item's epilogue).  Lane (g, t)
        // holds rows g and g + 8 of its tile.  Half h of the channels: Q2/T2 word h of its own 16 bytes' rows, Q4 a word of each
        // of the four lanes of its row in k block h (see tc_ts_channel_of).
        // (D <= S: the stages of a group find room in the ring before the results of the item before are taken)
        constexpr int WPR = PsUnpack<FMT>::WORDS;                  // words per half and row
        constexpr int D0 = (HALVES == 2 ? 3 : 4) - (FMT == GLQ_FMT_Q4 ? 1 : 0), D = D0 < S ? D0 : S;
        constexpr int NSZ = FMT == GLQ_FMT_Q4 ? HALVES : 1;        // (scale, zero) sets per stage
        uint32_t cq[D][HALVES][2][WPR], csz[D][NSZ][2];              // [stage][half][row][word]
        const unsigned char* blk = nullptr;                        // of the next stage to request
        int left = 0;                                              // k blocks of the item still to request
        bool live = false;
        auto fetch = [&](uint32_t (&qv)[HALVES][2][WPR], uint32_t (&zv)[NSZ][2]) {
            if constexpr (FMT == GLQ_FMT_Q4) {
#pragma unroll
                for (int h = 0; h < HALVES; ++h) {
                    const bool in = wh0 + h < left;
                    const unsigned char* src = blk + (wh0 + h) * (2 * BB);
                    const uint32_t* wsrc = reinterpret_cast<const uint32_t*>(src) + g * 16 + (t >> 1);
#pragma unroll
                    for (int n = 0; n < 4; ++n) {
                        qv[h][0][n] = in ? __ldg(wsrc + 4 * n) : 0u;
                        qv[h][1][n] = in ? __ldg(wsrc + 4 * n + 2) : 0u;
                    }
                    const uint2 z = in ? __ldg(reinterpret_cast<const uint2*>(src + 512) + g) : make_uint2(0, 0);
                    zv[h][0] = z.x, zv[h][1] = z.y;
                }
                left -= 2;
                blk += 4 * BB;
            } else {
                const bool in = left > 0;
                if constexpr (HALVES == 2) {
                    const uint4 v = in ? __ldg(reinterpret_cast<const uint4*>(blk) + lane) : make_uint4(0, 0, 0, 0);
                    qv[0][0][0] = v.x, qv[1][0][0] = v.y, qv[0][1][0] = v.z, qv[1][1][0] = v.w;
                } else {
                    const uint32_t* wsrc = reinterpret_cast<const uint32_t*>(blk) + lane * 4 + wh0;
                    qv[0][0][0] = in ? __ldg(wsrc) : 0u;
                    qv[0][1][0] = in ? __ldg(wsrc + 2) : 0u;
                }
                if constexpr (AFFINE) {
                    const uint2 z = in ? __ldg(reinterpret_cast<const uint2*>(blk + 512) + g) : make_uint2(0, 0);
                    zv[0][0] = z.x, zv[0][1] = z.y;
                }
                --left;
                blk += 2 * BB;
            }
        };
        uint32_t TL = 0, TH = 0;                  // codebook tables
        // tile of the matrix (destination tile of the fused layout for gate|up) that this warp unpacks in an item
        auto tile_of = [&](int ft) { return SW ? (ft * 8 + tl) * 2 + mx : (ft * NM + mx) * 8 + tl; };
        const int n_tiles = SW ? 2 * ((N + 15) / 16) : (N + 15) / 16;
        auto open_item = [&](int n) {
            const volatile PsItem& im = s_item[n % kPsQueue];
            const int d16 = tile_of(im.ft);
            live = d16 < n_tiles;
            left = live ? nblk : 0;
            blk = im.codes + ((size_t)(d16 >> 1) * nblk * 2 + (d16 & 1)) * BB;
            if constexpr (!AFFINE) make_t2_tables(im.centroids + (SW ? 4 * mx : 0), TL, TH);
#pragma unroll
            for (int d = 0; d < D; ++d) fetch(cq[d], csz[d]);
            // the low-rank rows come last: into L2 by then (each lane one of its 128-byte rows)
            if (live && im.sv && lane < 16)
                for (int sl = 0; sl < nst - p.nkb; ++sl)
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(im.sv + ((((size_t)(d16 >> 1) * p.ns + sl) * 32) + (d16 & 1) * 16 + lane) * 128));
        };
        // the 16 registers of a half's store: for k step n of the half {row g: positions 4t..4t+3, row g+8: the same}
        PsQ2 q2{};                                // of the stage in work (2-bit codes)
        auto unpack = [&](const uint32_t (&qv)[2][WPR], const uint32_t (&zv)[2], uint32_t (&r)[16], bool first) {
            if constexpr (FMT == GLQ_FMT_Q2) {
                if (first) q2 = ps_q2_setup(zv);
                if (q2.fast) ps_q2_fast(qv, q2, r);
                else ps_affine<FMT>(qv, zv, 0, r);
            } else if constexpr (AFFINE) {
                ps_affine<FMT>(qv, zv, 8 * (t & 1), r);
            } else {
#pragma unroll
                for (int hrow = 0; hrow < 2; ++hrow) {
                    uint32_t h[8];
                    unpack_t2(qv[hrow][0], TL, TH, h);
#pragma unroll
                    for (int j = 0; j < 8; ++j) r[4 * (j >> 1) + 2 * hrow + (j & 1)] = h[j];
                }
            }
        };
        // low-rank slice sl: SV rows in natural K order, four k steps per 64 columns
        auto load_sv = [&](const volatile PsItem& im, int sl, uint32_t (&v)[HALVES][8]) {
            const int d16 = tile_of(im.ft);
            const unsigned char* sv = im.sv;
#pragma unroll
            for (int h = 0; h < HALVES; ++h)
#pragma unroll
                for (int n = 0; n < 2; ++n)
#pragma unroll
                    for (int hrow = 0; hrow < 2; ++hrow) {
                        const int row = g + 8 * hrow;
                        const uint2* src = reinterpret_cast<const uint2*>(
                            sv + ((((size_t)(d16 >> 1) * p.ns + sl) * 32) + (d16 & 1) * 16 + row) * 128 + (2 * (wh0 + h) + n) * 32 + t * 8);
                        uint2 u = (live && sv) ? __ldg(src) : make_uint2(0, 0);
                        if constexpr (!AFFINE) {
                            // the epilogue scales by the row norm: the low-rank rows go in divided by it
                            const float nv = live ? __ldg(im.norms + (size_t)d16 * 16 + row) : 0.f;
                            const float inv = nv != 0.f ? 1.f / nv : 0.f;
                            __half2* hp = reinterpret_cast<__half2*>(&u);
#pragma unroll
                            for (int i = 0; i < 2; ++i) {
                                const float2 f = __half22float2(hp[i]);
                                hp[i] = __floats2half2_rn(f.x * inv, f.y * inv);
                            }
                        }
                        v[h][4 * n + 2 * hrow] = u.x;
                        v[h][4 * n + 2 * hrow + 1] = u.y;
                    }
        };
        const int n_sv = nst - p.nkb;
        auto publish_stage = [&]() {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_full + 8 * s);
            if (++s == S) {
                s = 0;
                ph ^= 1u;
            }
        };

        bool ok = true, more = have_item(0), pending = false;      // pending: the results of the item before are still to be taken
        if (more) open_item(0);
        for (int it = 0; more || pending; ++it) {
            const volatile PsItem& im = s_item[it % kPsQueue];
            const int nk = more ? p.nkb : 0;
            // Software pipeline: a stage's first half is unpacked while the stores of the stage before are on their way to
            // tensor memory, and before its ring slot is free.
            uint32_t r[16];
            unpack(cq[0][0], csz[0][0], r, true);
            for (int st0 = 0;; st0 += D) {
                if (pending && (st0 > 0 || nk == 0)) {
                    ok = results(it - 1) && ok;
                    pending = false;
                }
                if (st0 >= nk) break;
#pragma unroll
                for (int d = 0; d < D; ++d) {
                    const int st = st0 + d;
                    if (st < nk) {
                        ok = ps_wait_warp(bar_empty + 8 * s, ph ^ 1u, dead, 100) && ok;
                        tc_fence_after();
                        if (ok) {
                            const uint32_t acol = ring + (uint32_t)(s * NM * 64 + mx * 64 + wh0 * 32) + lane_base;
                            tc_st_x4(acol, r);
                            if constexpr (HALVES == 2) {
                                uint32_t r2[16];
                                unpack(cq[d][1], csz[d][NSZ - 1], r2, false);
                                tc_st_x4(acol + 32, r2);
                            }
                            fetch(cq[d], csz[d]);
                            unpack(cq[(d + 1) % D][0], csz[(d + 1) % D][0], r, true);
                            tc_st_wait();
                        }
                        publish_stage();
                    }
                }
            }
            if (!more) break;
            for (int sl = 0; sl < n_sv; ++sl) {
                uint32_t v[HALVES][8];
                load_sv(im, sl, v);
                ok = ps_wait_warp(bar_empty + 8 * s, ph ^ 1u, dead, 100) && ok;
                tc_fence_after();
                if (ok) {
#pragma unroll
                    for (int h = 0; h < HALVES; ++h)
                        tc_st_x2(ring + (uint32_t)(s * NM * 64 + mx * 64 + (wh0 + h) * 16) + lane_base, v[h]);
                    tc_st_wait();
                }
                publish_stage();
            }
            if (!ok) break;
            pending = true;
            more = have_item(it + 1);
            if (more) open_item(it + 1);
        }
        tc_fence_before();
    } else {
    if constexpr (C::SHIFT_REGS) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kPsRegsOther));
    if (warp == kTcProducers) {
        // ================= MMA issuer =================
        constexpr uint32_t idesc = tc_idesc(TN);
        constexpr uint32_t kAtom = TN * 128 / 16;            // an atom of the token operand in descriptor units
        const uint64_t bdesc0 = tc_smem_desc(sbase);
        int s = 0;
        uint32_t ph = 0;
        bool ok = true;
        for (int it = 0; ok; ++it) {
            const bool more = have_item(it);
            release_item(it);
            if (!more) break;
            for (int st = 0; st < nst && ok; ++st) {
                ok = ps_wait_warp(bar_full + 8 * s, ph, dead, 103);
                if (ok && st == 0 && it > 0) ok = ps_wait_warp(bar_acc_free, (uint32_t)((it - 1) & 1), dead, 104);
                if (!ok) break;
                tc_fence_after();
                const uint32_t acol = ring + (uint32_t)(s * NM * 64);
                const uint64_t bd = bdesc0 + (uint32_t)(s * (C::B_BYTES / 16));
                if (st < p.nkb) {
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const uint32_t acc = h == 0 ? (uint32_t)(st != 0) : 1u;
                        tc_mma4_f16_ts(tmem, acol + 32 * h, bd + (uint32_t)(h * kAtom), idesc, acc);
                        if (NM == 2) tc_mma4_f16_ts(tmem + TN, acol + 64 + 32 * h, bd + (uint32_t)(h * kAtom), idesc, acc);
                    }
                } else {
                    tc_mma4_f16_ts(tmem, acol, bd, idesc, 1);
                    if (NM == 2) tc_mma4_f16_ts(tmem + TN, acol + 64, bd + (SW ? kAtom : 0), idesc, 1);
                }
                tc_commit_warp(bar_empty + 8 * s);
                if (++s == S) {
                    s = 0;
                    ph ^= 1u;
                }
            }
            if (ok) tc_commit_warp(bar_acc);
        }
    } else if (warp == kTcProducers + 1) {
        // ================= results: staging tiles -> y, 16 bytes per lane, two token rows at a time =================
        int pass = 0;
        for (int it = 0; have_item(it); ++it) {
            const volatile PsItem& im = s_item[it % kPsQueue];
            const int ft = im.ft, lt = im.lt, cnt = im.cnt, e0 = im.e0;
            bool ok = true;
            for (int h = 0; h < C::NPASS && ok; ++h, ++pass) {
                const int b = pass & 1, f0 = (ft * C::NOUT + h / (TN / kPsRows)) * kTcFeat, nf = min(kTcFeat, N - f0);
                const int r0 = lt * TN + (h % (TN / kPsRows)) * kPsRows, rows = min(kPsRows, cnt - r0);
                // (the producers come to an item's results an item later: a longer limit)
                ok = __all_sync(0xffffffffu, tc_wait(bar_staged + 8 * b, (uint32_t)(pass >> 1) & 1u, dead, 107, 50000000ull));
                if (!ok) break;
                const uint32_t src = obase + (uint32_t)(b * kPsOut);
                if (nf > 0) {
                    __half* y = p.y + (size_t)(e0 + r0) * p.ldy + f0;
                    if (p.y_vec) {
                        // 16 bytes per lane, two token rows per instruction.  (A bulk copy of 256 bytes per row kept the pass
                        // 3600 cycles, 64 copies one after the other, and the tensor pipe idle behind it.)
                        const int c = lane & 15;
                        if (8 * c < nf)
#pragma unroll 8
                            for (int r = lane >> 4; r < rows; r += 2)
                                *reinterpret_cast<uint4*>(y + (size_t)r * p.ldy + 8 * c) = lds128(src + (uint32_t)(r * 256 + c * 16));
                    } else {
                        for (int r = lane; r < rows; r += 32)
                            for (int i = 0; i < nf; ++i) {
                                unsigned short hv;
                                asm volatile("ld.shared.u16 %0, [%1];" : "=h"(hv) : "r"(src + (uint32_t)r * 256u + (uint32_t)i * 2u) : "memory");
                                y[(size_t)r * p.ldy + i] = __ushort_as_half(hv);
                            }
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_stored + 8 * b);
            }
            release_item(it);
            if (!ok) break;
        }
    } else if (warp == kTcProducers + 2) {
        // ================= loader of the token operand =================
        // launched beside the pre-pass: its tiles are needed from here on (the other warps' first codes are not its work)
        int s = 0;
        uint32_t ph = 0;
        int issued = 0;
        asm volatile("griddepcontrol.wait;" ::: "memory");
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
        for (int it = 0; have_item(it); ++it) {
            const unsigned char* tile = p.xp + (size_t)static_cast<const volatile PsItem&>(s_item[it % kPsQueue]).gt * p.tile_bytes;
            release_item(it);
            if (lane == 0) {
                for (int st = 0; st < nst; ++st) {
                    if (!tc_wait(bar_empty + 8 * s, ph ^ 1u, dead, 105)) break;
                    const uint32_t bbase = sbase + (uint32_t)s * C::B_BYTES;
                    const unsigned char* src;
                    uint32_t bytes;
                    if (st < p.nkb) {
                        src = tile + (size_t)st * TN * 256;
                        bytes = TN * 256;
                    } else {
                        src = tile + (size_t)p.nkb * TN * 256 + (size_t)(st - p.nkb) * p.na * TN * 128;
                        bytes = (uint32_t)p.na * TN * 128;
                    }
                    mbar_expect_tx(bar_full + 8 * s, bytes);
                    bulk_g2s(bbase, src, bytes, bar_full + 8 * s);
                    ++issued;
                    if (++s == S) {
                        s = 0;
                        ph ^= 1u;
                    }
                }
            }
            s = __shfl_sync(0xffffffffu, s, 0);
            ph = __shfl_sync(0xffffffffu, ph, 0);
        }
        if (lane == 0 && *dead) {      // do not leave while copies are in flight
            int s2 = s;
            uint32_t ph2 = ph;
            for (int i = 0; i < S && i < issued; ++i) {
                if (--s2 < 0) {
                    s2 = S - 1;
                    ph2 ^= 1u;
                }
                const unsigned long long t0 = global_ns();
                while (!mbar_test_wait(bar_full + 8 * s2, ph2) && global_ns() - t0 < 2000000ull) __nanosleep(64);
            }
        }
        __syncwarp();
    } else {
        // ================= items: draw one (the first is the CTA's number, the others come from the grid-wide counter), look its
        // problem up, hand it out, up to kPsQueue ahead.  The loads of a look-up depend on one another, 3000 cycles in all; as a
        // part of the loader's loop they stood between the copies of two items and emptied its ring.
        bool more = true;
        for (int n = 0; more; ++n) {
            const int qi = n % kPsQueue;
            const bool room = __all_sync(0xffffffffu, tc_wait(bar_tq_empty + 8 * qi, (uint32_t)(((n / kPsQueue) & 1) ^ 1), dead, 109, 50000000ull));
            PsItem im;
            im.ft = -1;
            for (bool first = n == 0; room; first = false) {
                int w = blockIdx.x;
                if (!first) {
                    // (the pre-pass, beside which this grid is launched, zeroes the counter)
                    if (n <= 1) asm volatile("griddepcontrol.wait;" ::: "memory");
                    if (lane == 0) w = atomicAdd(p.tile_ctr, 1) + gridDim.x;
                    w = __shfl_sync(0xffffffffu, w, 0);
                }
                if (w >= n_work) break;
                const int tile = w / p.n_ft;
                int slot;
                if (tc_find_tile<TN>(p, tile, slot, im.lt, im.cnt, im.e0)) {
                    const int widx = p.slot_index ? __ldg(p.slot_index + slot) : slot;
                    const glq_weight_t* W = p.table ? p.table + widx : &p.w;
                    im.codes = reinterpret_cast<const unsigned char*>(W->codes);
                    im.sv = reinterpret_cast<const unsigned char*>(W->sv);
                    im.bias = reinterpret_cast<const __half*>(W->bias);
                    im.norms = W->norms;
                    im.centroids = W->centroids;
                    im.gt = tile;
                    im.ft = w - tile * p.n_ft;
                    break;
                }
            }
            if (lane == 0) {
                s_item[qi] = im;
                mbar_arrive(bar_tq_full + 8 * qi);
            }
            __syncwarp();
            more = im.ft >= 0;
        }
    }
    }

    __syncthreads();
    if (warp == kTcProducers) {
        tc_fence_after();
        tc_dealloc(tmem, 512);
    }
}

}  // namespace glq
