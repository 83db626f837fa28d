// Many activation rows per problem (prompts, large decode batches) on the 5th-generation tensor cores (tcgen05.mma,
// accumulators in TMEM): what its two kernels share -- the operands, the token tiles and their pre-pass, the
// primitives -- and the kernel for dense fp16 weights.  Packed codes: tc_ps.cuh.
//
//   D[feature, token] = sum_k W[feature, k] * X[token, k]
//
// The weights are the M operand ("swap AB"): an item is 128 output features of one problem and TN tokens.  The token
// operand arrives ready-made: the pre-pass (tc_pack_b_kernel) gathers the problem's activation rows and, for packed
// codes, those of x.U, orders k as the weight operand has it and writes 128-byte-swizzled tiles, so that each k stage
// is one bulk copy.  The kernel here (tc_kernel, one item per CTA) stores the tiled fp16 fragments as a K-major,
// swizzled operand in shared memory; one thread issues the MMAs, and the epilogue only rounds, applies bias and
// routing weight, and stores.
//
// k order inside a group of 16 input channels for dense weights: that of the stored fragments (lane t has channels 2t,
// 2t+1, 2t+8, 2t+9); both operands use it, so the dot products are unchanged.
//
// Every mbarrier wait is bounded (about 2 ms); a wait that runs out records error 100/101, marks the
// CTA dead, and all roles fall through to the common exit, which frees the tensor memory.
#pragma once

#include "stream_mm.cuh"

namespace glq {

constexpr int kTcFeat = 128;          // output features per CTA (UMMA M)
constexpr int kTcProducers = 16;      // producer (and epilogue) warps: 8 tiles of 16 rows x 2 row halves
constexpr int kTcThreads = (kTcProducers + 2) * 32;

struct TcParams {
    glq_weight_t w;
    const glq_weight_t* table;
    const int* slot_index;
    const int* n_slots;
    const int* slot_count;
    const int* slot_offset;
    const int* entry_row;
    const __half* entry_scale;
    const __half* x;
    long long ldx;
    const __half* a[2];
    long long lda;
    __half* y;
    long long ldy;
    unsigned char* xp;        // packed token operand: [token tile][k stages | low-rank stages]
    long long tile_bytes;     // bytes of one token tile in xp
    int n_problems, max_rows, rows_stride;
    int K, rank, nkb, ns, na; // ns: 64-wide low-rank slices, na: x.U operands per entry (1, or 2 for gate|up)
    int tiles_max;
    int fmt;                  // GLQ_FMT_*: fixes the K order of a stage
    int min_rows;             // only problems with more rows than this are this launch's
    int ts;                   // 1: K positions of a stage in the order of the tensor-memory kernel, 0: F16 fragment order
    int N, n_ft;              // output features of every problem; 128-feature tiles (persistent kernel)
    int y_vec;                // y rows allow 16-byte stores
    int x_vec16;              // x rows allow 16-byte loads
    int a_late;               // 1: a[] is written by the launch before this one, nothing else the call reads is
    int* tile_ctr;            // work-item counter of the persistent kernel (in the workspace, zeroed by the pre-pass)
};

// ---- token tile -> (problem slot, local tile) -----------------------------------------------------
// Problem p (slot position) with entries [off_p, off_p + cnt_p) owns the global token tiles
// [off_p / TN + p, off_p / TN + p + ceil(cnt_p / TN)): disjoint for consecutive problems, and at most
// total / TN + P + 1 tiles in all.  Warp-uniform result; every warp scans the (few) slots itself.
template <int TN>
__device__ __forceinline__ bool tc_find_tile(const TcParams& p, int gt, int& slot, int& lt, int& cnt, int& e0) {
    const int lane = threadIdx.x & 31;
    int P = p.n_problems;
    if (p.n_slots) P = min(P, __ldg(p.n_slots));
    for (int base = 0; base < P; base += 32) {
        const int pp = base + lane;
        int off = 0, c = 0;
        if (pp < P) {
            c = p.slot_count ? __ldg(p.slot_count + pp) : p.max_rows;
            off = p.slot_offset ? __ldg(p.slot_offset + pp) : pp * p.rows_stride;
        }
        const int start = off / TN + pp;
        const bool hit = pp < P && c > p.min_rows && gt >= start && gt < start + (c + TN - 1) / TN;
        const unsigned m = __ballot_sync(0xffffffffu, hit);
        if (m) {
            const int src = __ffs(m) - 1;
            slot = base + src;
            lt = gt - __shfl_sync(0xffffffffu, start, src);
            cnt = __shfl_sync(0xffffffffu, c, src);
            e0 = __shfl_sync(0xffffffffu, off, src);
            return true;
        }
    }
    return false;
}

// K position -> channel of the tensor-memory kernel (tc_ps.cuh).  Position P = 64*w + 16*n + 4*t + i of a 128-channel
// stage (w: producer half, n: repeat of its tensor-memory store = k step inside the half, t: lane mod 4, i: 0..3) holds
// value i & 1 of the pair 2*n + (i >> 1) that the format's unpack yields from the lane's 16 codes of that half; 4-bit: of pair
// 2*(t & 1) + (i >> 1) of word t >> 1 of the 16 consecutive channels 16*n.. of k block w, so that a k step is 16 consecutive
// channels in order (the order of the sums of the kernel for dense weights).
__host__ __device__ __forceinline__ int tc_ts_channel_of(int fmt, int P) {
    const int w = P >> 6, n = (P >> 4) & 3, t = (P >> 2) & 3, j = 2 * n + ((P >> 1) & 1), b = P & 1;
    if (fmt == GLQ_FMT_Q4) return 64 * w + 16 * n + 8 * (t >> 1) + 2 * (t & 1) + (j & 1) + 4 * b;
    const int c = fmt == GLQ_FMT_Q2 ? j + 8 * b : 4 * (j & 3) + (j >> 2) + 2 * b;
    return 32 * t + 16 * w + c;
}

// ---- pre-pass: token operand in UMMA layout ---------------------------------------------------------
// Tile layout in xp (TN rows): per k stage (128 input channels) two atoms [TN][128 B], then per
// low-rank slice `na` atoms [TN][128 B].  Inside an atom row r keeps its 16-byte chunk c at chunk
// position c ^ (r & 7) (the 128-byte swizzle).  grid = (tiles_max, nkb + ns), 256 threads.
template <int TN>
__global__ void __launch_bounds__(256) tc_pack_b_kernel(const TcParams p) {
    // Programmatic dependent launch: only the low-rank blocks read what the launch before this one writes (x.U); the blocks that
    // re-tile x run beside it.  They wait for it, so this grid ends after that one has.
    if ((int)blockIdx.y >= p.nkb || !p.a_late) asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (p.tile_ctr && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *p.tile_ctr = 0;
    int slot, lt, cnt, e0;
    if (!tc_find_tile<TN>(p, blockIdx.x, slot, lt, cnt, e0)) return;
    unsigned char* tile = p.xp + (size_t)blockIdx.x * p.tile_bytes;
    const int st = blockIdx.y;
    if (st < p.nkb && p.ts && p.x_vec16 && st * 128 + 128 <= p.K) {
        // tensor-memory order, whole stage inside K: a thread takes 16 consecutive channels (two 16-byte loads) of one
        // row.  Q2/T2: those that half w of lane t unpacks, in four 8-byte pieces, one for each of k steps 0..3 of atom w;
        // Q4: k step n of atom w, in four 8-byte pieces, one for each lane t.
        unsigned char* sdst = tile + (size_t)st * TN * 256;
#pragma unroll 2
        for (int idx = threadIdx.x; idx < TN * 8; idx += 256) {
            const int r = idx >> 3, q8 = idx & 7, t = q8 >> 1, w = q8 & 1;
            const int rr = lt * TN + r;
            uint4 lo = make_uint4(0, 0, 0, 0), hi = lo;
            if (rr < cnt) {
                const long long row = p.entry_row ? __ldg(p.entry_row + e0 + rr) : (long long)(e0 + rr);
                const uint4* src = reinterpret_cast<const uint4*>(p.x + row * p.ldx + st * 128 + (p.fmt == GLQ_FMT_Q4 ? 64 * w + 16 * t : 32 * t + 16 * w));
                lo = __ldg(src);
                hi = __ldg(src + 1);
            }
            const uint32_t a[4] = {lo.x, lo.y, lo.z, lo.w}, b[4] = {hi.x, hi.y, hi.z, hi.w};
            unsigned char* rdst = sdst + (size_t)w * (TN * 128) + (size_t)r * 128;
            if (p.fmt == GLQ_FMT_Q4) {
                // (c, c+4), (c+1, c+5): c = 0, 2 of the lower, of the upper eight channels for lanes 0..3 of step n = t
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const uint32_t(&u)[4] = h ? b : a;
                    const int c = (2 * t + h) ^ (r & 7);
                    *reinterpret_cast<uint4*>(rdst + c * 16) =
                        make_uint4(__byte_perm(u[0], u[2], 0x5410), __byte_perm(u[0], u[2], 0x7632), __byte_perm(u[1], u[3], 0x5410),
                                   __byte_perm(u[1], u[3], 0x7632));
                }
                continue;
            }
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                const int c = (2 * n + (t >> 1)) ^ (r & 7);
                uint2 v;
                if (p.fmt == GLQ_FMT_Q2) {            // (2n, 2n+8), (2n+1, 2n+9)
                    v = make_uint2(__byte_perm(a[n], b[n], 0x5410), __byte_perm(a[n], b[n], 0x7632));
                } else {                              // even (n < 2) or odd codes of eight: (c, c+2), (c+4, c+6)
                    const uint32_t(&u)[4] = n & 1 ? b : a;
                    const uint32_t sel = n < 2 ? 0x5410u : 0x7632u;
                    v = make_uint2(__byte_perm(u[0], u[1], sel), __byte_perm(u[2], u[3], sel));
                }
                *reinterpret_cast<uint2*>(rdst + (t & 1) * 8 + c * 16) = v;
            }
        }
    } else if (st < p.nkb) {
        uint4* dst = reinterpret_cast<uint4*>(tile + (size_t)st * TN * 256);
        for (int ci = threadIdx.x; ci < TN * 16; ci += 256) {
            const int atom = ci / (TN * 8), r = (ci >> 3) % TN, cpos = ci & 7;
            const int c = cpos ^ (r & 7);
            const int k0 = st * 128 + atom * 64 + (c >> 1) * 16, h = c & 1;
            const int rr = lt * TN + r;
            __align__(16) __half v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = __float2half(0.f);
            if (rr < cnt) {
                const long long row = p.entry_row ? __ldg(p.entry_row + e0 + rr) : (long long)(e0 + rr);
                const __half* src = p.x + row * p.ldx;
                if (p.ts) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int k = st * 128 + tc_ts_channel_of(p.fmt, atom * 64 + c * 8 + i);
                        if (k < p.K) v[i] = __ldg(src + k);
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int k = k0 + 2 * ((8 * h + i) >> 2) + (i & 1) + 8 * ((i >> 1) & 1);       // F16 fragment order
                        if (k < p.K) v[i] = __ldg(src + k);
                    }
                }
            }
            dst[ci] = *reinterpret_cast<const uint4*>(v);
        }
    } else {
        const int sl = st - p.nkb;
        uint4* dst = reinterpret_cast<uint4*>(tile + (size_t)p.nkb * TN * 256 + (size_t)sl * p.na * TN * 128);
        for (int ci = threadIdx.x; ci < p.na * TN * 8; ci += 256) {
            const int ai = ci / (TN * 8), r = (ci >> 3) % TN, cpos = ci & 7;
            const int c = cpos ^ (r & 7);
            const int col = sl * 64 + c * 8;
            const int rr = lt * TN + r;
            __align__(16) __half v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = __float2half(0.f);
            const __half* a = p.a[ai];
            if (rr < cnt && a != nullptr) {
                const __half* src = a + (long long)(e0 + rr) * p.lda + col;
                if (col + 8 <= p.rank) {
                    *reinterpret_cast<uint4*>(v) = __ldg(reinterpret_cast<const uint4*>(src));   // lda % 8 == 0, a 16-byte aligned
                } else {
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        if (col + i < p.rank) v[i] = __ldg(src + i);
                }
            }
            dst[ci] = *reinterpret_cast<const uint4*>(v);
        }
    }
}

// ---- tcgen05 primitives -----------------------------------------------------------------------------
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_alloc(uint32_t smem_dst, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tc_mma_f16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc)
        : "memory");
}
// 32 lanes x 16 consecutive 32-bit columns: thread i of the warp gets lane (base lane + i)
__device__ __forceinline__ void tc_ld16(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tc_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void sts128(uint32_t a, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
    asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(a), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}

// K-major operand, 128-byte swizzle: rows 128 B apart, 8-row groups 1024 B apart, version 1
__device__ __forceinline__ uint64_t tc_smem_desc(uint32_t saddr) {
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) |
           ((uint64_t)2 << 61);
}
// kind::f16: D fp32, A and B fp16, both K-major, M = 128, N = n
__host__ __device__ constexpr uint32_t tc_idesc(int n) {
    return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kTcFeat >> 4) << 24);
}

// bounded wait shared by all roles; `dead` lives in shared memory so that every role sees it
__device__ __forceinline__ bool tc_wait(uint32_t bar, uint32_t parity, volatile int* dead, int code,
                                        unsigned long long limit_ns = 2000000ull) {
    if (*dead) return false;
    if (mbar_try_wait(bar, parity)) return true;
    const unsigned long long t0 = global_ns();
    // try_wait suspends the thread in hardware for a bounded time, so a waiting warp takes no issue slots
    // from the working ones; the loop only re-arms it and enforces the overall limit
    for (bool late = false;;) {
        if (mbar_try_wait(bar, parity)) return true;
        if (*dead) return false;
        if (late) {
            glq_ok(false, code, bar, parity);
            *dead = 1;
            return false;
        }
        late = global_ns() - t0 > limit_ns;
    }
}

template <int TN> struct TcCfg {
    static constexpr int A_BYTES = kTcFeat * 256;                 // 128 rows x 128 channels fp16
    static constexpr int B_BYTES = TN * 256;
    static constexpr int STAGE = A_BYTES + B_BYTES;
    static constexpr int S = (200 * 1024) / STAGE >= 4 ? 4 : (200 * 1024) / STAGE;
    static constexpr size_t SMEM = (size_t)S * STAGE + 1024;
};

// Dense fp16 weights: the fragments are stored as a swizzled shared-memory operand, one tile per CTA.
template <int TN>
__global__ void __launch_bounds__(kTcThreads, 1) tc_kernel(const TcParams p) {
    using C = TcCfg<TN>;
    constexpr int S = C::S;
    extern __shared__ unsigned char tc_smem_raw[];
    __shared__ __align__(8) unsigned long long bars[2 * S + 1];
    __shared__ uint32_t s_tmem;
    __shared__ int s_dead;

    int slot, lt, cnt, e0;
    if (!tc_find_tile<TN>(p, blockIdx.y, slot, lt, cnt, e0)) return;    // uniform: a padding tile
    const int widx = p.slot_index ? __ldg(p.slot_index + slot) : slot;
    const glq_weight_t W = p.table ? p.table[widx] : p.w;
    const int N = W.N;
    const int ft = blockIdx.x;
    if (ft * kTcFeat >= N) return;
    const int nst = p.nkb;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t sbase = (smem_u32(tc_smem_raw) + 1023u) & ~1023u;
    const uint32_t bar_full = smem_u32(bars), bar_empty = bar_full + 8 * S, bar_acc = bar_full + 16 * S;
    volatile int* dead = &s_dead;

    if (threadIdx.x == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(bar_full + 8 * s, kTcProducers + 1);
            mbar_init(bar_empty + 8 * s, 1);
        }
        mbar_init(bar_acc, 1);
        s_dead = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kTcProducers) tc_alloc(smem_u32(&s_tmem), TN);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;

    if (warp < kTcProducers) {
        // ================= producers: the weight operand =================
        // warp = (row half, 16-row tile): lane (g, t) owns row 8*hrow + g of tile `warp & 7`
        const int g = lane >> 2, t = lane & 3;
        const int hrow = warp >> 3;
        const int tile16 = ft * 8 + (warp & 7);
        const bool live = tile16 < (N + 15) / 16;               // tiles past the matrix contribute zero rows
        constexpr int D = 2;                                    // register prefetch depth (stages of two 64-channel blocks)
        const int nblk = (p.K + 63) / 64;
        const unsigned char* blk = reinterpret_cast<const unsigned char*>(W.codes) + (size_t)tile16 * nblk * 2048;
        uint32_t cq[D][2][8];
        auto fetch = [&](int st, uint32_t (&q)[2][8]) {
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                const int kb = st * 2 + b;
                const bool in = live && st < p.nkb && kb < nblk;
                // fragment (ks, lane): words 0,2 = row g (channels 2t,2t+1 | 2t+8,2t+9), words 1,3 = row g+8
                const uint32_t* src = reinterpret_cast<const uint32_t*>(blk + (size_t)kb * 2048) + lane * 4 + hrow;
#pragma unroll
                for (int ks = 0; ks < 4; ++ks) {
                    q[b][2 * ks] = in ? __ldg(src + 128 * ks) : 0u;
                    q[b][2 * ks + 1] = in ? __ldg(src + 128 * ks + 2) : 0u;
                }
            }
        };
#pragma unroll
        for (int d = 0; d < D; ++d) fetch(d, cq[d]);

        int s = 0;
        uint32_t ph = 0;
        // this lane's row of the A tile; its swizzle key (row & 7) is g
        const uint32_t row_off = (uint32_t)((warp & 7) * 16 + hrow * 8 + g) * 128u;
        for (int st0 = 0; st0 < nst; st0 += D) {
#pragma unroll
            for (int d = 0; d < D; ++d) {
                const int st = st0 + d;
                if (st < nst) {
                    const bool ok = tc_wait(bar_empty + 8 * s, ph ^ 1u, dead, 100);
                    const uint32_t mbase = sbase + (uint32_t)s * C::STAGE + row_off;
                    if (ok) {
                        // block b = atom b; (ks, lane) holds channels 16ks + {2t, 2t+1, 2t+8, 2t+9} of its row: 8 bytes at
                        // chunk 2ks + t/2, half t%2
#pragma unroll
                        for (int b = 0; b < 2; ++b)
#pragma unroll
                            for (int ks = 0; ks < 4; ++ks) {
                                const uint32_t a = mbase + (uint32_t)b * (kTcFeat * 128) +
                                                   (uint32_t)((2 * ks + (t >> 1)) ^ g) * 16u + (uint32_t)(t & 1) * 8u;
                                asm volatile("st.shared.v2.u32 [%0], {%1,%2};" ::"r"(a), "r"(cq[d][b][2 * ks]), "r"(cq[d][b][2 * ks + 1])
                                             : "memory");
                            }
                        fetch(st + D, cq[d]);
                    }
                    fence_async_smem();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar_full + 8 * s);
                    if (++s == S) {
                        s = 0;
                        ph ^= 1u;
                    }
                }
            }
        }
        // ================= epilogue: TMEM -> registers -> global =================
        const bool acc_ok = tc_wait(bar_acc, 0, dead, 101);
        tc_fence_after();
        const int q = warp & 3, part = warp >> 2;      // TMEM lane quarter, quarter of the token columns
        const int f = ft * kTcFeat + q * 32 + lane;
        const uint32_t trow = tmem + ((uint32_t)(q * 32) << 16);
        const __half* bias = reinterpret_cast<const __half*>(W.bias);
        const float bv = (bias && f < N) ? __half2float(__ldg(bias + f)) : 0.f;
        for (int c0 = part * (TN / 4); c0 < (part + 1) * (TN / 4); c0 += 16) {
            uint32_t vg[16];
            tc_ld16(trow + (uint32_t)c0, vg);
            tc_ld_wait();
            if (acc_ok && f < N) {
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const int rr = lt * TN + c0 + j;
                    if (rr < cnt) {
                        float v = round16(__uint_as_float(vg[j]));
                        if (bias) v = round16(v + bv);
                        if (p.entry_scale) v = round16(__half2float(__ldg(p.entry_scale + e0 + rr)) * v);
                        p.y[(size_t)(e0 + rr) * p.ldy + f] = __float2half_rn(v);
                    }
                }
            }
        }
        tc_fence_before();
    } else if (warp == kTcProducers) {
        // ================= MMA issuer =================
        if (lane == 0) {
            constexpr uint32_t idesc = tc_idesc(TN);
            int s = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int st = 0; st < nst && ok; ++st) {
                ok = tc_wait(bar_full + 8 * s, ph, dead, 100);
                if (!ok) break;
                tc_fence_after();
                const uint32_t abase = sbase + (uint32_t)s * C::STAGE, bbase = abase + C::A_BYTES;
#pragma unroll
                for (int kk = 0; kk < 8; ++kk) {
                    const uint32_t ao = (uint32_t)(kk >> 2) * (kTcFeat * 128) + (uint32_t)(kk & 3) * 32u;
                    const uint32_t bo = (uint32_t)(kk >> 2) * (TN * 128) + (uint32_t)(kk & 3) * 32u;
                    tc_mma_f16(tmem, tc_smem_desc(abase + ao), tc_smem_desc(bbase + bo), idesc, (st | kk) != 0);
                }
                tc_commit(bar_empty + 8 * s);
                if (++s == S) {
                    s = 0;
                    ph ^= 1u;
                }
            }
            if (ok) tc_commit(bar_acc);
        }
        __syncwarp();
    } else {
        // ================= loader of the token operand =================
        if (lane == 0) {
            const unsigned char* tile = p.xp + (size_t)blockIdx.y * p.tile_bytes;
            int s = 0;
            uint32_t ph = 0;
            int issued = 0;
            for (int st = 0; st < nst; ++st) {
                if (!tc_wait(bar_empty + 8 * s, ph ^ 1u, dead, 100)) break;
                const uint32_t bbase = sbase + (uint32_t)s * C::STAGE + C::A_BYTES;
                mbar_expect_tx(bar_full + 8 * s, TN * 256);
                bulk_g2s(bbase, tile + (size_t)st * TN * 256, TN * 256, bar_full + 8 * s);
                ++issued;
                if (++s == S) {
                    s = 0;
                    ph ^= 1u;
                }
            }
            // a CTA that gave up must not leave while its copies are in flight: wait (bounded) for the
            // barriers of the last copies issued
            if (*dead) {
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
        }
        __syncwarp();
    }

    __syncthreads();
    if (warp == kTcProducers) {
        tc_fence_after();
        tc_dealloc(tmem, TN);
    }
}

}  // namespace glq
