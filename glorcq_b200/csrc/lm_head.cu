// Output projection of the decoder ("lm_head"): logits = x . W^T for a dense fp16 W (V, H) kept in the
// row-major layout of the checkpoint, for the few rows of a decode step, with the greedy arg-max folded in.
// The reference leaves this product to the transformers model it wraps and takes the arg-max on the
// host side of every step (inference/graph_wrapper.py:186-208); at a vocabulary of 151936 x 2048 it
// is 622 MB per token, the largest single read of a decode step, so it is a pure HBM stream:
//   * a tile is 16 vocabulary rows; the four quarters of H are four warps, summed through shared memory in a fixed order
//     (deterministic, no atomics).  Four such groups per CTA, each with its own barrier, one CTA per SM: a group that is
//     done with its tiles holds up no other;
//   * every lane reads 16 bytes (8 consecutive channels of one row) per load, 2 D loads in flight, and the first
//     loads of a tile leave while the one before is still in use, so that sums and outputs never drain the stream
//     (a pipeline that refilled per tile: 140 us for 151936 x 2048, 79 us for 32000 x 4096);
//   * those 8 channels feed two m16n8k16 tensor-core ops as they are: the op's k index is only a
//     summation index, so the activations are read from shared memory in the matching order
//     (lane t of a 32-channel chunk takes channels 8t..8t+7) and nothing is shuffled;
//   * NT x 8 activation rows ride along as the op's columns, so that a batch reads W once per 32 rows;
//   * arg-max: every CTA keeps the best (fp16-rounded value, lowest index) per activation row, writes
//     it to the workspace, and the CTA that arrives last reduces the CTAs' candidates.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "glq_common.cuh"

using namespace glq;

namespace {

constexpr int kLmSplit = 4;                          // warps sharing one 16-row tile (quarters of H)
constexpr int kLmGroups = 4;                         // tiles in work per CTA
constexpr int kLmThreads = kLmGroups * kLmSplit * 32;
constexpr int kLmMaxRows = 32;                       // activation rows per pass of W

__device__ __forceinline__ uint4 ldg_stream(const uint4* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
    return v;
}

struct LmParams {
    const __half* x;
    long long ldx;
    const __half* W;
    int B, V, H;
    __half* logits;
    long long ldl;
    long long* argmax_out;
    float* cand_val;      // [grid][kLmMaxRows]
    int* cand_idx;        // [grid][kLmMaxRows]
    int* counter;
};

size_t lm_smem_bytes(int nt, int H) {
    return (size_t)nt * 8 * (H + 32) * 2 + (size_t)kLmGroups * (kLmSplit - 1) * nt * 32 * sizeof(float4);
}

// Bound by the read of W: 95 to 98 us for 1 row of 151936 x 2048, the rate of a plain copy (137 before); 16 rows of 32000 x 4096 55 us (148 in two
// passes), 64 of 151936 x 2048 283 us (1127 in eight).  NT 1, 2, 4: 8, 16, 32 activation rows; D: chunks of 32 channels a warp
// has in flight.  D 4 is 64 KB per SM and all that the stream needs; 6 and 8 spill and took 102 and 117 us.
template <int NT, int D>
__global__ void __launch_bounds__(kLmThreads, 1) lm_head_kernel(const LmParams p) {
    extern __shared__ __align__(16) unsigned char lm_smem[];
    // activation rows are padded by 64 bytes, so that the 16-byte reads of the lanes of a quarter warp (two
    // activation rows x four chunks) fall into distinct banks
    const int HS = p.H + 32;
    __half* xs = reinterpret_cast<__half*>(lm_smem);                                        // [8 NT][HS]
    float4* red = reinterpret_cast<float4*>(lm_smem + (size_t)NT * 8 * HS * 2);             // [groups][3][NT][32]
    __shared__ float s_best[kLmGroups][8 * NT];
    __shared__ int s_besti[kLmGroups][8 * NT];
    __shared__ int s_last;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int H = p.H, V = p.V, B = p.B;
    const int ntiles = (V + 15) / 16, stride = (int)gridDim.x * kLmGroups;
    const int tw = w / kLmSplit, s = w % kLmSplit;      // the warp's tile group, its quarter of H
    const int chunks = H / 32;                          // 32-channel chunks in H
    const int c_lo = (int)((long)s * chunks / kLmSplit), c_hi = (int)((long)(s + 1) * chunks / kLmSplit);
    red += tw * (kLmSplit - 1) * NT * 32;
    // group-major: the tiles of a last, partial round lie on all SMs
    int tile = tw * (int)gridDim.x + (int)blockIdx.x;
    // 16-byte chunk t of this quarter in the tile's rows g and g + 8
    auto row_of = [&](int tl, int r) { return reinterpret_cast<const uint4*>(p.W + (size_t)min(tl * 16 + r, V - 1) * H) + c_lo * 4 + t; };
    const uint4 *w0 = row_of(min(tile, ntiles - 1), g), *w1 = row_of(min(tile, ntiles - 1), g + 8);
    const int nc = c_hi - c_lo;
    uint4 qa[D], qb[D];
#pragma unroll
    for (int d = 0; d < D; ++d)
        if (tile < ntiles && d < nc) {
            qa[d] = ldg_stream(w0 + d * 4);
            qb[d] = ldg_stream(w1 + d * 4);
        }
    // activations, staged while the first of W are on their way: rows beyond B are zero
    for (int i = tid; i < 8 * NT * (H / 8); i += kLmThreads) {
        const int row = i / (H / 8), c = i % (H / 8);
        uint4 v = make_uint4(0, 0, 0, 0);
        if (row < B) v = *reinterpret_cast<const uint4*>(p.x + (size_t)row * p.ldx + c * 8);
        *reinterpret_cast<uint4*>(xs + (size_t)row * HS + c * 8) = v;
    }
    __syncthreads();
    // candidates of the activation rows 8 n + 2 t + e, in the lanes that own those output columns
    float best[NT][2];
    int besti[NT][2];
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int e = 0; e < 2; ++e) best[n][e] = -INFINITY, besti[n][e] = 0x7fffffff;
    const uint4* xb = reinterpret_cast<const uint4*>(xs + (size_t)g * HS) + c_lo * 4 + t;
    bool first = true;
    for (; tile < ntiles; tile += stride) {
        const int next = tile + stride;
        const uint4 *n0 = row_of(min(next, ntiles - 1), g), *n1 = row_of(min(next, ntiles - 1), g + 8);
        float acc[NT][4];
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[n][q] = 0.f;
        for (int c0 = 0; c0 < nc; c0 += D) {
            // what replaces these chunks: the next of this tile, or the first of the next tile
            const bool wrap = c0 + D >= nc;
            const uint4 *l0 = wrap ? n0 : w0 + (c0 + D) * 4, *l1 = wrap ? n1 : w1 + (c0 + D) * 4;
            const int left = wrap ? (next < ntiles ? nc : 0) : nc - (c0 + D);
#pragma unroll
            for (int d = 0; d < D; ++d) {
                const uint4 a = qa[d], b = qb[d];
                if (d < left) {
                    qa[d] = ldg_stream(l0 + d * 4);
                    qb[d] = ldg_stream(l1 + d * 4);
                }
                if (c0 + d < nc) {
#pragma unroll
                    for (int n = 0; n < NT; ++n) {
                        const uint4 xv = xb[n * HS + (c0 + d) * 4];       // 8 rows of HS halves = HS 16-byte chunks
                        mma16816(acc[n], a.x, b.x, a.y, b.y, xv.x, xv.y);
                        mma16816(acc[n], a.z, b.z, a.w, b.w, xv.z, xv.w);
                    }
                }
            }
        }
        w0 = n0;
        w1 = n1;
        // quarters of H: fixed-order sum through shared memory (the barrier before: the last tile's sums have been read)
        if (!first) asm volatile("bar.sync %0, 128;" ::"r"(1 + tw) : "memory");
        first = false;
        if (s != 0)
#pragma unroll
            for (int n = 0; n < NT; ++n) red[((s - 1) * NT + n) * 32 + lane] = make_float4(acc[n][0], acc[n][1], acc[n][2], acc[n][3]);
        asm volatile("bar.sync %0, 128;" ::"r"(1 + tw) : "memory");
        if (s == 0) {
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                for (int s2 = 0; s2 < kLmSplit - 1; ++s2) {
                    const float4 v = red[(s2 * NT + n) * 32 + lane];
                    acc[n][0] += v.x;
                    acc[n][1] += v.y;
                    acc[n][2] += v.z;
                    acc[n][3] += v.w;
                }
                // acc[0], acc[1]: vocabulary row g, activation rows 2t, 2t+1; acc[2], acc[3]: vocabulary row g+8
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int row = 8 * n + 2 * t + e;
                    if (row >= B) continue;
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int v = tile * 16 + g + 8 * h;
                        if (v >= V) continue;
                        const __half hv = __float2half_rn(acc[n][2 * h + e]);
                        if (p.logits) p.logits[(size_t)row * p.ldl + v] = hv;
                        const float f = __half2float(hv);
                        // a value that is not a number never wins, as long as some number is there
                        if (f > best[n][e] || (f == best[n][e] && v < besti[n][e])) best[n][e] = f, besti[n][e] = v;
                    }
                }
            }
        }
    }
    if (!p.argmax_out) return;
    // the 8 lanes g of one t hold candidates of the same activation rows: reduce over g, then over the groups
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
#pragma unroll
            for (int o = 4; o < 32; o <<= 1) {
                const float ov = __shfl_xor_sync(0xffffffffu, best[n][e], o);
                const int oi = __shfl_xor_sync(0xffffffffu, besti[n][e], o);
                if (ov > best[n][e] || (ov == best[n][e] && oi < besti[n][e])) best[n][e] = ov, besti[n][e] = oi;
            }
            if (s == 0 && g == 0) {
                s_best[tw][8 * n + 2 * t + e] = best[n][e];
                s_besti[tw][8 * n + 2 * t + e] = besti[n][e];
            }
        }
    __syncthreads();
    if (tid < 8 * NT) {
        float bv = s_best[0][tid];
        int bi = s_besti[0][tid];
        for (int j = 1; j < kLmGroups; ++j) {
            const float ov = s_best[j][tid];
            const int oi = s_besti[j][tid];
            if (ov > bv || (ov == bv && oi < bi)) bv = ov, bi = oi;
        }
        __stcg(&p.cand_val[(size_t)blockIdx.x * kLmMaxRows + tid], bv);
        __stcg(&p.cand_idx[(size_t)blockIdx.x * kLmMaxRows + tid], bi);
        __threadfence();
    }
    __syncthreads();
    if (tid == 0) {
        const int old = atomicAdd(p.counter, 1);
        s_last = (old == (int)gridDim.x - 1);
        if (s_last) *p.counter = 0;      // left zero for the next call
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    // last CTA: one warp per activation row reduces the CTAs' candidates
    for (int row = w; row < B; row += kLmThreads / 32) {
        float bv = -INFINITY;
        int bi = 0x7fffffff;
        for (int c = lane; c < (int)gridDim.x; c += 32) {
            const float ov = __ldcg(&p.cand_val[(size_t)c * kLmMaxRows + row]);
            const int oi = __ldcg(&p.cand_idx[(size_t)c * kLmMaxRows + row]);
            if (ov > bv || (ov == bv && oi < bi)) bv = ov, bi = oi;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ov > bv || (ov == bv && oi < bi)) bv = ov, bi = oi;
        }
        if (lane == 0) p.argmax_out[row] = bi == 0x7fffffff ? 0 : bi;
    }
}
int lm_grid() {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)
        sms = 148;
    return sms;
}

template <int NT, int D>
int lm_pass(const LmParams& p, int grid, cudaStream_t st) {
    const size_t smem = lm_smem_bytes(NT, p.H);
    static glq::SmemLimit limit;
    if (smem > 48 * 1024 && glq::reserve_smem(reinterpret_cast<const void*>(lm_head_kernel<NT, D>), limit, smem) != cudaSuccess) return GLQ_ERR_CUDA;
    lm_head_kernel<NT, D><<<grid, kLmThreads, smem, st>>>(p);
    return cudaGetLastError() == cudaSuccess ? GLQ_OK : GLQ_ERR_CUDA;
}

}  // namespace

extern "C" size_t glq_lm_head_workspace_bytes(void) { return (size_t)lm_grid() * kLmMaxRows * (sizeof(float) + sizeof(int)); }

extern "C" int glq_lm_head_rows(const void* x, int64_t ldx, const void* W, int B, int V, int H, void* logits, int64_t ldl,
                                int64_t* argmax_out, void* workspace, size_t workspace_bytes, int32_t* counter,
                                void* stream) {
    if (!x || !W || B < 0 || V < 0 || H <= 0 || (!logits && !argmax_out)) return GLQ_ERR_ARG;
    if (B == 0 || V == 0) return GLQ_OK;
    if (H % 32 != 0 || H > 8192) return GLQ_ERR_UNSUPPORTED;
    if ((reinterpret_cast<uintptr_t>(x) & 15u) || (reinterpret_cast<uintptr_t>(W) & 15u) || ldx % 8 != 0 ||
        (reinterpret_cast<uintptr_t>(logits) & 1u) || (reinterpret_cast<uintptr_t>(argmax_out) & 7u))
        return GLQ_ERR_ALIGN;
    const int grid = std::min(lm_grid(), (V + 16 * kLmGroups - 1) / (16 * kLmGroups));
    LmParams p{};
    p.W = reinterpret_cast<const __half*>(W);
    p.ldx = ldx;
    p.V = V;
    p.H = H;
    p.ldl = ldl;
    if (argmax_out) {
        if (!workspace || workspace_bytes < glq_lm_head_workspace_bytes() || !counter) return GLQ_ERR_WORKSPACE;
        if (reinterpret_cast<uintptr_t>(workspace) & 15u) return GLQ_ERR_ALIGN;
        p.cand_val = reinterpret_cast<float*>(workspace);
        p.cand_idx = reinterpret_cast<int*>(p.cand_val + (size_t)lm_grid() * kLmMaxRows);
        p.counter = counter;
    }
    // as few passes of W as the rows that fit beside each other in shared memory allow, equally many rows in each
    int cap = 1;
    while (cap < kLmMaxRows / 8 && lm_smem_bytes(2 * cap, H) <= (size_t)220 * 1024) cap *= 2;
    const int passes = (B + 8 * cap - 1) / (8 * cap), per = (B + passes - 1) / passes;
    for (int r = 0; r < B; r += per) {
        p.B = std::min(per, B - r);
        p.x = reinterpret_cast<const __half*>(x) + (size_t)r * ldx;
        p.logits = logits ? reinterpret_cast<__half*>(logits) + (size_t)r * ldl : nullptr;
        p.argmax_out = argmax_out ? reinterpret_cast<long long*>(argmax_out) + r : nullptr;
        cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
        const int rc = p.B <= 8 ? lm_pass<1, 4>(p, grid, st) : p.B <= 16 ? lm_pass<2, 4>(p, grid, st) : lm_pass<4, 3>(p, grid, st);
        if (rc != GLQ_OK) return rc;
    }
    return GLQ_OK;
}

extern "C" int glq_lm_head(const void* x, int64_t ldx, const void* W, int B, int V, int H, void* logits, int64_t ldl,
                           int64_t* argmax_out, void* workspace, size_t workspace_bytes, int32_t* counter,
                           void* stream) {
    if (B > 8 && x && W && V > 0 && H > 0 && (logits || argmax_out)) return GLQ_ERR_UNSUPPORTED;
    return glq_lm_head_rows(x, ldx, W, B, V, H, logits, ldl, argmax_out, workspace, workspace_bytes, counter, stream);
}
