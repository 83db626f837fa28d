// Dense skinny product y = x . W^T of 9 and more rows with few output columns (N <= 512): the x.U and h.U products of
// the low-rank terms and the router.
//
// What bounds it: one pass over the rows of x (and over W, which stays in L2).  The tcgen05 kernel (tc_mm.cuh) gives a
// product with 64 columns ONE 128-feature tile per 128 rows -- three CTAs for 333 rows, each walking the whole of K, and
// a pre-pass that re-tiles x first.  Here the work is cut along rows and K instead:
//   * a CTA owns 32 rows x 64 columns; its eight warps take every eighth 64-channel block of K and meet in shared memory;
//   * when rows and columns alone leave SMs idle, a cluster of 2, 4 or 8 CTAs shares one tile's K and sums through
//     distributed shared memory -- always in the same order, no global scratch, no atomics;
//   * every warp streams its own blocks of x (32 rows x 128 B, cp.async, three stages, rows gathered through entry_row,
//     no block-wide barrier in the loop) and reads the fragments of W, which are tiled in operand order, straight from L2;
//   * m16n8k16 fp16 products, fp32 sums: W's 16 columns are the M side, 8 rows of x the N side, so a tile with few live
//     rows skips whole operand tiles.
#pragma once

#include <cooperative_groups.h>

#include "tc_mm.cuh"

namespace glq {

constexpr int kXuRows = 32, kXuCols = 64, kXuStages = 3;
constexpr int kXuStage = kXuRows * 128;                       // bytes of one warp's stage
constexpr int kXuLd = 68;                                     // row pitch of a partial tile (floats): conflict-free writes
constexpr size_t kXuSmem = (size_t)kWarpsPerCta * kXuStages * kXuStage;
static_assert((size_t)kWarpsPerCta * kXuRows * kXuLd * 4 <= kXuSmem, "partial tiles reuse the stages");

__device__ __forceinline__ void cp_async16_zfill(uint32_t dst, const void* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void ldsm_x4(uint32_t a, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}

// grid = (CTAs per tile along K = cluster, 64-column slices, row tiles)
__global__ void __launch_bounds__(kThreads, 2) xu_kernel(const TcParams p) {
    extern __shared__ __align__(128) unsigned char smem[];
    namespace cg = cooperative_groups;
    asm volatile("griddepcontrol.wait;" ::: "memory");              // no-ops for a plain launch
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    int slot, lt, cnt, e0;
    if (!tc_find_tile<kXuRows>(p, blockIdx.z, slot, lt, cnt, e0)) return;   // the same for every CTA of a cluster
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int widx = p.slot_index ? __ldg(p.slot_index + slot) : slot;
    const glq_weight_t* W = p.table ? p.table + widx : &p.w;
    const int r0 = lt * kXuRows, rows = min(kXuRows, cnt - r0), nt_live = (rows + 7) >> 3;
    const int nkb = p.nkb, cs = gridDim.x, kb_lo = nkb * (int)blockIdx.x / cs, kb_hi = nkb * ((int)blockIdx.x + 1) / cs;
    const int mt0 = blockIdx.y * 4, nm = min(4, (p.N + 15) / 16 - mt0);
    const uint4* frag = reinterpret_cast<const uint4*>(W->codes) + (size_t)mt0 * nkb * 128 + lane;   // 4 x 32 uint4 per block

    // this lane copies chunk lane & 7 of rows (lane >> 3) + 4 i
    const __half* src[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int r = (lane >> 3) + 4 * i;
        long long row = e0 + r0 + min(r, rows - 1);
        if (p.entry_row) row = __ldg(p.entry_row + row);
        src[i] = r < rows ? p.x + row * p.ldx + (lane & 7) * 8 : nullptr;
    }
    const uint32_t stage0 = smem_u32(smem) + (uint32_t)w * (kXuStages * kXuStage);
    auto issue = [&](int s, int kb) {
        if (kb < kb_hi) {
            const int k = kb * 64;
            const bool in = k + (lane & 7) * 8 < p.K;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                if (i >= 2 * nt_live) break;
                const int r = (lane >> 3) + 4 * i;
                const bool ok = in && src[i] != nullptr;
                cp_async16_zfill(stage0 + (uint32_t)(s * kXuStage + r * 128 + (((lane & 7) ^ (r & 7)) << 4)), ok ? src[i] + k : p.x, ok ? 16 : 0);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float acc[4][4][4];
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int n = 0; n < 4; ++n)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[m][n][q] = 0.f;
    uint4 a[2][4];      // the fragments of a step are requested one step ahead
    auto load_a = [&](int kb, int ks, uint4 (&dst)[4]) {
#pragma unroll
        for (int m = 0; m < 4; ++m)
            dst[m] = (m < nm && kb < kb_hi) ? __ldg(frag + ((size_t)m * nkb + kb) * 128 + ks * 32) : make_uint4(0, 0, 0, 0);
    };
    int kb = kb_lo + w;
#pragma unroll
    for (int s = 0; s < kXuStages - 1; ++s) issue(s, kb + s * kWarpsPerCta);
    load_a(kb, 0, a[0]);
    int s = 0;
    for (; kb < kb_hi; kb += kWarpsPerCta) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kXuStages - 2) : "memory");
        __syncwarp();
        issue(s == 0 ? kXuStages - 1 : s - 1, kb + (kXuStages - 1) * kWarpsPerCta);
        const uint32_t st = stage0 + (uint32_t)(s * kXuStage);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            uint32_t b[4][4];
#pragma unroll
            for (int n = 0; n < 4; ++n)
                if (n < nt_live) ldsm_x4(st + (uint32_t)((n * 8 + (lane & 7)) * 128 + (((4 * h + (lane >> 3)) ^ (lane & 7)) << 4)), b[n]);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int ks = 2 * h + e;
                if (ks < 3) load_a(kb, ks + 1, a[(ks + 1) & 1]);
                else load_a(kb + kWarpsPerCta, 0, a[0]);
#pragma unroll
                for (int n = 0; n < 4; ++n)
                    if (n < nt_live)
#pragma unroll
                        for (int m = 0; m < 4; ++m)
                            mma16816(acc[m][n], a[ks & 1][m].x, a[ks & 1][m].y, a[ks & 1][m].z, a[ks & 1][m].w, b[n][2 * e], b[n][2 * e + 1]);
            }
        }
        __syncwarp();
        s = s + 1 == kXuStages ? 0 : s + 1;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();

    // ---- sum of the warps, then of the cluster's CTAs, in fixed order ----
    float* part = reinterpret_cast<float*>(smem);
#pragma unroll
    for (int n = 0; n < 4; ++n)
        if (n < nt_live)
#pragma unroll
            for (int m = 0; m < 4; ++m)
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    part[(w * kXuRows + n * 8 + 2 * t + (q & 1)) * kXuLd + m * 16 + g + 8 * (q >> 1)] = acc[m][n][q];
    __syncthreads();
    const int row = threadIdx.x >> 3, c0 = (threadIdx.x & 7) * 8;     // this thread: 8 columns of a row
    float v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = 0.f;
    if (row < nt_live * 8)
#pragma unroll
        for (int i = 0; i < kWarpsPerCta; ++i) {
            const float4* q = reinterpret_cast<const float4*>(part + (i * kXuRows + row) * kXuLd + c0);
            const float4 lo = q[0], hi = q[1];
            v[0] += lo.x; v[1] += lo.y; v[2] += lo.z; v[3] += lo.w;
            v[4] += hi.x; v[5] += hi.y; v[6] += hi.z; v[7] += hi.w;
        }
    bool mine = true;
    if (cs > 1) {
        cg::cluster_group cl = cg::this_cluster();
        // (each thread overwrites words of partial tile 0 that only it has read)
        float4* own = reinterpret_cast<float4*>(part + row * kXuLd + c0);
        own[0] = make_float4(v[0], v[1], v[2], v[3]);
        own[1] = make_float4(v[4], v[5], v[6], v[7]);
        cl.sync();
        mine = row % cs == (int)blockIdx.x;
        if (mine) {
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = 0.f;
            for (int c = 0; c < cs; ++c) {
                const float4* q = reinterpret_cast<const float4*>(cl.map_shared_rank(part, c) + row * kXuLd + c0);
                const float4 lo = q[0], hi = q[1];
                v[0] += lo.x; v[1] += lo.y; v[2] += lo.z; v[3] += lo.w;
                v[4] += hi.x; v[5] += hi.y; v[6] += hi.z; v[7] += hi.w;
            }
        }
        cl.sync();      // no CTA leaves while another reads its tile
    }
    if (!mine || row >= rows) return;
    const int n0 = blockIdx.y * kXuCols + c0;
    __half* dst = p.y + (long long)(e0 + r0 + row) * p.ldy + n0;
    const __half* bias = reinterpret_cast<const __half*>(W->bias);
    __align__(16) __half o[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        o[j] = __float2half_rn(v[j]);
        if (bias && n0 + j < p.N) o[j] = __float2half_rn(__half2float(o[j]) + __half2float(__ldg(bias + n0 + j)));
    }
    if (p.y_vec && n0 + 8 <= p.N) {
        *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(o);
    } else {
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (n0 + j < p.N) dst[j] = o[j];
    }
}

}  // namespace glq
