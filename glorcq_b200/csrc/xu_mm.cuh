// Dense skinny product y = x . W^T of more than 32 rows with few output columns (N <= 512): the x.U and h.U products of
// the low-rank terms and the router of a prompt.
//
// What bounds it: one pass over the rows of x (and over W, which stays in L2).  The tcgen05 kernel (tc_mm.cuh) gives a
// product with 64 columns ONE 128-feature tile per 128 rows -- three CTAs for 333 rows -- whose producers set the pace
// (0.9 us per 128 channels), after a pre-pass that re-tiles x: 35.6 + 5.3 us for 333 x 4096 x 64, here 17.0;
// 21.6 + 6 and 12.6 in a 512-token prompt.  Stages of 64 channels paid the wait, the barrier and the first fragments' latency
// twice as often: 22.4 us, and 75 against 59 for the 65536 rows of a 4096-token prompt's h.U.
//   * a CTA owns 16 NT / 2 rows x 64 columns: four warps, each 16 columns (the M side, one operand fragment of W per step) against
//     NT tiles of 8 rows; a problem with few live rows skips whole operand tiles;
//   * x (rows gathered through entry_row, 128-byte swizzle) and the fragments of W, which are tiled in operand order, arrive by
//     cp.async in stages of 128 channels;
//   * K is walked in ascending steps of 16 into one fp32 accumulator, no splits.  That is the order of the tcgen05 kernel, and
//     m16n8k16 and tcgen05.mma round alike (no output of 1.4 million differed), so the kernels agree bit for bit and
//     a prompt's results do not depend on which one took a product.  The chain of 128 steps for 2048 channels takes
//     less time than a second launch to sum splits would.
#pragma once

#include "tc_mm.cuh"

namespace glq {

constexpr int kXuCols = 64, kXuThreads = 128;
constexpr int kXuW = 4 * 8 * 512;                             // bytes of a stage's W fragments: 4 column tiles x 8 steps
template <int NT> struct XuCfg {
    // stages: about 100 KB, two CTAs per SM -- a copy takes a microsecond to arrive, a stage's products an eighth of that
    static constexpr int ROWS = 8 * NT, X = ROWS * 256, STAGE = X + kXuW, S = NT == 4 ? 4 : 3;
    static constexpr size_t SMEM = (size_t)S * STAGE;
};

__device__ __forceinline__ void cp_async16_zfill(uint32_t dst, const void* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void ldsm_x4(uint32_t a, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}

// VEC: rows of x start on 16-byte boundaries; others are loaded value by value.
// grid = (row tiles, 64-column slices)
template <int NT, bool VEC>
__global__ void __launch_bounds__(kXuThreads) xu_kernel(const TcParams p) {
    using C = XuCfg<NT>;
    extern __shared__ __align__(128) unsigned char smem[];
    // (in this order: the pre-pass of the product that takes x.U may start beside this kernel, but after all before it)
    asm volatile("griddepcontrol.wait;\n griddepcontrol.launch_dependents;" ::: "memory");
    int slot, lt, cnt, e0;
    if (!tc_find_tile<C::ROWS>(p, blockIdx.x, slot, lt, cnt, e0)) return;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, g = lane >> 2, t = lane & 3;
    const int widx = p.slot_index ? __ldg(p.slot_index + slot) : slot;
    const glq_weight_t* W = p.table ? p.table + widx : &p.w;
    const int r0 = lt * C::ROWS, rows = min(C::ROWS, cnt - r0), nt_live = (rows + 7) >> 3;
    const int nkb = p.nkb;
    const int mt = blockIdx.y * 4 + w, n_mt = (p.N + 15) / 16;          // this warp's column tile

    // copies: thread = chunk tid & 7 of rows (tid >> 3) + 16 i; four chunks of W
    const __half* src[NT / 2];
#pragma unroll
    for (int i = 0; i < NT / 2; ++i) {
        const int r = (tid >> 3) + 16 * i;
        long long row = e0 + r0 + min(r, rows - 1);
        if (p.entry_row) row = __ldg(p.entry_row + row);
        src[i] = r < rows ? p.x + row * p.ldx + (tid & 7) * 8 : nullptr;
    }
    const unsigned char* wsrc = reinterpret_cast<const unsigned char*>(W->codes);
    const uint32_t base = smem_u32(smem);
    // stage of k blocks 2 st, 2 st + 1: two x tiles [ROWS][128 B], then per column tile the fragments of eight steps
    const int nst = (nkb + 1) / 2;
    auto issue = [&](int slot, int stg) {
        if (stg < nst) {
            const uint32_t dst = base + (uint32_t)(slot * C::STAGE);
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int kb = 2 * stg + u, k = kb * 64;
                const bool in = k + (tid & 7) * 8 < p.K;
#pragma unroll
                for (int i = 0; i < NT / 2; ++i) {
                    const int r = (tid >> 3) + 16 * i;
                    const bool ok = in && src[i] != nullptr;
                    const uint32_t d = dst + (uint32_t)(u * (C::X / 2) + r * 128 + (((tid & 7) ^ (r & 7)) << 4));
                    if constexpr (VEC) {
                        cp_async16_zfill(d, ok ? src[i] + k : p.x, ok ? 16 : 0);
                    } else {
                        __align__(16) __half v[8];
#pragma unroll
                        for (int j = 0; j < 8; ++j) v[j] = ok ? __ldg(src[i] + k + j) : __float2half(0.f);
                        const uint4 q = *reinterpret_cast<const uint4*>(v);
                        sts128(d, q.x, q.y, q.z, q.w);
                    }
                }
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    const int tile = blockIdx.y * 4 + m;
                    const bool ok = tile < n_mt && kb < nkb;
                    cp_async16_zfill(dst + C::X + (uint32_t)(m * 4096 + u * 2048 + tid * 16),
                                     wsrc + ((size_t)(ok ? tile : 0) * nkb + (ok ? kb : 0)) * 2048 + tid * 16, ok ? 16 : 0);
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float acc[NT][4];
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[n][q] = 0.f;
#pragma unroll
    for (int i = 0; i < C::S - 1; ++i) issue(i, i);
    int s = 0;
    uint4 a[2][2];
    uint32_t b[2][NT][4];
    for (int stg = 0; stg < nst; ++stg) {
        asm volatile("cp.async.wait_group %0;" ::"n"(C::S - 2) : "memory");
        __syncthreads();
        const uint32_t st = base + (uint32_t)(s * C::STAGE), wst = st + C::X + (uint32_t)(w * 4096 + lane * 16);
        auto frags = [&](int h, uint4 (&fa)[2], uint32_t (&fb)[NT][4]) {       // two steps: quarter h of the stage
            fa[0] = lds128(wst + h * 1024);
            fa[1] = lds128(wst + h * 1024 + 512);
#pragma unroll
            for (int n = 0; n < NT; ++n)
                if (n < nt_live)
                    ldsm_x4(st + (uint32_t)((h >> 1) * (C::X / 2) + (n * 8 + (lane & 7)) * 128 + (((4 * (h & 1) + (lane >> 3)) ^ (lane & 7)) << 4)), fb[n]);
        };
        frags(0, a[0], b[0]);
        issue(s == 0 ? C::S - 1 : s - 1, stg + C::S - 1);
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            if (h < 3) frags(h + 1, a[(h + 1) & 1], b[(h + 1) & 1]);
            const uint4(&fa)[2] = a[h & 1];
            const uint32_t(&fb)[NT][4] = b[h & 1];
#pragma unroll
            for (int n = 0; n < NT; ++n)
                if (n < nt_live) mma16816(acc[n], fa[0].x, fa[0].y, fa[0].z, fa[0].w, fb[n][0], fb[n][1]);
#pragma unroll
            for (int n = 0; n < NT; ++n)
                if (n < nt_live) mma16816(acc[n], fa[1].x, fa[1].y, fa[1].z, fa[1].w, fb[n][2], fb[n][3]);
        }
        s = s + 1 == C::S ? 0 : s + 1;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();

    // ---- through shared memory (row pitch 144 bytes) to 16-byte row pieces ----
    __half* out = reinterpret_cast<__half*>(smem);
    const __half* bias = reinterpret_cast<const __half*>(W->bias);
    const int n0 = mt * 16 + g;
    const float b0 = bias && n0 < p.N ? __half2float(__ldg(bias + n0)) : 0.f, b1 = bias && n0 + 8 < p.N ? __half2float(__ldg(bias + n0 + 8)) : 0.f;
#pragma unroll
    for (int n = 0; n < NT; ++n)
        if (n < nt_live)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                float v = acc[n][q];
                if (bias) v = round16(v) + (q < 2 ? b0 : b1);
                out[(n * 8 + 2 * t + (q & 1)) * 72 + w * 16 + g + 8 * (q >> 1)] = __float2half_rn(v);
            }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < NT / 2; ++i) {
        const int r = (tid >> 3) + 16 * i, c = blockIdx.y * kXuCols + (tid & 7) * 8;
        if (r >= rows) break;
        const __half* v = out + r * 72 + (tid & 7) * 8;
        __half* dst = p.y + (long long)(e0 + r0 + r) * p.ldy + c;
        if (p.y_vec && c + 8 <= p.N) {
            *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(v);
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j)
                if (c + j < p.N) dst[j] = v[j];
        }
    }
}

}  // namespace glq
