// One decode step of grouped-query attention over a static key/value cache, in one launch: optional
// per-head RMS norm of q and k, rotary embedding (rotate-half convention) of q and of the new key at
// the current position, cache write, softmax(q k^T / sqrt(hd)) v over positions 0..pos.
// The position is read from device memory, so a captured launch serves every step of a replayed graph
// and only the live part of the cache is read.  Host model code around the quantized projections
// (inference/graph_wrapper.py:84-127 drives the transformers attention modules for this).
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstdlib>

#include "glq_common.cuh"

using namespace glq;

namespace {

constexpr int kAttnWarps = 8;

// EPL: head_dim / 32 elements per lane; lane l owns elements [l*EPL, (l+1)*EPL); its rotate-half partner
// (element +- hd/2) sits in lane l ^ 16 at the same offset.
template <int EPL>
__device__ __forceinline__ void rope_norm(float (&v)[EPL], const __half* __restrict__ norm_w, float eps, int hd,
                                          const float (&c)[EPL], const float (&sn)[EPL], int lane) {
    if (norm_w) {   // RMS norm over the head, weight applied, rounded to fp16 as a tensor op does
        float ss = 0.f;
#pragma unroll
        for (int i = 0; i < EPL; ++i) ss += v[i] * v[i];
        ss = warp_sum(ss);
        const float r = rsqrtf(ss / hd + eps);
#pragma unroll
        for (int i = 0; i < EPL; ++i) v[i] = round16(__half2float(norm_w[lane * EPL + i]) * (v[i] * r));
    }
#pragma unroll
    for (int i = 0; i < EPL; ++i) {
        const float partner = __shfl_xor_sync(0xffffffffu, v[i], 16);
        const float rot = lane < 16 ? -partner : partner;          // rotate_half: (-x2, x1)
        v[i] = round16(round16(v[i] * c[i]) + round16(rot * sn[i]));
    }
}

// EPL consecutive values of a row; vec: every row starts at an 8-byte boundary
template <int EPL>
__device__ __forceinline__ void load_row(const __half* p, bool vec, __half (&h)[EPL]) {
    if (EPL == 4 && vec) *reinterpret_cast<uint2*>(h) = *reinterpret_cast<const uint2*>(p);
    else
#pragma unroll
        for (int i = 0; i < EPL; ++i) h[i] = p[i];
}
template <int EPL>
__device__ __forceinline__ void store_row(__half* p, bool vec, const __half (&h)[EPL]) {
    if (EPL == 4 && vec) *reinterpret_cast<uint2*>(p) = *reinterpret_cast<const uint2*>(h);
    else
#pragma unroll
        for (int i = 0; i < EPL; ++i) p[i] = h[i];
}

// What bounds it: the wait for the cached rows, at one CTA per SM (few heads; issue slots 22 % used) as at the two that
// registers allow (16 sequences of 32 heads; 45 %, a quarter of the HBM rate).  One position at a time, every score
// waited for five shuffles and every update for two exponentials.  Now eight positions make one step: their partial scores are
// summed by a transposing butterfly (the same pairs of lanes in the same order, so the same bits), the running maximum is
// a scan, each exponential is taken once per position instead of by every lane, only l and o are chains, and the rows of
// the next step are requested before this one's are used.  G = 2 heads that share their keys and values read and convert
// them once.  16 x 32 heads x 1024 positions, 8 key heads: 72 -> 40 us (46 with rows selected by 64-bit positions, 74 with one
// head per CTA); 9 x 32 x 500: 25 -> 15; 16 heads x 512 in a decode step: 8.2 -> 7.5; 64 x 16 x 300 without sharing: 45 -> 42
// (four CTAs per SM: with three, 46).  G = 4 leaves too few warps: 64 x 32 x 500 took 82 us, 75 with G = 2, 97 before.
template <int EPL, int G>
__global__ void __launch_bounds__(kAttnWarps * 32, EPL == 4 && G == 1 ? 4 : 1) attn_decode_kernel(
    const __half* __restrict__ q, const __half* __restrict__ k_new, const __half* __restrict__ v_new,
    const __half* __restrict__ cos_t, const __half* __restrict__ sin_t, const long long* __restrict__ pos_p,
    __half* __restrict__ k_cache, __half* __restrict__ v_cache, __half* __restrict__ out, int n_heads, int n_kv, int max_len,
    const __half* __restrict__ q_norm_w, const __half* __restrict__ k_norm_w, float eps, float* __restrict__ partial,
    int* __restrict__ arrivals) {
    constexpr int HD = EPL * 32;
    const int h = blockIdx.x * G, b = blockIdx.y, z = blockIdx.z, nsplit = gridDim.z;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int group = n_heads / n_kv, kvh = h / group;
    __half* kc = k_cache + ((size_t)b * n_kv + kvh) * max_len * HD;
    __half* vc = v_cache + ((size_t)b * n_kv + kvh) * max_len * HD;
    // (launched plainly, after all before it: in the places that the projections leave free beside them the CTAs would lie two to an SM,
    // 8.9 us instead of 7.5; the output projection behind it may fetch its first weights meanwhile)
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    long long pos = *pos_p;
    if (pos < 0) pos = 0;
    if (pos >= max_len) pos = max_len - 1;
    // this CTA's share of the cached positions (the grid's z dimension splits them), interleaved over its warps; a step is
    // kAhead of a warp's positions, its keys and values at constant distances from one row
    const int per = ((int)pos + nsplit - 1) / nsplit;
    const int t_lo = z * per, t_hi = min(t_lo + per, (int)pos);
    constexpr int kAhead = 8;
    __half kr[kAhead][EPL], vr[kAhead][EPL];
    auto live_from = [&](int t0) { return t0 < t_hi ? min(kAhead, (t_hi - t0 + kAttnWarps - 1) / kAttnWarps) : 0; };
    // rows of the step at t0: n of them
    auto request = [&](const __half* cache, int t0, int n, __half (&r)[kAhead][EPL]) {
        const __half* row = cache + (size_t)t0 * HD + lane * EPL;
        if (n == kAhead) {
#pragma unroll
            for (int u = 0; u < kAhead; ++u) load_row<EPL>(row + u * (kAttnWarps * HD), true, r[u]);
        } else {
#pragma unroll
            for (int u = 0; u < kAhead; ++u)
                if (u < n) load_row<EPL>(row + u * (kAttnWarps * HD), true, r[u]);
        }
    };
    int nv = live_from(t_lo + warp);
    request(kc, t_lo + warp, nv, kr);
    request(vc, t_lo + warp, nv, vr);
    float cs[EPL], sn[EPL];
#pragma unroll
    for (int i = 0; i < EPL; ++i) {
        cs[i] = __half2float(cos_t[(size_t)pos * HD + lane * EPL + i]);
        sn[i] = __half2float(sin_t[(size_t)pos * HD + lane * EPL + i]);
    }

    float qv[G][EPL], kn[EPL], vn[EPL];
#pragma unroll
    for (int i = 0; i < EPL; ++i) {
#pragma unroll
        for (int j = 0; j < G; ++j) qv[j][i] = __half2float(q[((size_t)b * n_heads + h + j) * HD + lane * EPL + i]);
        kn[i] = __half2float(k_new[((size_t)b * n_kv + kvh) * HD + lane * EPL + i]);
        vn[i] = __half2float(v_new[((size_t)b * n_kv + kvh) * HD + lane * EPL + i]);
    }
#pragma unroll
    for (int j = 0; j < G; ++j) rope_norm<EPL>(qv[j], q_norm_w, eps, HD, cs, sn, lane);
    rope_norm<EPL>(kn, k_norm_w, eps, HD, cs, sn, lane);
    if (h % group == 0 && warp == 0 && z == 0) {     // one CTA per key/value head stores the new entry
#pragma unroll
        for (int i = 0; i < EPL; ++i) {
            kc[(size_t)pos * HD + lane * EPL + i] = __float2half_rn(kn[i]);
            vc[(size_t)pos * HD + lane * EPL + i] = __float2half_rn(vn[i]);
        }
    }
    const float scale = rsqrtf((float)HD);
    // online softmax per warp over its share of positions 0..pos-1 (the new position is warp 0's, from
    // registers: other CTAs of the group may not have stored it yet)
    float m[G], l[G], o[G][EPL];
#pragma unroll
    for (int j = 0; j < G; ++j) {
        m[j] = -INFINITY;
        l[j] = 0.f;
#pragma unroll
        for (int i = 0; i < EPL; ++i) o[j][i] = 0.f;
    }
    const bool b16 = (lane & 16) != 0, b8 = (lane & 8) != 0, b4 = (lane & 4) != 0;
    for (int t0 = t_lo + warp; nv > 0; t0 += kAttnWarps * kAhead) {
        const int t1 = t0 + kAttnWarps * kAhead, nv1 = live_from(t1);      // the next step
        float s[G][kAhead], ea[G], ep[G];
#pragma unroll
        for (int u = 0; u < kAhead; ++u)
#pragma unroll
            for (int j = 0; j < G; ++j) {
                s[j][u] = 0.f;
#pragma unroll
                for (int i = 0; i < EPL; ++i) s[j][u] += qv[j][i] * __half2float(kr[u][i]);
            }
        request(kc, t1, nv1, kr);
#pragma unroll
        for (int j = 0; j < G; ++j) {
            // sums over the lanes, in warp_sum's order; lanes 4 u .. 4 u + 3 end up with position u
            float r4[4], r2[2], v;
#pragma unroll
            for (int n = 0; n < 4; ++n)
                r4[n] = (b16 ? s[j][n + 4] : s[j][n]) + __shfl_xor_sync(0xffffffffu, b16 ? s[j][n] : s[j][n + 4], 16);
#pragma unroll
            for (int n = 0; n < 2; ++n) r2[n] = (b8 ? r4[n + 2] : r4[n]) + __shfl_xor_sync(0xffffffffu, b8 ? r4[n] : r4[n + 2], 8);
            v = (b4 ? r2[1] : r2[0]) + __shfl_xor_sync(0xffffffffu, b4 ? r2[0] : r2[1], 4);
            v += __shfl_xor_sync(0xffffffffu, v, 2);
            v += __shfl_xor_sync(0xffffffffu, v, 1);
            v = (lane >> 2) < nv ? v * scale : -INFINITY;
            // running maximum up to and including, and before, each position
            float mi = fmaxf(m[j], v);
#pragma unroll
            for (int d = 4; d < 32; d <<= 1) {
                const float o2 = __shfl_up_sync(0xffffffffu, mi, d);
                if (lane >= d) mi = fmaxf(mi, o2);
            }
            float mp = __shfl_up_sync(0xffffffffu, mi, 4);
            if (lane < 4) mp = m[j];
            ea[j] = __expf(mp - mi);
            ep[j] = __expf(v - mi);
            m[j] = __shfl_sync(0xffffffffu, mi, 31);
        }
        auto take = [&](int u) {
#pragma unroll
            for (int j = 0; j < G; ++j) {
                const float a = __shfl_sync(0xffffffffu, ea[j], 4 * u), p = __shfl_sync(0xffffffffu, ep[j], 4 * u);
                l[j] = l[j] * a + p;
#pragma unroll
                for (int i = 0; i < EPL; ++i) o[j][i] = o[j][i] * a + p * __half2float(vr[u][i]);
            }
        };
        if (nv == kAhead) {
#pragma unroll
            for (int u = 0; u < kAhead; ++u) take(u);
        } else {
#pragma unroll
            for (int u = 0; u < kAhead; ++u)
                if (u < nv) take(u);
        }
        request(vc, t1, nv1, vr);
        nv = nv1;
    }
    if (warp == 0 && z == 0) {
#pragma unroll
        for (int j = 0; j < G; ++j) {
            float s = 0.f;
#pragma unroll
            for (int i = 0; i < EPL; ++i) s += qv[j][i] * kn[i];
            s = warp_sum(s) * scale;
            const float mn = fmaxf(m[j], s);
            const float a = __expf(m[j] - mn), p = __expf(s - mn);
            l[j] = l[j] * a + p;
#pragma unroll
            for (int i = 0; i < EPL; ++i) o[j][i] = o[j][i] * a + p * vn[i];
            m[j] = mn;
        }
    }
    // combine the warps
    __shared__ float sm_ml[G][kAttnWarps][2], sm_ov[G][kAttnWarps][HD];
#pragma unroll
    for (int j = 0; j < G; ++j) {
        if (lane == 0) {
            sm_ml[j][warp][0] = m[j];
            sm_ml[j][warp][1] = l[j];
        }
#pragma unroll
        for (int i = 0; i < EPL; ++i) sm_ov[j][warp][lane * EPL + i] = o[j][i];
    }
    __syncthreads();
    if (warp < G) {                                  // warp j merges head j
        const int hj = h + warp;
        const float(*sm_o)[HD] = sm_ov[warp];
        const float(*ml)[2] = sm_ml[warp];
        float mm = -INFINITY;
        for (int w = 0; w < kAttnWarps; ++w) mm = fmaxf(mm, ml[w][0]);
        float ll = 0.f, oo[EPL];
#pragma unroll
        for (int i = 0; i < EPL; ++i) oo[i] = 0.f;
        for (int w = 0; w < kAttnWarps; ++w) {
            const float a = ml[w][0] == -INFINITY ? 0.f : __expf(ml[w][0] - mm);
            ll += ml[w][1] * a;
#pragma unroll
            for (int i = 0; i < EPL; ++i) oo[i] += sm_o[w][lane * EPL + i] * a;
        }
        if (nsplit == 1) {
#pragma unroll
            for (int i = 0; i < EPL; ++i) out[((size_t)b * n_heads + hj) * HD + lane * EPL + i] = __float2half_rn(oo[i] / ll);
            return;
        }
        // several CTAs per head: leave (max, sum, weighted values) of this share; the CTA that arrives last
        // (counter per head, reset by it) merges the shares in a fixed order
        float* mine = partial + (((size_t)b * n_heads + hj) * nsplit + z) * (HD + 2);
        if (lane == 0) {
            mine[0] = mm;
            mine[1] = ll;
        }
#pragma unroll
        for (int i = 0; i < EPL; ++i) mine[2 + lane * EPL + i] = oo[i];
        __threadfence();
        __syncwarp();
        int last = 0;
        if (lane == 0) last = atomicAdd(arrivals + (size_t)b * n_heads + hj, 1) == nsplit - 1;
        if (!__shfl_sync(0xffffffffu, last, 0)) return;
        __threadfence();
        const float* all = partial + ((size_t)b * n_heads + hj) * nsplit * (HD + 2);
        // (at most 16 shares: lane s2 takes the maximum and the sum of share s2)
        const float pm = lane < nsplit ? __ldcg(all + (size_t)lane * (HD + 2)) : -INFINITY;
        const float pl = lane < nsplit ? __ldcg(all + (size_t)lane * (HD + 2) + 1) : 0.f;
        float gm = pm;
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) gm = fmaxf(gm, __shfl_xor_sync(0xffffffffu, gm, d));
        const float pa = pm == -INFINITY ? 0.f : __expf(pm - gm);
        float gl = 0.f, go[EPL];
#pragma unroll
        for (int i = 0; i < EPL; ++i) go[i] = 0.f;
        for (int s0 = 0; s0 < nsplit; s0 += 8) {
            float pv[8][EPL];
#pragma unroll
            for (int u = 0; u < 8; ++u)
#pragma unroll
                for (int i = 0; i < EPL; ++i)
                    pv[u][i] = s0 + u < nsplit ? __ldcg(all + (size_t)(s0 + u) * (HD + 2) + 2 + lane * EPL + i) : 0.f;
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const float a = __shfl_sync(0xffffffffu, pa, s0 + u), ls = __shfl_sync(0xffffffffu, pl, s0 + u);
                if (s0 + u < nsplit) {
                    gl += ls * a;
#pragma unroll
                    for (int i = 0; i < EPL; ++i) go[i] += pv[u][i] * a;
                }
            }
        }
#pragma unroll
        for (int i = 0; i < EPL; ++i) out[((size_t)b * n_heads + hj) * HD + lane * EPL + i] = __float2half_rn(go[i] / gl);
        if (lane == 0) arrivals[(size_t)b * n_heads + hj] = 0;
    }
}

// The prompt's form of the first half of attn_decode_kernel: per (token, head) one warp applies the optional RMS norm
// and the rotary embedding at the token's position to q and k in place, and writes the new keys and values into the
// static cache.  Same arithmetic (rope_norm) as the decode step.  Bound by memory: one CTA per token, whose warps share the
// tables' row over their heads, 8 bytes per lane (a CTA for every eight heads with 2-byte accesses took 38 us for 4096 tokens
// of 32 + 2 x 4 heads, 29.5 now).
template <int EPL>
__global__ void __launch_bounds__(kAttnWarps * 32) rope_prefill_kernel(
    __half* __restrict__ q, __half* __restrict__ k, const __half* __restrict__ v, const __half* __restrict__ cos_t,
    const __half* __restrict__ sin_t, const long long* __restrict__ positions, __half* __restrict__ k_cache,
    __half* __restrict__ v_cache, int T, int n_heads, int n_kv, int max_len, const __half* __restrict__ q_norm_w,
    const __half* __restrict__ k_norm_w, float eps, int vec_i) {
    constexpr int HD = EPL * 32;
    const bool vec = vec_i != 0;
    const int lane = threadIdx.x & 31;
    const int bt = blockIdx.x, b = bt / T, t = bt - b * T;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    long long pos = positions[t];
    if (pos < 0) pos = 0;
    if (pos >= max_len) pos = max_len - 1;
    float cs[EPL], sn[EPL];
    {
        __half h[EPL];
        load_row<EPL>(cos_t + (size_t)pos * HD + lane * EPL, vec, h);
#pragma unroll
        for (int i = 0; i < EPL; ++i) cs[i] = __half2float(h[i]);
        load_row<EPL>(sin_t + (size_t)pos * HD + lane * EPL, vec, h);
#pragma unroll
        for (int i = 0; i < EPL; ++i) sn[i] = __half2float(h[i]);
    }
    for (int hw = threadIdx.x >> 5; hw < n_heads + 2 * n_kv; hw += kAttnWarps) {
        __half h[EPL];
        if (hw >= n_heads + n_kv) {
            const int kvh = hw - n_heads - n_kv;
            load_row<EPL>(v + ((size_t)bt * n_kv + kvh) * HD + lane * EPL, vec, h);
            store_row<EPL>(v_cache + (((size_t)b * n_kv + kvh) * max_len + pos) * HD + lane * EPL, vec, h);
            continue;
        }
        const bool is_q = hw < n_heads;
        const int kvh = hw - n_heads;
        __half* row = is_q ? q + ((size_t)bt * n_heads + hw) * HD + lane * EPL : k + ((size_t)bt * n_kv + kvh) * HD + lane * EPL;
        load_row<EPL>(row, vec, h);
        float val[EPL];
#pragma unroll
        for (int i = 0; i < EPL; ++i) val[i] = __half2float(h[i]);
        rope_norm<EPL>(val, is_q ? q_norm_w : k_norm_w, eps, HD, cs, sn, lane);
#pragma unroll
        for (int i = 0; i < EPL; ++i) h[i] = __float2half_rn(val[i]);
        store_row<EPL>(row, vec, h);
        if (!is_q) store_row<EPL>(k_cache + (((size_t)b * n_kv + kvh) * max_len + pos) * HD + lane * EPL, vec, h);
    }
}

// ---------------------------------------------------------------------------------------------
// Causal attention of a prompt written at positions 0..T-1: y[t] = softmax(q[t] . k[0..t]^T / sqrt(hd)) v[0..t] per
// (batch, head), keys and values of the head's group (grouped-query attention).  One CTA = 64 queries of one head
// (four warps x 16 rows), key blocks of 64 up to the diagonal only; scores and the weighted values on the fp16
// `mma.m16n8k16` op with fp32 accumulators, softmax in base 2 with a running row maximum and row sum in registers
// (the probabilities are rounded to fp16 as the second product's operand), key / value blocks double-buffered in
// shared memory by 16-byte asynchronous copies (rows past T arrive as zeros).  q (B, T, n_heads, HD),
// k / v (B, T, n_kv, HD), y (B, T, n_heads, HD): the layout the projections write and the output projection reads.
// (inference/graph_wrapper.py:84-127 leaves this to the transformers attention modules.)
template <int HD>
struct PrefillCfg {
    static constexpr int BM = 64, BN = 64, LD = HD + 8;          // 16-byte pad per row: conflict-free fragment reads
    static constexpr int STAGE = 2 * BN * LD;                    // halfs per stage: keys, then values
    static constexpr size_t SMEM = (size_t)2 * STAGE * sizeof(__half);
};

__device__ __forceinline__ uint32_t pf_smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp_async_16(uint32_t dst, const void* src, bool live) {
    const int bytes = live ? 16 : 0;     // 0: the 16 bytes are filled with zeros, nothing is read
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void ldsm_x4_trans(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(addr));
}
// 2^x by the special-function unit alone (2 ulp; -inf -> 0; results below the normal range flush to zero)
__device__ __forceinline__ float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ uint32_t pack_half2(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}

template <int HD>
__global__ void __launch_bounds__(128, 3) attn_prefill_kernel(const __half* __restrict__ q, const __half* __restrict__ k,
                                                           const __half* __restrict__ v, __half* __restrict__ y, int B,
                                                           int T, int n_heads, int n_kv) {
    using C = PrefillCfg<HD>;
    constexpr int LD = C::LD, KS = HD / 16, NT = HD / 8;
    extern __shared__ __align__(16) unsigned char pf_smem[];
    __half* sm = reinterpret_cast<__half*>(pf_smem);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    // launch order = work order: the query blocks with the most keys first, over all heads and batch rows
    const int n_hb = n_heads * B;
    const int qb = (int)(gridDim.x / n_hb) - 1 - (int)(blockIdx.x / n_hb);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int h = (int)(blockIdx.x % n_hb) % n_heads, b = (int)(blockIdx.x % n_hb) / n_heads;
    const int kvh = h / (n_heads / n_kv);
    const int q0 = qb * C::BM + warp * 16;                      // first query row of this warp
    const __half* kbase = k + ((size_t)b * T * n_kv + kvh) * HD;
    const __half* vbase = v + ((size_t)b * T * n_kv + kvh) * HD;
    const size_t kv_row = (size_t)n_kv * HD;

    auto load_block = [&](int kb, int stage) {
        __half* ks = sm + (size_t)stage * C::STAGE;
        __half* vs = ks + C::BN * LD;
        for (int idx = tid; idx < C::BN * (HD / 8); idx += 128) {
            const int r = idx / (HD / 8), c = idx % (HD / 8);
            const int key = kb * C::BN + r;
            const bool live = key < T;
            const size_t off = (size_t)(live ? key : 0) * kv_row + c * 8;
            cp_async_16(pf_smem_addr(ks + r * LD + c * 8), kbase + off, live);
            cp_async_16(pf_smem_addr(vs + r * LD + c * 8), vbase + off, live);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    const int nkb = qb + 1;            // key blocks 0 .. qb (BM == BN)
    load_block(0, 0);

    // the warp's 16 query rows as the first operand's fragments: rows g and g + 8, channels 16*ks + 2t (+8)
    uint32_t qf[KS][4];
    {
        const int r0 = q0 + g, r1 = q0 + g + 8;
        const __half* p0 = q + (((size_t)b * T + min(r0, T - 1)) * n_heads + h) * HD;
        const __half* p1 = q + (((size_t)b * T + min(r1, T - 1)) * n_heads + h) * HD;
#pragma unroll
        for (int ks = 0; ks < KS; ++ks) {
            qf[ks][0] = r0 < T ? *reinterpret_cast<const uint32_t*>(p0 + 16 * ks + 2 * t) : 0u;
            qf[ks][1] = r1 < T ? *reinterpret_cast<const uint32_t*>(p1 + 16 * ks + 2 * t) : 0u;
            qf[ks][2] = r0 < T ? *reinterpret_cast<const uint32_t*>(p0 + 16 * ks + 8 + 2 * t) : 0u;
            qf[ks][3] = r1 < T ? *reinterpret_cast<const uint32_t*>(p1 + 16 * ks + 8 + 2 * t) : 0u;
        }
    }
    float o[NT][4];
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[j][e] = 0.f;
    float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;     // rows g and g + 8: running maximum, this lane's share of the sum
    const float sc = rsqrtf((float)HD) * 1.4426950408889634f;     // scores in base 2

    for (int kb = 0; kb < nkb; ++kb) {
        if (kb + 1 < nkb) {
            load_block(kb + 1, (kb + 1) & 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        const __half* ks_ = sm + (size_t)(kb & 1) * C::STAGE;
        const __half* vs_ = ks_ + C::BN * LD;
        // a warp whose rows all lie before this key block has nothing to add (only in the diagonal block, never)
        float sacc[8][4];
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) sacc[j][e] = 0.f;
#pragma unroll
        for (int ks = 0; ks < KS; ++ks) {
            // keys as the second operand: 8x8 matrix loads, rows = keys (two 8-key tiles x two channel halves each)
            const int krow = (lane & 7) + (lane >> 4) * 8, kcol = 16 * ks + ((lane >> 3) & 1) * 8;
#pragma unroll
            for (int jp = 0; jp < 4; ++jp) {
                uint32_t b0, b1, b2, b3;
                ldsm_x4(pf_smem_addr(ks_ + (16 * jp + krow) * LD + kcol), b0, b1, b2, b3);
                mma16816(sacc[2 * jp], qf[ks][0], qf[ks][1], qf[ks][2], qf[ks][3], b0, b1);
                mma16816(sacc[2 * jp + 1], qf[ks][0], qf[ks][1], qf[ks][2], qf[ks][3], b2, b3);
            }
        }
        // scale; the diagonal block hides keys after the query and keys past T
        const bool diag = kb == nkb - 1;
        float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                float sv = sacc[j][e] * sc;
                if (diag) {
                    const int key = kb * C::BN + 8 * j + 2 * t + (e & 1);
                    const int row = q0 + g + 8 * (e >> 1);
                    if (key > row || key >= T) sv = -INFINITY;
                }
                sacc[j][e] = sv;
                if (e < 2) mx0 = fmaxf(mx0, sv);
                else mx1 = fmaxf(mx1, sv);
            }
        mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 1));
        mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 2));
        mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 1));
        mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 2));
        const float n0 = fmaxf(m0, mx0), n1 = fmaxf(m1, mx1);
        // a row with nothing visible so far keeps a zero offset (its probabilities are all exp2(-inf) = 0)
        const float f0 = n0 == -INFINITY ? 0.f : n0, f1 = n1 == -INFINITY ? 0.f : n1;
        const float a0 = ex2_approx(m0 - f0), a1 = ex2_approx(m1 - f1);
        m0 = n0;
        m1 = n1;
        float s0 = 0.f, s1 = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            sacc[j][0] = ex2_approx(sacc[j][0] - f0);
            sacc[j][1] = ex2_approx(sacc[j][1] - f0);
            sacc[j][2] = ex2_approx(sacc[j][2] - f1);
            sacc[j][3] = ex2_approx(sacc[j][3] - f1);
            s0 += sacc[j][0] + sacc[j][1];
            s1 += sacc[j][2] + sacc[j][3];
        }
        l0 = l0 * a0 + s0;
        l1 = l1 * a1 + s1;
#pragma unroll
        for (int j = 0; j < NT; ++j) {
            o[j][0] *= a0;
            o[j][1] *= a0;
            o[j][2] *= a1;
            o[j][3] *= a1;
        }
        // weighted values: probabilities as the first operand (keys 16*kk .. +15), values through transposing
        // 8x8 matrix loads (rows = keys, two 8-channel tiles per instruction)
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            const uint32_t pa0 = pack_half2(sacc[2 * kk][0], sacc[2 * kk][1]);
            const uint32_t pa1 = pack_half2(sacc[2 * kk][2], sacc[2 * kk][3]);
            const uint32_t pa2 = pack_half2(sacc[2 * kk + 1][0], sacc[2 * kk + 1][1]);
            const uint32_t pa3 = pack_half2(sacc[2 * kk + 1][2], sacc[2 * kk + 1][3]);
            const int vrow = 16 * kk + (lane & 7) + ((lane >> 3) & 1) * 8;
#pragma unroll
            for (int jp = 0; jp < NT / 2; ++jp) {
                uint32_t b0, b1, b2, b3;
                ldsm_x4_trans(pf_smem_addr(vs_ + vrow * LD + 16 * jp + (lane >> 4) * 8), b0, b1, b2, b3);
                mma16816(o[2 * jp], pa0, pa1, pa2, pa3, b0, b1);
                mma16816(o[2 * jp + 1], pa0, pa1, pa2, pa3, b2, b3);
            }
        }
        __syncthreads();          // the stage is overwritten by the copy issued in the next iteration
    }
    l0 += __shfl_xor_sync(0xffffffffu, l0, 1);
    l0 += __shfl_xor_sync(0xffffffffu, l0, 2);
    l1 += __shfl_xor_sync(0xffffffffu, l1, 1);
    l1 += __shfl_xor_sync(0xffffffffu, l1, 2);
    const float i0 = l0 > 0.f ? 1.f / l0 : 0.f, i1 = l1 > 0.f ? 1.f / l1 : 0.f;
    const int r0 = q0 + g, r1 = q0 + g + 8;
#pragma unroll
    for (int j = 0; j < NT; ++j) {
        if (r0 < T)
            *reinterpret_cast<uint32_t*>(y + (((size_t)b * T + r0) * n_heads + h) * HD + 8 * j + 2 * t) =
                pack_half2(o[j][0] * i0, o[j][1] * i0);
        if (r1 < T)
            *reinterpret_cast<uint32_t*>(y + (((size_t)b * T + r1) * n_heads + h) * HD + 8 * j + 2 * t) =
                pack_half2(o[j][2] * i1, o[j][3] * i1);
    }
}

// x_out = x + delta (fp16), h_out = rms_norm(x_out) * w: the residual add and the layer norm that follow the
// attention output projection in a decoder layer, one CTA per row (H <= 8192, a multiple of 8).
__global__ void __launch_bounds__(256) add_rmsnorm_kernel(const __half* __restrict__ x, const __half* __restrict__ delta,
                                                          const __half* __restrict__ w, float eps, int H,
                                                          __half* __restrict__ x_out, __half* __restrict__ h_out) {
    const size_t row = (size_t)blockIdx.x * H;
    float val[4][8];
    float ss = 0.f;
    // (launched beside the projection that writes delta, for which it waits.  The weight is the caller's and may come from the launch
    // ahead as well: it is requested behind the wait, together with x and delta; a token of 24 layers 1432 us, 1436 with the weight asked for ahead)
    __align__(16) __half wv[4][8];
    asm volatile("griddepcontrol.wait;" ::: "memory");
#pragma unroll
    for (int step = 0; step < 4; ++step) {
        const int c0 = (step * 256 + threadIdx.x) * 8;
        if (c0 >= H) continue;
        __align__(16) __half a[8], b[8], o[8];
        *reinterpret_cast<uint4*>(a) = *reinterpret_cast<const uint4*>(x + row + c0);
        *reinterpret_cast<uint4*>(b) = *reinterpret_cast<const uint4*>(delta + row + c0);
        if (w) *reinterpret_cast<uint4*>(wv[step]) = *reinterpret_cast<const uint4*>(w + c0);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            o[i] = __float2half_rn(__half2float(a[i]) + __half2float(b[i]));
            val[step][i] = __half2float(o[i]);
            ss += val[step][i] * val[step][i];
        }
        *reinterpret_cast<uint4*>(x_out + row + c0) = *reinterpret_cast<const uint4*>(o);
    }
    __shared__ float red[8];
    ss = warp_sum(ss);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    float tot = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) tot += red[i];
    const float r = rsqrtf(tot / H + eps);
#pragma unroll
    for (int step = 0; step < 4; ++step) {
        const int c0 = (step * 256 + threadIdx.x) * 8;
        if (c0 >= H) continue;
        __align__(16) __half o[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] = __float2half_rn(w ? __half2float(wv[step][i]) * (val[step][i] * r) : val[step][i] * r);
        *reinterpret_cast<uint4*>(h_out + row + c0) = *reinterpret_cast<const uint4*>(o);
    }
}

}  // namespace

extern "C" int glq_add_rmsnorm(const void* x, const void* delta, const void* weight, float eps, int rows, int H, void* x_out,
                               void* h_out, void* stream) {
    if (!x || !delta || !x_out || !h_out || rows < 0 || H <= 0) return GLQ_ERR_ARG;
    if (H % 8 != 0 || H > 8192) return GLQ_ERR_UNSUPPORTED;
    if (rows == 0) return GLQ_OK;
    return launch_kernel(true, add_rmsnorm_kernel, dim3(rows), dim3(256), 0, reinterpret_cast<cudaStream_t>(stream), reinterpret_cast<const __half*>(x),
                            reinterpret_cast<const __half*>(delta), reinterpret_cast<const __half*>(weight), eps, H,
                            reinterpret_cast<__half*>(x_out), reinterpret_cast<__half*>(h_out)) == cudaSuccess
               ? GLQ_OK : GLQ_ERR_CUDA;
}

// position splits per head: enough CTAs to fill the device for long caches
static int attn_sms() {
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}
static int attn_splits(int B, int n_heads, int max_len) {
    const int sms = attn_sms();
    int s = (2 * sms + B * n_heads - 1) / (B * n_heads);
    s = std::max(1, std::min(s, 16));
    return std::min(s, std::max(1, max_len / 64));
}

extern "C" size_t glq_attn_decode_workspace_bytes(int B, int n_heads, int head_dim, int max_len) {
    if (B <= 0 || n_heads <= 0 || head_dim <= 0) return 0;
    const int s = attn_splits(B, n_heads, max_len);
    return s == 1 ? 0 : (size_t)B * n_heads * s * (head_dim + 2) * sizeof(float);
}

extern "C" int glq_attn_decode(const void* q, const void* k_new, const void* v_new, const void* cos_t, const void* sin_t,
                               const int64_t* pos, void* k_cache, void* v_cache, void* out, int B, int n_heads, int n_kv,
                               int head_dim, int max_len, const void* q_norm_w, const void* k_norm_w, float eps,
                               void* workspace, size_t workspace_bytes, int32_t* counters, size_t n_counters,
                               void* stream) {
    if (!q || !k_new || !v_new || !cos_t || !sin_t || !pos || !k_cache || !v_cache || !out) return GLQ_ERR_ARG;
    if (B < 0 || n_heads <= 0 || n_kv <= 0 || n_heads % n_kv != 0 || max_len <= 0) return GLQ_ERR_ARG;
    if (B == 0) return GLQ_OK;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const int nsplit = attn_splits(B, n_heads, max_len);
    if (nsplit > 1) {
        if (!workspace || workspace_bytes < glq_attn_decode_workspace_bytes(B, n_heads, head_dim, max_len)) return GLQ_ERR_WORKSPACE;
        if (!counters || n_counters < (size_t)B * n_heads) return GLQ_ERR_WORKSPACE;
    }
    // Heads of a CTA: two that share their keys and values read and convert these once, as long as that leaves a CTA for every
    // SM; with fewer a warp's own chain sets the pace.
    const bool two = head_dim == 128 && (n_heads / n_kv) % 2 == 0 && (long long)B * n_heads * nsplit >= 2 * attn_sms();
    const int heads = two ? 2 : 1;
    const dim3 grid(n_heads / heads, B, nsplit), block(kAttnWarps * 32);
#define GLQ_ATTN(EPL, G)                                                                                           \
    attn_decode_kernel<EPL, G><<<grid, block, 0, st>>>(                                                            \
        reinterpret_cast<const __half*>(q), reinterpret_cast<const __half*>(k_new), reinterpret_cast<const __half*>(v_new), \
        reinterpret_cast<const __half*>(cos_t), reinterpret_cast<const __half*>(sin_t),                           \
        reinterpret_cast<const long long*>(pos), reinterpret_cast<__half*>(k_cache), reinterpret_cast<__half*>(v_cache), \
        reinterpret_cast<__half*>(out), n_heads, n_kv, max_len, reinterpret_cast<const __half*>(q_norm_w),         \
        reinterpret_cast<const __half*>(k_norm_w), eps, reinterpret_cast<float*>(workspace), counters)
    switch (head_dim) {
        case 32: GLQ_ATTN(1, 1); break;
        case 64: GLQ_ATTN(2, 1); break;
        case 128:
            if (two) GLQ_ATTN(4, 2);
            else GLQ_ATTN(4, 1);
            break;
        case 256: GLQ_ATTN(8, 1); break;
        default: return GLQ_ERR_UNSUPPORTED;
    }
#undef GLQ_ATTN
    return cudaGetLastError() == cudaSuccess ? GLQ_OK : GLQ_ERR_CUDA;
}

extern "C" int glq_rope_prefill(void* q, void* k, const void* v, const void* cos_t, const void* sin_t, const int64_t* positions,
                                void* k_cache, void* v_cache, int B, int T, int n_heads, int n_kv, int head_dim, int max_len,
                                const void* q_norm_w, const void* k_norm_w, float eps, void* stream) {
    if (!q || !k || !v || !cos_t || !sin_t || !positions || !k_cache || !v_cache) return GLQ_ERR_ARG;
    if (B < 0 || T < 0 || n_heads <= 0 || n_kv <= 0 || max_len <= 0) return GLQ_ERR_ARG;
    if (B == 0 || T == 0) return GLQ_OK;
    const dim3 grid(B * T);
    int vec = 1;
    for (const void* ptr : {(const void*)q, (const void*)k, v, cos_t, sin_t, (const void*)k_cache, (const void*)v_cache})
        if (reinterpret_cast<uintptr_t>(ptr) & 7u) vec = 0;
    auto st = reinterpret_cast<cudaStream_t>(stream);
    cudaError_t rc = cudaSuccess;
#define GLQ_ROPE_CASE(EPL)                                                                                                  \
    rc = launch_kernel(true, rope_prefill_kernel<EPL>, grid, dim3(kAttnWarps * 32), 0, st,                                        \
        reinterpret_cast<__half*>(q), reinterpret_cast<__half*>(k), reinterpret_cast<const __half*>(v),                     \
        reinterpret_cast<const __half*>(cos_t), reinterpret_cast<const __half*>(sin_t),                                     \
        reinterpret_cast<const long long*>(positions), reinterpret_cast<__half*>(k_cache), reinterpret_cast<__half*>(v_cache), \
        T, n_heads, n_kv, max_len, reinterpret_cast<const __half*>(q_norm_w), reinterpret_cast<const __half*>(k_norm_w), eps, vec)
    switch (head_dim) {
        case 32: GLQ_ROPE_CASE(1); break;
        case 64: GLQ_ROPE_CASE(2); break;
        case 128: GLQ_ROPE_CASE(4); break;
        case 256: GLQ_ROPE_CASE(8); break;
        default: return GLQ_ERR_UNSUPPORTED;
    }
#undef GLQ_ROPE_CASE
    return rc == cudaSuccess ? GLQ_OK : GLQ_ERR_CUDA;
}

extern "C" int glq_attn_prefill(const void* q, const void* k, const void* v, void* y, int B, int T, int n_heads, int n_kv,
                                int head_dim, void* stream) {
    if (!q || !k || !v || !y) return GLQ_ERR_ARG;
    if (B < 0 || T < 0 || n_heads <= 0 || n_kv <= 0 || n_heads % n_kv != 0) return GLQ_ERR_ARG;
    if (B == 0 || T == 0) return GLQ_OK;
    if (head_dim != 64 && head_dim != 128) return GLQ_ERR_UNSUPPORTED;
    if ((long long)((T + 63) / 64) * n_heads * B > 0x7fffffffll) return GLQ_ERR_UNSUPPORTED;
    for (const void* ptr : {q, k, v, (const void*)y})
        if ((reinterpret_cast<uintptr_t>(ptr) & 15u) != 0) return GLQ_ERR_ALIGN;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const dim3 grid((unsigned)((T + 63) / 64 * n_heads * B));     // every (query block, head, batch row), most keys first
    cudaError_t rc = cudaSuccess;
#define GLQ_PREFILL(HD)                                                                                                  \
    {                                                                                                                    \
        static SmemLimit limit;                                                                                          \
        if (reserve_smem(reinterpret_cast<const void*>(attn_prefill_kernel<HD>), limit, PrefillCfg<HD>::SMEM) != cudaSuccess) \
            return GLQ_ERR_CUDA;                                                                                         \
        rc = launch_kernel(true, attn_prefill_kernel<HD>, grid, dim3(128), PrefillCfg<HD>::SMEM, st,                           \
            reinterpret_cast<const __half*>(q), reinterpret_cast<const __half*>(k), reinterpret_cast<const __half*>(v),  \
            reinterpret_cast<__half*>(y), B, T, n_heads, n_kv);                                                              \
    }
    if (head_dim == 64) GLQ_PREFILL(64) else GLQ_PREFILL(128)
#undef GLQ_PREFILL
    return rc == cudaSuccess ? GLQ_OK : GLQ_ERR_CUDA;
}
