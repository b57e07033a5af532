// Decode-side operations around the quantized GEMMs of a Llama-architecture layer (bf16, sm_100a): what the
// reference fuses around its int4 matmul in PTQ/quant —
//   * RMSNorm                      (PTQ/quant/triton_norm.py:7-39), here with the residual add that precedes it,
//   * rotate-half RoPE on q and k  (PTQ/quant/fused_attn.py:8-58), here writing k and v straight into the KV cache,
//   * silu(gate) * up              (epilogue of PTQ/quant/fused_mlp.py:84-168),
//   * single-query attention over the KV cache (the reference calls F.scaled_dot_product_attention,
//     PTQ/quant/fused_attn.py:148-149).
// A decode step then is nine launches per layer instead of the ~45 elementwise kernels of the eager modules.
// All kernels are HBM/L2 streaming kernels over a few hundred KB: one pass, 16-byte accesses, no scratch
// besides the attention's split partials.
//
// Rounding: `hf_rounding != 0` reproduces the bf16 tensor-op chain of the eager HF modules (every op result
// rounded to bf16); 0 keeps fp32 up to the single final cast like the reference's Triton kernels do.
#include "lq_common.cuh"

namespace lq {

__device__ __forceinline__ float bf_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }
__device__ __forceinline__ uint32_t pack_bf2(float a, float b) {
    __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&v);
}

// ---------------------------------------------------------------------------------------------
// h += delta (optional); y = RMSNorm(h) * gamma.  One CTA per token row.
// ---------------------------------------------------------------------------------------------
constexpr int NORM_THREADS = 256;
__global__ void __launch_bounds__(NORM_THREADS) k_add_rmsnorm(__nv_bfloat16* __restrict__ h, const __nv_bfloat16* __restrict__ delta,
                                                               const __nv_bfloat16* __restrict__ gamma, float eps,
                                                               __nv_bfloat16* __restrict__ y, int K, int hf_rounding) {
    __shared__ float red[NORM_THREADS / 32];
    pdl_launch_dependents();                          // (decode chain) the successor may be launched; it waits for this grid
    pdl_wait();                                       // h / delta may be the predecessor's output
    const size_t row = (size_t)blockIdx.x * K;
    uint4* hv = reinterpret_cast<uint4*>(h + row);
    const uint4* dv = delta ? reinterpret_cast<const uint4*>(delta + row) : nullptr;
    float ss = 0.0f;
    for (int i = threadIdx.x; i < K / 8; i += NORM_THREADS) {
        uint4 a = hv[i];
        uint32_t w[4] = {a.x, a.y, a.z, a.w};
        if (dv) {                                      // residual + hidden_states: one bf16 rounding of the fp32 sum
            const uint4 d = __ldg(dv + i);
            const uint32_t e[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) w[j] = pack_bf2(__fadd_rn(bf_lo(w[j]), bf_lo(e[j])), __fadd_rn(bf_hi(w[j]), bf_hi(e[j])));
            hv[i] = make_uint4(w[0], w[1], w[2], w[3]);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) { const float lo = bf_lo(w[j]), hi = bf_hi(w[j]); ss = fmaf(lo, lo, ss); ss = fmaf(hi, hi, ss); }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    float tot = 0.0f;
#pragma unroll
    for (int wv = 0; wv < NORM_THREADS / 32; ++wv) tot += red[wv];          // same order in every thread
    const float rstd = hf_rounding ? rsqrtf(tot / (float)K + eps) : 1.0f / sqrtf(tot / (float)K + eps);
    const uint4* gv = reinterpret_cast<const uint4*>(gamma);
    uint4* yv = reinterpret_cast<uint4*>(y + row);
    for (int i = threadIdx.x; i < K / 8; i += NORM_THREADS) {
        const uint4 a = hv[i], g = __ldg(gv + i);          // this thread wrote hv[i] itself
        const uint32_t w[4] = {a.x, a.y, a.z, a.w}, gw[4] = {g.x, g.y, g.z, g.w};
        uint32_t o[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float lo = __fmul_rn(bf_lo(w[j]), rstd), hi = __fmul_rn(bf_hi(w[j]), rstd);
            if (hf_rounding) { lo = bf16r(lo); hi = bf16r(hi); }
            o[j] = pack_bf2(__fmul_rn(lo, bf_lo(gw[j])), __fmul_rn(hi, bf_hi(gw[j])));
        }
        yv[i] = make_uint4(o[0], o[1], o[2], o[3]);
    }
}

// Register-resident variant for K <= 2048 * VPT: every thread requests all its vectors of h, delta and gamma before
// anything is reduced (one round of memory latency instead of three), and the row is never re-read.
template <int VPT>
__global__ void __launch_bounds__(NORM_THREADS) k_add_rmsnorm_r(__nv_bfloat16* __restrict__ h, const __nv_bfloat16* __restrict__ delta,
                                                                 const __nv_bfloat16* __restrict__ gamma, float eps,
                                                                 __nv_bfloat16* __restrict__ y, int K, int hf_rounding) {
    __shared__ float red[NORM_THREADS / 32];
    const uint4* gv = reinterpret_cast<const uint4*>(gamma);
    const int nvec = K / 8;
    uint4 g[VPT], a[VPT], d[VPT];
#pragma unroll
    for (int u = 0; u < VPT; ++u) {                   // gamma is a parameter: fetched before the dependency wait
        const int i = threadIdx.x + u * NORM_THREADS;
        g[u] = i < nvec ? __ldg(gv + i) : make_uint4(0, 0, 0, 0);
    }
    pdl_launch_dependents();
    pdl_wait();                                       // h / delta may be the predecessor's output
    const size_t row = (size_t)blockIdx.x * K;
    uint4* hv = reinterpret_cast<uint4*>(h + row);
    const uint4* dv = delta ? reinterpret_cast<const uint4*>(delta + row) : nullptr;
#pragma unroll
    for (int u = 0; u < VPT; ++u) {
        const int i = threadIdx.x + u * NORM_THREADS;
        a[u] = i < nvec ? hv[i] : make_uint4(0, 0, 0, 0);
        d[u] = (dv && i < nvec) ? __ldg(dv + i) : make_uint4(0, 0, 0, 0);
    }
    float ss = 0.0f;
#pragma unroll
    for (int u = 0; u < VPT; ++u) {
        uint32_t* w = reinterpret_cast<uint32_t*>(&a[u]);
        const uint32_t* e = reinterpret_cast<const uint32_t*>(&d[u]);
        if (dv) {
#pragma unroll
            for (int j = 0; j < 4; ++j) w[j] = pack_bf2(__fadd_rn(bf_lo(w[j]), bf_lo(e[j])), __fadd_rn(bf_hi(w[j]), bf_hi(e[j])));
            const int i = threadIdx.x + u * NORM_THREADS;
            if (i < nvec) hv[i] = a[u];
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) { const float lo = bf_lo(w[j]), hi = bf_hi(w[j]); ss = fmaf(lo, lo, ss); ss = fmaf(hi, hi, ss); }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    float tot = 0.0f;
#pragma unroll
    for (int wv = 0; wv < NORM_THREADS / 32; ++wv) tot += red[wv];
    const float rstd = hf_rounding ? rsqrtf(tot / (float)K + eps) : 1.0f / sqrtf(tot / (float)K + eps);
    uint4* yv = reinterpret_cast<uint4*>(y + row);
#pragma unroll
    for (int u = 0; u < VPT; ++u) {
        const int i = threadIdx.x + u * NORM_THREADS;
        if (i >= nvec) continue;
        const uint32_t* w = reinterpret_cast<const uint32_t*>(&a[u]);
        const uint32_t* gw = reinterpret_cast<const uint32_t*>(&g[u]);
        uint32_t o[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float lo = __fmul_rn(bf_lo(w[j]), rstd), hi = __fmul_rn(bf_hi(w[j]), rstd);
            if (hf_rounding) { lo = bf16r(lo); hi = bf16r(hi); }
            o[j] = pack_bf2(__fmul_rn(lo, bf_lo(gw[j])), __fmul_rn(hi, bf_hi(gw[j])));
        }
        yv[i] = make_uint4(o[0], o[1], o[2], o[3]);
    }
}

// ---------------------------------------------------------------------------------------------
// RoPE (rotate-half) on the q and k heads of a fused qkv row, k and v stored into the cache at the token's position.
// grid (token, head of q|k|v), hd/2 threads.  Cache layout [batch, kv head, max_len, hd].
// ---------------------------------------------------------------------------------------------
__global__ void k_rope_kv_store(__nv_bfloat16* __restrict__ qkv, const long long* __restrict__ positions,
                                const float* __restrict__ inv_freq, __nv_bfloat16* __restrict__ k_cache,
                                __nv_bfloat16* __restrict__ v_cache, int tokens_per_seq, int Hq, int Hkv, int hd, int max_len,
                                int hf_rounding) {
    const int m = blockIdx.x, head = blockIdx.y, i = threadIdx.x, half = hd >> 1;
    pdl_launch_dependents();
    pdl_wait();                                       // qkv is the predecessor's output
    const long long pos = positions[m];
    __nv_bfloat16* src = qkv + (size_t)m * (size_t)(Hq + 2 * Hkv) * hd + (size_t)head * hd;
    const int b = m / tokens_per_seq;
    if (head >= Hq + Hkv) {                                   // v: plain copy into the cache
        if (pos < 0 || pos >= max_len) return;
        __nv_bfloat16* dst = v_cache + (((size_t)b * Hkv + (head - Hq - Hkv)) * max_len + (size_t)pos) * hd;
        reinterpret_cast<uint32_t*>(dst)[i] = reinterpret_cast<const uint32_t*>(src)[i];
        return;
    }
    const float x = __bfloat162float(src[i]), yv = __bfloat162float(src[i + half]);
    float s, c;
    sincosf((float)pos * inv_freq[i], &s, &c);
    float ox, oy;
    if (hf_rounding) {        // cos / sin cast to bf16, then q*cos + rotate_half(q)*sin as bf16 tensor ops
        c = bf16r(c); s = bf16r(s);
        ox = __fadd_rn(bf16r(__fmul_rn(x, c)), bf16r(__fmul_rn(-yv, s)));
        oy = __fadd_rn(bf16r(__fmul_rn(yv, c)), bf16r(__fmul_rn(x, s)));
    } else {
        ox = __fsub_rn(__fmul_rn(x, c), __fmul_rn(yv, s));
        oy = __fadd_rn(__fmul_rn(x, s), __fmul_rn(yv, c));
    }
    const __nv_bfloat16 bx = __float2bfloat16_rn(ox), by = __float2bfloat16_rn(oy);
    if (head < Hq) { src[i] = bx; src[i + half] = by; return; }                 // q: in place
    if (pos < 0 || pos >= max_len) return;
    __nv_bfloat16* dst = k_cache + (((size_t)b * Hkv + (head - Hq)) * max_len + (size_t)pos) * hd;
    dst[i] = bx; dst[i + half] = by;
}

// The same, four rotation pairs and several heads per thread: a thread's cosines and sines are computed once and serve its heads, and it moves 8 bytes
// at a time.  A CTA takes one token and the heads blockIdx.y, blockIdx.y + gridDim.y, ... of every set of 256 / (hd / 8).  The kernel above computes an
// angle for every pair of every head: 40 us for 400 tokens of 96 heads of 128 (20 MB), here 5.7 (3.5 TB/s), 3000 tokens 297 -> 33 (4.5 TB/s).
__global__ void __launch_bounds__(256) k_rope_kv_store4(__nv_bfloat16* __restrict__ qkv, const long long* __restrict__ positions, const float* __restrict__ inv_freq,
                                                        __nv_bfloat16* __restrict__ k_cache, __nv_bfloat16* __restrict__ v_cache, int tokens_per_seq, int Hq, int Hkv, int hd,
                                                        int max_len, int hf_rounding) {
    const int tph = hd >> 3, per = 256 / tph, hs = threadIdx.x / tph, i = (threadIdx.x - hs * tph) * 4, half = hd >> 1;
    const int m = blockIdx.x, heads = Hq + 2 * Hkv;
    if (hs >= per) return;
    pdl_launch_dependents();
    pdl_wait();                                       // qkv is the predecessor's output
    const long long pos = positions[m];
    const int b = m / tokens_per_seq;
    const bool pos_ok = pos >= 0 && pos < max_len;
    float c[4], s[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        sincosf((float)pos * inv_freq[i + j], &s[j], &c[j]);
        if (hf_rounding) { c[j] = bf16r(c[j]); s[j] = bf16r(s[j]); }
    }
    for (int head = blockIdx.y * per + hs; head < heads; head += gridDim.y * per) {
        __nv_bfloat16* src = qkv + (size_t)m * (size_t)heads * hd + (size_t)head * hd + i;
        const uint2 xv = *reinterpret_cast<const uint2*>(src), yv = *reinterpret_cast<const uint2*>(src + half);
        uint2 ox = xv, oy = yv;
        if (head < Hq + Hkv) {
            const float x[4] = {bf_lo(xv.x), bf_hi(xv.x), bf_lo(xv.y), bf_hi(xv.y)}, y[4] = {bf_lo(yv.x), bf_hi(yv.x), bf_lo(yv.y), bf_hi(yv.y)};
            float rx[4], ry[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (hf_rounding) {        // q*cos + rotate_half(q)*sin as bf16 tensor ops
                    rx[j] = __fadd_rn(bf16r(__fmul_rn(x[j], c[j])), bf16r(__fmul_rn(-y[j], s[j])));
                    ry[j] = __fadd_rn(bf16r(__fmul_rn(y[j], c[j])), bf16r(__fmul_rn(x[j], s[j])));
                } else {
                    rx[j] = __fsub_rn(__fmul_rn(x[j], c[j]), __fmul_rn(y[j], s[j]));
                    ry[j] = __fadd_rn(__fmul_rn(x[j], s[j]), __fmul_rn(y[j], c[j]));
                }
            }
            ox = make_uint2(pack_bf2(rx[0], rx[1]), pack_bf2(rx[2], rx[3]));
            oy = make_uint2(pack_bf2(ry[0], ry[1]), pack_bf2(ry[2], ry[3]));
        }
        if (head >= Hq && !pos_ok) continue;
        const int kh = head - Hq;                     // q in place, rotated k and v as they are into the caches
        __nv_bfloat16* dst = kh < 0 ? src : (kh < Hkv ? k_cache + (((size_t)b * Hkv + kh) * max_len + (size_t)pos) * hd + i
                                                      : v_cache + (((size_t)b * Hkv + kh - Hkv) * max_len + (size_t)pos) * hd + i);
        *reinterpret_cast<uint2*>(dst) = ox;
        *reinterpret_cast<uint2*>(dst + half) = oy;
    }
}

// ---------------------------------------------------------------------------------------------
// Single-query attention over the cache: out[b, h, :] = softmax(q . K[0..pos] * scale) . V[0..pos].
// grid (batch * q heads, splits); 128 threads = 16 key slots of 8 lanes, a lane holds hd/8 dims (hd = 64 or 128).
// Each split covers a contiguous range of keys.  CLUSTER: the splits of a (batch, head) are one cluster and leave (max, sum, weighted V)
// in their own shared memory, where the first reads them.  Otherwise they go to the workspace and the split that finishes last
// combines them (a ticket counter; nobody waits for anybody): store, fence, ticket and two dependent reads are five trips to L2 at
// the end of a launch of a few microseconds.
// In a chain every CTA asks for its first keys and values in L2 before the dependency wait (`prefetch`): the position it goes by may still be
// the previous step's (the rows then differ by one key), and it is read again behind the wait.
// ---------------------------------------------------------------------------------------------
constexpr int ATT_THREADS = 128, ATT_SLOTS = ATT_THREADS / 8, ATT_CLUSTER_MAX = 8;
__device__ __forceinline__ float ld_cluster(const float* local, int rank) {            // the same variable of the cluster's CTA `rank`
    uint32_t a;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(local)), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void att_cluster_sync() { asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory"); }
template <int HD, bool CLUSTER>
__global__ void __launch_bounds__(ATT_THREADS) k_decode_attn(const __nv_bfloat16* __restrict__ q, int q_row_stride,
                                                              const __nv_bfloat16* __restrict__ k_cache,
                                                              const __nv_bfloat16* __restrict__ v_cache,
                                                              const long long* __restrict__ positions, __nv_bfloat16* __restrict__ out,
                                                              int Hq, int Hkv, int max_len, float scale, float* __restrict__ part,
                                                              unsigned int* __restrict__ tickets, int prefetch) {
    constexpr int D = HD / 8;                                 // dims per lane
    __shared__ float sm_m[ATT_SLOTS], sm_l[ATT_SLOTS], sm_acc[ATT_SLOTS][HD];
    __shared__ bool is_last;
    __shared__ float cl_acc[HD], cl_ml[2];
    const int bh = blockIdx.x, b = bh / Hq, h = bh - b * Hq, hk = h / (Hq / Hkv);
    const int splits = gridDim.y, split = blockIdx.y;
    const int slot = threadIdx.x >> 3, sub = threadIdx.x & 7;
    constexpr int KPI = 4;                                    // keys per slot in flight
    const __nv_bfloat16* kb = k_cache + ((size_t)b * Hkv + hk) * (size_t)max_len * HD + sub * D;
    const __nv_bfloat16* vb = v_cache + ((size_t)b * Hkv + hk) * (size_t)max_len * HD + sub * D;
    pdl_launch_dependents();
    if (prefetch) {
        const long long n = min(max(__ldcv(positions + b) + 1, 0ll), (long long)max_len);
        const int per = (int)((n + splits - 1) / splits), j0 = split * per + slot, j1 = (int)min((long long)(split + 1) * per, n);
#pragma unroll
        for (int u = 0; u < KPI; ++u)
            if (j0 + u * ATT_SLOTS < j1) {
                asm volatile("prefetch.global.L2 [%0];" ::"l"(kb + (size_t)(j0 + u * ATT_SLOTS) * HD));
                asm volatile("prefetch.global.L2 [%0];" ::"l"(vb + (size_t)(j0 + u * ATT_SLOTS) * HD));
            }
    }
    pdl_wait();                                       // q and the newest cache row are the predecessor's output
    long long n_keys = __ldcv(positions + b) + 1;
    if (n_keys > max_len) n_keys = max_len;
    if (n_keys < 0) n_keys = 0;
    const int per = (int)((n_keys + splits - 1) / splits);
    const int j0 = split * per, j1 = (int)min((long long)(j0 + per), n_keys);

    float qf[D];
    {
        const __nv_bfloat16* qp = q + (size_t)b * q_row_stride + (size_t)h * HD + sub * D;
#pragma unroll
        for (int d = 0; d < D; d += 2) {
            const uint32_t w = *reinterpret_cast<const uint32_t*>(qp + d);
            qf[d] = bf_lo(w) * scale; qf[d + 1] = bf_hi(w) * scale;
        }
    }
    const unsigned int slot_mask = 0xffu << (8 * (slot & 3));
    float mx = -INFINITY, l = 0.0f, acc[D];
#pragma unroll
    for (int d = 0; d < D; ++d) acc[d] = 0.0f;
    // KPI keys per slot in flight: the K and V rows of all of them are requested before any arithmetic (the kernel is a
    // chain of memory latencies otherwise; a ticket's split covers about 64 keys, one such round per slot, a cluster's up to a few hundred).  A key beyond the
    // range reads key j1-1 again and gets weight zero.
    for (int j = j0 + slot; j < j1; j += KPI * ATT_SLOTS) {
        uint4 kq[KPI][D / 8], vq[KPI][D / 8];
        bool on[KPI];
#pragma unroll
        for (int u = 0; u < KPI; ++u) {
            const int ju = j + u * ATT_SLOTS;
            on[u] = ju < j1;
            const size_t row = (size_t)(on[u] ? ju : j1 - 1) * HD;
#pragma unroll
            for (int d = 0; d < D / 8; ++d) {
                kq[u][d] = __ldg(reinterpret_cast<const uint4*>(kb + row) + d);
                vq[u][d] = __ldg(reinterpret_cast<const uint4*>(vb + row) + d);
            }
        }
        float sc[KPI];
#pragma unroll
        for (int u = 0; u < KPI; ++u) {
            float a = 0.0f;
#pragma unroll
            for (int d = 0; d < D / 8; ++d) {
                const uint32_t w[4] = {kq[u][d].x, kq[u][d].y, kq[u][d].z, kq[u][d].w};
#pragma unroll
                for (int e = 0; e < 4; ++e) { a = fmaf(qf[d * 8 + 2 * e], bf_lo(w[e]), a); a = fmaf(qf[d * 8 + 2 * e + 1], bf_hi(w[e]), a); }
            }
            // the four key slots of a warp run different numbers of iterations: only this slot's 8 lanes take part
            a += __shfl_xor_sync(slot_mask, a, 1); a += __shfl_xor_sync(slot_mask, a, 2); a += __shfl_xor_sync(slot_mask, a, 4);
            sc[u] = on[u] ? a : -INFINITY;
        }
        float mn = mx;
#pragma unroll
        for (int u = 0; u < KPI; ++u) mn = fmaxf(mn, sc[u]);
        const float corr = __expf(mx - mn);
        float pw[KPI];
        l *= corr;
#pragma unroll
        for (int u = 0; u < KPI; ++u) { pw[u] = on[u] ? __expf(sc[u] - mn) : 0.0f; l += pw[u]; }
#pragma unroll
        for (int d = 0; d < D; ++d) acc[d] *= corr;
#pragma unroll
        for (int u = 0; u < KPI; ++u) {
#pragma unroll
            for (int d = 0; d < D / 8; ++d) {
                const uint32_t w[4] = {vq[u][d].x, vq[u][d].y, vq[u][d].z, vq[u][d].w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    acc[d * 8 + 2 * e] = fmaf(pw[u], bf_lo(w[e]), acc[d * 8 + 2 * e]);
                    acc[d * 8 + 2 * e + 1] = fmaf(pw[u], bf_hi(w[e]), acc[d * 8 + 2 * e + 1]);
                }
            }
        }
        mx = mn;
    }
    // combine the 16 key slots of the CTA
    if (sub == 0) { sm_m[slot] = mx; sm_l[slot] = l; }
#pragma unroll
    for (int d = 0; d < D; ++d) sm_acc[slot][sub * D + d] = acc[d];
    __syncthreads();
    float* my = part + ((size_t)bh * splits + split) * (HD + 2);
    if (threadIdx.x < HD) {
        float M = -INFINITY;
#pragma unroll
        for (int s2 = 0; s2 < ATT_SLOTS; ++s2) M = fmaxf(M, sm_m[s2]);
        float L = 0.0f, a = 0.0f;
#pragma unroll
        for (int s2 = 0; s2 < ATT_SLOTS; ++s2) {
            const float w = (sm_m[s2] == -INFINITY) ? 0.0f : __expf(sm_m[s2] - M);
            L = fmaf(sm_l[s2], w, L); a = fmaf(sm_acc[s2][threadIdx.x], w, a);
        }
        if (CLUSTER) {
            cl_acc[threadIdx.x] = a;
            if (threadIdx.x == 0) { cl_ml[0] = M; cl_ml[1] = L; }
        } else if (splits == 1) {
            out[(size_t)b * Hq * HD + (size_t)h * HD + threadIdx.x] = __float2bfloat16_rn(L > 0.0f ? a / L : 0.0f);
        } else {
            my[threadIdx.x] = a;
            if (threadIdx.x == 0) { my[HD] = M; my[HD + 1] = L; }
        }
    }
    if constexpr (CLUSTER) {
        att_cluster_sync();
        if (split == 0 && threadIdx.x < HD) {                   // the cluster's CTA ranks are its split numbers
            float ms[ATT_CLUSTER_MAX], ls[ATT_CLUSTER_MAX], v[ATT_CLUSTER_MAX], M = -INFINITY;
#pragma unroll
            for (int i = 0; i < ATT_CLUSTER_MAX; ++i) {
                ms[i] = -INFINITY;
                if (i < splits) { ms[i] = ld_cluster(cl_ml, i); ls[i] = ld_cluster(cl_ml + 1, i); v[i] = ld_cluster(cl_acc + threadIdx.x, i); }
            }
#pragma unroll
            for (int i = 0; i < ATT_CLUSTER_MAX; ++i) M = fmaxf(M, ms[i]);
            float L = 0.0f, a = 0.0f;
#pragma unroll
            for (int i = 0; i < ATT_CLUSTER_MAX; ++i)
                if (i < splits) {
                    const float w = (ms[i] == -INFINITY) ? 0.0f : __expf(ms[i] - M);
                    L = fmaf(ls[i], w, L); a = fmaf(v[i], w, a);
                }
            out[(size_t)b * Hq * HD + (size_t)h * HD + threadIdx.x] = __float2bfloat16_rn(L > 0.0f ? a / L : 0.0f);
        }
        att_cluster_sync();                                     // the others' shared memory has been read
        return;
    }
    if (splits == 1) return;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned int t = atomicAdd(tickets + bh, 1u);
        is_last = (t == (unsigned int)splits - 1u);
        if (is_last) tickets[bh] = 0u;                          // leave the counter as it was found
    }
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    // The splits' (max, sum) come in one load per lane and their weights go through shared memory; the weighted values of eight
    // splits are requested together.  (Read split by split the combination was a chain of L2 round trips: two per split.)
    __shared__ float sp_w[32], sp_l[32];                        // splits <= 32
    const float* base = part + (size_t)bh * splits * (HD + 2);
    if (threadIdx.x < 32) {
        const int s2 = threadIdx.x;
        const bool have = s2 < splits;
        const float ms = have ? __ldcg(base + (size_t)s2 * (HD + 2) + HD) : -INFINITY;
        const float ls = have ? __ldcg(base + (size_t)s2 * (HD + 2) + HD + 1) : 0.0f;
        float M = ms;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
        sp_w[s2] = (ms == -INFINITY) ? 0.0f : __expf(ms - M);
        sp_l[s2] = ls;
    }
    __syncthreads();
    if (threadIdx.x < HD) {
        float L = 0.0f, a = 0.0f;
        for (int s0 = 0; s0 < splits; s0 += 8) {
            float v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = (s0 + i < splits) ? __ldcg(base + (size_t)(s0 + i) * (HD + 2) + threadIdx.x) : 0.0f;
#pragma unroll
            for (int i = 0; i < 8; ++i)
                if (s0 + i < splits) { L = fmaf(sp_l[s0 + i], sp_w[s0 + i], L); a = fmaf(v[i], sp_w[s0 + i], a); }
        }
        out[(size_t)b * Hq * HD + (size_t)h * HD + threadIdx.x] = __float2bfloat16_rn(L > 0.0f ? a / L : 0.0f);
    }
}

// ---------------------------------------------------------------------------------------------
// act[m, i] = silu(gu[m, i]) * gu[m, I + i]
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_silu_mul(const __nv_bfloat16* __restrict__ gu, __nv_bfloat16* __restrict__ act,
                                                  int64_t M, int I, int hf_rounding) {
    const int64_t vec_per_row = I / 8, total = M * vec_per_row;
    pdl_launch_dependents();
    pdl_wait();                                       // gate | up is the predecessor's output
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < total; v += (int64_t)gridDim.x * blockDim.x) {
        const int64_t m = v / vec_per_row, c = v - m * vec_per_row;
        const uint4 g = __ldg(reinterpret_cast<const uint4*>(gu + m * 2 * (int64_t)I) + c);
        const uint4 u = __ldg(reinterpret_cast<const uint4*>(gu + m * 2 * (int64_t)I + I) + c);
        const uint32_t gw[4] = {g.x, g.y, g.z, g.w}, uw[4] = {u.x, u.y, u.z, u.w};
        uint32_t o[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float g0 = bf_lo(gw[j]), g1 = bf_hi(gw[j]);
            float s0 = g0 / (1.0f + expf(-g0)), s1 = g1 / (1.0f + expf(-g1));
            if (hf_rounding) { s0 = bf16r(s0); s1 = bf16r(s1); }
            o[j] = pack_bf2(__fmul_rn(s0, bf_lo(uw[j])), __fmul_rn(s1, bf_hi(uw[j])));
        }
        reinterpret_cast<uint4*>(act + m * (int64_t)I)[c] = make_uint4(o[0], o[1], o[2], o[3]);
    }
}

// ---------------------------------------------------------------------------------------------
// End of a greedy decode step in one launch: tok[b] = argmax_v logits[b, v] (the first maximum, NaN counts as the
// largest value, as torch.argmax), positions[b] += 1, h[b, :] = embed[tok[b], :] (the next step's input row).
// One CTA per sequence; a thread walks its vectors in ascending order, so "first" survives the reduction by
// preferring the smaller index among equal values.
// ---------------------------------------------------------------------------------------------
constexpr int AM_THREADS = 1024;
__device__ __forceinline__ bool am_better(float v, int i, float bv, int bi) {
    const bool vn = v != v, bn = bv != bv;
    if (vn != bn) return vn;
    if (!vn && v != bv) return v > bv;
    return i < bi;
}
__global__ void __launch_bounds__(AM_THREADS) k_argmax_embed(const __nv_bfloat16* __restrict__ logits, int64_t logits_stride, int V,
                                                             int vec, const __nv_bfloat16* __restrict__ embed, int D,
                                                             long long* __restrict__ tok, long long* __restrict__ positions,
                                                             __nv_bfloat16* __restrict__ h) {
    __shared__ float sv[AM_THREADS / 32];
    __shared__ int si[AM_THREADS / 32];
    __shared__ int winner;
    const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    pdl_launch_dependents();
    pdl_wait();                                       // the logits are the predecessor's output
    const __nv_bfloat16* row = logits + (size_t)b * logits_stride;
    float bv = -INFINITY;
    int bi = 0x7fffffff;
    if (vec) {                                        // rows start on 16-byte boundaries and hold whole vectors
        for (int v = tid; v < V / 8; v += AM_THREADS) {
            const uint4 q = __ldg(reinterpret_cast<const uint4*>(row) + v);
            const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float lo = bf_lo(w[j]), hi = bf_hi(w[j]);
                if (am_better(lo, v * 8 + 2 * j, bv, bi)) { bv = lo; bi = v * 8 + 2 * j; }
                if (am_better(hi, v * 8 + 2 * j + 1, bv, bi)) { bv = hi; bi = v * 8 + 2 * j + 1; }
            }
        }
    } else {
        for (int v = tid; v < V; v += AM_THREADS) {
            const float x = __bfloat162float(row[v]);
            if (am_better(x, v, bv, bi)) { bv = x; bi = v; }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (am_better(ov, oi, bv, bi)) { bv = ov; bi = oi; }
    }
    if (lane == 0) { sv[warp] = bv; si[warp] = bi; }
    __syncthreads();
    if (warp == 0) {
        bv = sv[lane]; bi = si[lane];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (am_better(ov, oi, bv, bi)) { bv = ov; bi = oi; }
        }
        if (lane == 0) {
            winner = bi;
            tok[b] = bi;
            if (positions) positions[b] += 1;
        }
    }
    __syncthreads();
    if (!embed) return;
    const uint4* src = reinterpret_cast<const uint4*>(embed + (size_t)winner * D);
    uint4* dst = reinterpret_cast<uint4*>(h + (size_t)b * D);
    for (int v = tid; v < D / 8; v += AM_THREADS) dst[v] = __ldg(src + v);
}

// The same with a cluster of eight CTAs per sequence, for rows of whole vectors.  A launch is a chain of latencies (32000 logits: the kernel above loops four
// times over a trip to L2 and compares 32 numbers per thread on one SM, 5.2 us in a chain): a CTA takes an eighth of the row, two or three vectors per thread in
// flight together, the candidates meet in shared memory of the cluster, and every CTA copies its eighth of the winner's row.  3.9 us.
constexpr int AMC = 8, AMC_THREADS = 256, AMC_VEC = 4;
__device__ __forceinline__ void am_warp_best(float& bv, int& bi) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (am_better(ov, oi, bv, bi)) { bv = ov; bi = oi; }
    }
}
__global__ void __cluster_dims__(AMC, 1, 1) __launch_bounds__(AMC_THREADS)
k_argmax_embed_cluster(const __nv_bfloat16* __restrict__ logits, int64_t logits_stride, int V, const __nv_bfloat16* __restrict__ embed, int D, long long* __restrict__ tok,
                       long long* __restrict__ positions, __nv_bfloat16* __restrict__ h) {
    __shared__ float sv[AMC_THREADS / 32], cv;
    __shared__ int si[AMC_THREADS / 32], ci;
    const int b = blockIdx.x / AMC, rank = blockIdx.x % AMC, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nv = V / 8, per = (nv + AMC - 1) / AMC, v0 = rank * per, v1 = min(nv, v0 + per);
    pdl_launch_dependents();
    pdl_wait();                                       // the logits are the predecessor's output
    const uint4* row = reinterpret_cast<const uint4*>(logits + (size_t)b * logits_stride);
    float bv = -INFINITY;
    int bi = 0x7fffffff;
    for (int v = v0 + tid; v < v1; v += AMC_VEC * AMC_THREADS) {
        uint4 q[AMC_VEC];
#pragma unroll
        for (int u = 0; u < AMC_VEC; ++u)
            if (v + u * AMC_THREADS < v1) q[u] = __ldg(row + v + u * AMC_THREADS);
#pragma unroll
        for (int u = 0; u < AMC_VEC; ++u) {
            if (v + u * AMC_THREADS >= v1) break;
            const uint32_t w[4] = {q[u].x, q[u].y, q[u].z, q[u].w};
            const int at = (v + u * AMC_THREADS) * 8;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float lo = bf_lo(w[j]), hi = bf_hi(w[j]);
                if (am_better(lo, at + 2 * j, bv, bi)) { bv = lo; bi = at + 2 * j; }
                if (am_better(hi, at + 2 * j + 1, bv, bi)) { bv = hi; bi = at + 2 * j + 1; }
            }
        }
    }
    am_warp_best(bv, bi);
    if (lane == 0) { sv[warp] = bv; si[warp] = bi; }
    __syncthreads();
    if (warp == 0) {
        bv = lane < AMC_THREADS / 32 ? sv[lane] : -INFINITY; bi = lane < AMC_THREADS / 32 ? si[lane] : 0x7fffffff;
        am_warp_best(bv, bi);
        if (lane == 0) { cv = bv; ci = bi; }
    }
    att_cluster_sync();
    bv = -INFINITY; bi = 0x7fffffff;
    if (lane < AMC) { bv = ld_cluster(&cv, lane); bi = __float_as_int(ld_cluster(reinterpret_cast<const float*>(&ci), lane)); }
    am_warp_best(bv, bi);                             // every warp knows the winner
    if (rank == 0 && tid == 0) {
        tok[b] = bi;
        if (positions) positions[b] += 1;
    }
    if (embed) {
        const uint4* src = reinterpret_cast<const uint4*>(embed + (size_t)bi * D);
        uint4* dst = reinterpret_cast<uint4*>(h + (size_t)b * D);
        for (int v = rank * AMC_THREADS + tid; v < D / 8; v += AMC * AMC_THREADS) dst[v] = __ldg(src + v);
    }
    att_cluster_sync();                               // the others' shared memory has been read
}

// ---------------------------------------------------------------------------------------------
// y[M, N] = x[M, K] . W[N, K]^T in bf16 for up to 8 tokens: the head of a decode step, a stream of W.  One CTA of 16 warps per SM walks over blocks of 16 rows,
// and the warps share K, so that a row is read in one piece.  (A warp with 16 rows of its own over the whole of K needs no sums between warps, but keeps
// 32000 rows open at a time, 64 bytes each: 4.95 TB/s.)  A lane loads 16 bytes of its two rows per 32 k, a block of rows ahead of the arithmetic (128 KB in
// flight per SM at K = 4096); they are the A fragments of two mma.sync as they lie, the tokens' 16 bytes at the same k the B fragments, because a contraction
// does not care which k meet in which lane.  32000 x 4096 in a chain: 38.7 us for one or two tokens (6.78 TB/s), 39.9 for eight, against 45 .. 47 of the
// library and a launch gap before it; K = 2048, 1 / 3 / 8 tokens: 32000 rows 20.7 / 21.3 / 21.3 against 23.0 / 23.2 / 24.0, 50272 rows 31.2 / 32.0 / 32.2 against 36.2 / 36.7 / 37.0.  (With two
// groups of tokens 16 tokens took 45.0 / 44.3: the library's.)
// ---------------------------------------------------------------------------------------------
constexpr int LR_WARPS = 16;
__device__ __forceinline__ void lr_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// NS: steps of 32 k per warp and block (K = 512 NS)
template <int NS>
__global__ void __launch_bounds__(LR_WARPS * 32, 1) k_linear_rows(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ y, int M, int N) {
    constexpr int VECS = 64 * NS, X_STRIDE = VECS + 4;  // 16-byte vectors of a row; token rows 64 bytes apart modulo 128, so that fragment loads are free of bank conflicts
    extern __shared__ __align__(128) uint4 lr_x[];                                   // [M][X_STRIDE]
    __shared__ float red[2][LR_WARPS][128];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int n_blocks = (N + 15) / 16;
    const uint4* base = reinterpret_cast<const uint4*>(w) + warp * (4 * NS) + t;
    auto row = [&](int b, int r) { return base + (size_t)min(b * 16 + r, N - 1) * VECS; };    // clamped loads, guarded stores
    uint4 qa[NS], qb[NS];
    {
        const uint4 *wa = row(blockIdx.x, g), *wb = row(blockIdx.x, g + 8);
#pragma unroll
        for (int u = 0; u < NS; ++u) { qa[u] = __ldg(wa + u * 4); qb[u] = __ldg(wb + u * 4); }
    }
    pdl_launch_dependents();
    pdl_wait();                                       // the tokens are the predecessor's output
    for (int m = 0; m < M; ++m)
        for (int i = tid; i < VECS; i += LR_WARPS * 32) lr_x[m * X_STRIDE + i] = reinterpret_cast<const uint4*>(x)[(size_t)m * VECS + i];
    __syncthreads();
    const uint4* xr = lr_x + min(g, M - 1) * X_STRIDE + warp * (4 * NS) + t;          // a token that does not exist reads the last: its results are dropped
    int buf = 0;
    for (int blk = blockIdx.x; blk < n_blocks; blk += gridDim.x, buf ^= 1) {
        const bool next = blk + (int)gridDim.x < n_blocks;
        const uint4 *na = next ? row(blk + gridDim.x, g) : nullptr, *nb = next ? row(blk + gridDim.x, g + 8) : nullptr;
        float acc[2][4] = {};
#pragma unroll
        for (int u = 0; u < NS; ++u) {
            const uint4 a = qa[u], b = qb[u];
            if (next) { qa[u] = __ldg(na + u * 4); qb[u] = __ldg(nb + u * 4); }
            const uint4 f = xr[u * 4];
            lr_mma(acc[0], a.x, b.x, a.y, b.y, f.x, f.y);
            lr_mma(acc[1], a.z, b.z, a.w, b.w, f.z, f.w);
        }
        *reinterpret_cast<float4*>(&red[buf][warp][lane * 4]) = make_float4(acc[0][0] + acc[1][0], acc[0][1] + acc[1][1], acc[0][2] + acc[1][2], acc[0][3] + acc[1][3]);
        __syncthreads();                              // one barrier per block: the other buffer is rewritten only after the next
        if (tid < 128) {                              // d0,d1 = (row g, tokens 2t, 2t+1); d2,d3 = (row g+8, same tokens)
            const int ln = tid >> 2, i = tid & 3, tok = 2 * (ln & 3) + (i & 1), r = blk * 16 + (ln >> 2) + (i >= 2 ? 8 : 0);
            if (r < N && tok < M) {
                float v[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) v[k] = red[buf][k][tid];
#pragma unroll
                for (int k = 4; k < LR_WARPS; ++k) v[k & 3] += red[buf][k][tid];
                y[(size_t)tok * N + r] = __float2bfloat16_rn((v[0] + v[1]) + (v[2] + v[3]));
            }
        }
    }
}

static inline bool al16p(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace lq

using namespace lq;

template <int HD>
static void launch_attn_cluster(cudaLaunchConfig_t cfg, const __nv_bfloat16* q, int q_row_stride, const __nv_bfloat16* k, const __nv_bfloat16* v, const long long* positions,
                                __nv_bfloat16* out, int Hq, int Hkv, int max_len, float scale, int prefetch) {
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = decode_chain_enabled() ? 1 : 0;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 1; attr[1].val.clusterDim.y = cfg.gridDim.y; attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = 2;
    cudaLaunchKernelEx(&cfg, k_decode_attn<HD, true>, q, q_row_stride, k, v, positions, out, Hq, Hkv, max_len, scale, (float*)nullptr, (unsigned int*)nullptr, prefetch);
}

template <int NS>
static int launch_linear_rows(const void* x, const void* w, void* y, int64_t M, int64_t N, cudaStream_t st) {
    static bool attr_done[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return LQ_EUNSUPPORTED;
    constexpr int row = (64 * NS + 4) * 16;                  // bytes of a staged token
    if (!attr_done[dev]) {
        cudaError_t e = cudaFuncSetAttribute(k_linear_rows<NS>, cudaFuncAttributeMaxDynamicSharedMemorySize, 8 * row);
        if (e != cudaSuccess) { set_cuda_error(e, "cudaFuncSetAttribute(k_linear_rows)"); return LQ_ECUDA; }
        attr_done[dev] = true;
    }
    const int64_t blocks = (N + 15) / 16;
    launch_pdl(k_linear_rows<NS>, dim3((unsigned)(blocks < sm_count() ? blocks : sm_count())), (unsigned)(LR_WARPS * 32), (size_t)M * row, st, (const __nv_bfloat16*)x,
               (const __nv_bfloat16*)w, (__nv_bfloat16*)y, (int)M, (int)N);
    return check_launch("k_linear_rows");
}

extern "C" {

int lq_add_rmsnorm(void* h, const void* delta, const void* gamma, float eps, void* y, int64_t M, int64_t K, int hf_rounding,
                   lq_stream_t stream) {
    if (!h || !gamma || !y || !al16p(h) || !al16p(gamma) || !al16p(y) || (delta && !al16p(delta))) return LQ_EINVAL;
    if (M < 0 || K <= 0 || (K % 8) != 0 || M >= (1ll << 31) || K >= (1ll << 24)) return LQ_EUNSUPPORTED;
    if (M == 0) return LQ_OK;
    { int rc = ensure_device_for(h); if (rc) return rc; }
    const int vpt = (int)((K / 8 + NORM_THREADS - 1) / NORM_THREADS);
#define LQ_NORM_ARGS dim3((unsigned)M), NORM_THREADS, 0, (cudaStream_t)stream, (__nv_bfloat16*)h, (const __nv_bfloat16*)delta, \
                     (const __nv_bfloat16*)gamma, eps, (__nv_bfloat16*)y, (int)K, hf_rounding
    if (vpt <= 1) launch_pdl(k_add_rmsnorm_r<1>, LQ_NORM_ARGS);
    else if (vpt <= 2) launch_pdl(k_add_rmsnorm_r<2>, LQ_NORM_ARGS);
    else if (vpt <= 4) launch_pdl(k_add_rmsnorm_r<4>, LQ_NORM_ARGS);
    else if (vpt <= 6) launch_pdl(k_add_rmsnorm_r<6>, LQ_NORM_ARGS);
    else launch_pdl(k_add_rmsnorm, LQ_NORM_ARGS);
#undef LQ_NORM_ARGS
    return check_launch("k_add_rmsnorm");
}

int lq_rope_kv_store(void* qkv, const int64_t* positions, const float* inv_freq, void* k_cache, void* v_cache, int64_t M,
                     int tokens_per_seq, int Hq, int Hkv, int hd, int64_t max_len, int hf_rounding, lq_stream_t stream) {
    if (!qkv || !positions || !inv_freq || !k_cache || !v_cache) return LQ_EINVAL;
    if (M < 0 || tokens_per_seq < 1 || Hq < 1 || Hkv < 1 || (Hq % Hkv) != 0 || hd < 8 || hd > 512 || (hd % 4) != 0 || max_len < 1 ||
        max_len >= (1ll << 31) || M >= (1ll << 31) || Hq + 2 * Hkv > 65535)
        return LQ_EUNSUPPORTED;
    if (M == 0) return LQ_OK;
    { int rc = ensure_device_for(qkv); if (rc) return rc; }
    // Several heads per thread where all of the work does not fit the chip at once, in vectors of four pairs (8 bytes): 64 tokens of 96 heads of 128 6.9 -> 3.2 us,
    // 400 40 -> 5.7, 3000 297 -> 33.  A thread's four angles come one after the other, and with few heads or heads above 128 a CTA has few to share them, so small
    // calls keep the kernel of one pair per thread: time against it at 1536 / 1792 / 2048 / 2560 / 3072 / 4096 / 6144 (token, head) pairs 1.04 / 0.96 / 0.85 / 0.81 / 0.74 /
    // 0.64 / 0.48 with 48 heads of 128, 1.33 / 1.16 / 1.20 / 1.06 / 0.88 / 0.78 / 0.58 with 48 of 256, 1.16 / 1.04 / 1.06 / 0.94 / 0.81 / 0.69 / 0.48 with 8 of 128,
    // 1.49 / 1.32 / 1.16 / 1.00 / 1.12 / 0.98 / 0.90 with 3 of 128 (heads of 16, 64 and 512, and 4, 6, 12, 24 and 96 of them, lie in between).
    const int heads_all = Hq + 2 * Hkv;
    const int64_t pairs_min = heads_all < 4 ? 6144 : (heads_all < 12 || hd > 128 ? 3072 : 1792);
    if (M * heads_all >= pairs_min && (hd % 8) == 0 && ((reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache)) & 7) == 0) {
        const int per = 256 / (hd / 8), sets = (Hq + 2 * Hkv + per - 1) / per;
        const int64_t want = (4 * (int64_t)sm_count() + M - 1) / M;
        const dim3 grid4((unsigned)M, (unsigned)(want < sets ? want : sets));
        launch_pdl(k_rope_kv_store4, grid4, 256, 0, (cudaStream_t)stream, (__nv_bfloat16*)qkv, (const long long*)positions, inv_freq, (__nv_bfloat16*)k_cache,
                   (__nv_bfloat16*)v_cache, tokens_per_seq, Hq, Hkv, hd, (int)max_len, hf_rounding);
        return check_launch("k_rope_kv_store4");
    }
    dim3 grid((unsigned)M, (unsigned)(Hq + 2 * Hkv));
    launch_pdl(k_rope_kv_store, grid, (unsigned)(hd / 2), 0, (cudaStream_t)stream, (__nv_bfloat16*)qkv, (const long long*)positions, inv_freq,
               (__nv_bfloat16*)k_cache, (__nv_bfloat16*)v_cache, tokens_per_seq, Hq, Hkv, hd, (int)max_len, hf_rounding);
    return check_launch("k_rope_kv_store");
}

static int attn_splits(int64_t B, int Hq, int64_t max_len) {
    const int64_t ctas = B * Hq;
    // As many splits as fit beside one another (four CTAs per SM by registers): rounded up, a few CTAs more than that made a second
    // wave of the whole kernel.  Measured with 32 heads (us, up / down): 4 sequences of 512 keys 14.9 / 11.0, 8: 18.1 / 14.8, 16: 25.9 / 21.3,
    // one of 1500 keys 11.7 / 10.3, four 23.9 / 19.2; also where half of the slots stay empty: 10 sequences (one split instead of two) of 128
    // keys 10.9 / 6.9, of 512 19.5 / 15.0, of 1500 37.9 / 31.6; 12: 20.5 / 16.7 of 512, 47.9 / 41.2 of 1500; 18: 27.2 / 22.5 and 54.5 / 50.5.
    // Nothing lost with 16 heads, or 32 on 8 key heads, at 1 .. 64 sequences of 128 to 1500 keys; from 19 sequences of 32 heads on one split either way.
    int64_t s = 4 * (int64_t)sm_count() / ctas;
    const int64_t cap = (max_len + 63) / 64;                        // at least 64 keys (two rounds of the 16 slots x 2) per split
    if (s > cap) s = cap;
    if (s > 32) s = 32;
    if (s < 1) s = 1;
    return (int)s;
}
// Splits of a (batch, head) that run as one cluster, or 0: tickets.  Eight, four or two (clusters of three, six or sixteen leave room on the
// chip's SM groups: a second wave, up to 40 % slower), from the context lengths at which so many pay, as long as all clusters are
// resident together.  With 65 or more rows the tickets' finer splits win where they are half as many again: 96 rows of 1500 keys 15.0 / 14.1 us,
// 160 rows of 1500 24.0 / 21.9.  Cluster / tickets (us; 32 heads): 1 sequence of 100 keys 4.1 / 5.2, 520 6.1 / 7.4, 1500 9.3 / 10.3; 2: 4.6 / 5.5, 7.5 / 8.5, 11.0 /
// 12.1; 4: 5.8 / 6.7, 9.5 / 9.9, 14.9 / 15.3; 8: 7.2 / 7.5, 12.9 / 13.4, 27.9 / 28.8.
// What a cluster saves at the end is fixed; what it loses by its coarser splits grows with the context (`extra` keys per CTA, 17 to 23 ns each as
// a chain of latencies), and it starts only when a whole cluster finds room beside the predecessor's last CTAs.  So the lines lie where they cross behind a
// projection with weights from memory, in a chain.  Projection and attention, tickets / cluster (us; heads (key heads) x head size): 8 x 128 1000 keys 12.1 / 11.5,
// 2048 13.2 / 15.0; 32 x 128 1500 19.6 / 18.7, 2048 20.0 / 20.8, 4096 24.9 / 27.2; 32 (8) x 128 1500 16.8 / 15.4, 3072 18.2 / 19.5; 7 x 8 x 128 1500 16.8 /
// 15.6; 8 x 8 x 128 1000 15.1 / 16.0, 2048 20.1 / 23.3; 4 x 16 x 64 1000 14.5 / 12.5; clusters of four: 64 x 128 760 25.8 / 24.7, 1000 26.3 / 26.7.  Launched by itself the attention
// would still gain from clusters up to about twice as many extra keys (32 x 128 3072 keys 15.0 / 14.0 us, from 16384 on 46.8 / 49.6; 8 x 128 8192 14.1 / 22.0), and so do
// caches that are partly filled (70 %: 32 x 128 2048 keys 19.6 / 18.7, 16 x 128 16.0 / 14.8): the line is drawn a little beyond the crossing of full ones.
// Above 60 rows of 128-wide heads eight splits leave no room beside the projection: they lose from 24 extra keys on (1700 keys), and up to there whole
// decode steps differ by 2 % either way (2 x 32 heads 1500 keys 102.5 / 100.9 us, 4 x 16 82.1 / 84.0).
static int attn_cluster(int64_t B, int Hq, int hd, int64_t max_len) {
    const int64_t rows = B * Hq, sms = sm_count();
    const int c = max_len >= 512 && rows * 16 <= 7 * sms ? 8 : max_len >= 192 && rows * 8 <= 7 * sms ? 4 : max_len > 64 && rows * 2 <= 4 * sms ? 2 : 0;
    const int tickets = attn_splits(B, Hq, max_len);
    if (!c || (rows > 64 && 10 * c < 7 * tickets)) return 0;
    const int64_t extra = (max_len + c - 1) / c - (max_len + tickets - 1) / tickets;
    return extra <= (c < 8 ? 96 : hd == 64 || rows * 32 <= 13 * sms ? 144 : 24) ? c : 0;
}

size_t lq_decode_attention_workspace_bytes(int64_t B, int Hq, int hd, int64_t max_len) {
    if (B <= 0 || Hq <= 0 || hd <= 0 || max_len <= 0) return 0;
    const int s = attn_splits(B, Hq, max_len);
    return (size_t)B * Hq * ((size_t)s * (hd + 2) * sizeof(float) + sizeof(unsigned int));
}

int lq_decode_attention(const void* q, int64_t q_row_stride, const void* k_cache, const void* v_cache, const int64_t* positions,
                        void* out, int64_t B, int Hq, int Hkv, int hd, int64_t max_len, float scale, void* workspace,
                        size_t workspace_bytes, lq_stream_t stream) {
    if (!q || !k_cache || !v_cache || !positions || !out || !al16p(q) || !al16p(k_cache) || !al16p(v_cache)) return LQ_EINVAL;
    if (B < 0 || Hq < 1 || Hkv < 1 || (Hq % Hkv) != 0 || (hd != 64 && hd != 128) || max_len < 1 || max_len >= (1ll << 31) ||
        B * Hq >= (1ll << 31) || (q_row_stride % 8) != 0)
        return LQ_EUNSUPPORTED;
    if (B == 0) return LQ_OK;
    { int rc = ensure_device_for(q); if (rc) return rc; }
    const int cluster = attn_cluster(B, Hq, hd, max_len), splits = cluster ? cluster : attn_splits(B, Hq, max_len);
    float* part = nullptr; unsigned int* tickets = nullptr;
    if (attn_splits(B, Hq, max_len) > 1) {              // (clusters leave it untouched)
        if (!workspace || workspace_bytes < lq_decode_attention_workspace_bytes(B, Hq, hd, max_len) || !al16p(workspace)) return LQ_EWORKSPACE;
        part = (float*)workspace;
        tickets = (unsigned int*)(part + (size_t)B * Hq * splits * (hd + 2));
    }
    dim3 grid((unsigned)(B * Hq), (unsigned)splits);
    cudaStream_t st = (cudaStream_t)stream;
    // The early request: in a chain only, where there is a wait to hide it behind (outside, the position read twice costs 0.4 us: 4 % over 239 shapes,
    // 16 x 32 heads of 32 keys 4.1 / 4.9), where all CTAs start beside the predecessor's last ones and no two of them read the same keys
    // (640 rows of 100 keys 9.4 / 9.9 us with it, 320 rows on 80 key heads 5.6 / 5.9; 1 to 16 sequences of 32 heads 2 to 7 % shorter with it).
    // (A template parameter in its place: 0.07 us less for a launch outside a chain, 0.2 % more for a decode step of 16 sequences.)
    const int prefetch = decode_chain_enabled() && Hq == Hkv && B * Hq * splits <= 4 * (int64_t)sm_count() ? 1 : 0;
    auto launch = [&](auto kern) {
        launch_pdl(kern, grid, (unsigned)ATT_THREADS, 0, st, (const __nv_bfloat16*)q, (int)q_row_stride, (const __nv_bfloat16*)k_cache, (const __nv_bfloat16*)v_cache,
                   (const long long*)positions, (__nv_bfloat16*)out, Hq, Hkv, (int)max_len, scale, part, tickets, prefetch);
    };
    if (cluster) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = grid; cfg.blockDim = dim3(ATT_THREADS); cfg.stream = st;
        (hd == 128 ? launch_attn_cluster<128> : launch_attn_cluster<64>)(
            cfg, (const __nv_bfloat16*)q, (int)q_row_stride, (const __nv_bfloat16*)k_cache, (const __nv_bfloat16*)v_cache, (const long long*)positions,
            (__nv_bfloat16*)out, Hq, Hkv, (int)max_len, scale, prefetch);
    } else if (hd == 128) {
        launch(k_decode_attn<128, false>);
    } else {
        launch(k_decode_attn<64, false>);
    }
    return check_launch("k_decode_attn");
}

int lq_argmax_embed(const void* logits, int64_t logits_stride, int64_t B, int64_t V, const void* embed, int64_t D, int64_t* tok,
                    int64_t* positions, void* h, lq_stream_t stream) {
    if (!logits || !tok || (embed && (!h || !al16p(embed) || !al16p(h)))) return LQ_EINVAL;
    if (B < 0 || V < 1 || V >= (1ll << 31) - 8 || B >= (1ll << 31) || logits_stride < V || (embed && (D < 8 || (D % 8) != 0 || D >= (1ll << 31))))
        return LQ_EUNSUPPORTED;
    if (B == 0) return LQ_OK;
    { int rc = ensure_device_for(logits); if (rc) return rc; }
    const int vec = al16p(logits) && (logits_stride % 8) == 0 && (V % 8) == 0;
    // One CTA / a cluster per row, us in a chain: 32000 logits 1 or 2 rows 5.2 / 3.9, 16 rows 5.4 / 4.6, 64 rows 5.5 / 7.4 (four waves of barriers); 8192 logits 3.2 / 3.5;
    // 16384 logits 12 rows 0.96 of the time, 18 rows 1.05, 24576 logits 18 rows 0.98; 50272 logits 2 rows 7.0 / 4.5.  Rows beyond the SMs' number of clusters pay
    // for large vocabularies, except where single CTAs fill the chip just once: 98304 logits 64 rows 11.0 / 10.9, 128 rows 11.3 / 14.4, 256 rows 20.9 / 23.6;
    // 150000 logits 48 / 96 / 128 / 192 / 256 / 1000 rows 0.77 / 0.93 / 1.15 / 0.86 / 0.96 / 0.84 of the time, 256000 logits 0.69 / 0.85 / 1.00 / 0.68 / 0.81 / 0.79.
    const int64_t sms = sm_count();
    const bool few_rows = B * AMC <= sms && (V >= 24576 || 3 * B * AMC <= 2 * sms);
    const bool long_rows = (V >= 98304 && B <= 64) || (V >= 131072 && (3 * B <= 2 * sms || B > sms) && B <= (1 << 27));
    if (vec && V >= 16384 && (few_rows || long_rows)) {
        launch_pdl(k_argmax_embed_cluster, dim3((unsigned)(B * AMC)), (unsigned)AMC_THREADS, 0, (cudaStream_t)stream, (const __nv_bfloat16*)logits, logits_stride, (int)V,
                   (const __nv_bfloat16*)embed, (int)D, (long long*)tok, (long long*)positions, (__nv_bfloat16*)h);
        return check_launch("k_argmax_embed_cluster");
    }
    launch_pdl(k_argmax_embed, dim3((unsigned)B), (unsigned)AM_THREADS, 0, (cudaStream_t)stream, (const __nv_bfloat16*)logits,
               logits_stride, (int)V, vec, (const __nv_bfloat16*)embed, (int)D, (long long*)tok, (long long*)positions,
               (__nv_bfloat16*)h);
    return check_launch("k_argmax_embed");
}

int lq_linear_rows(const void* x, const void* w, void* y, int64_t M, int64_t N, int64_t K, lq_stream_t stream) {
    if (!x || !w || !y || !al16p(x) || !al16p(w)) return LQ_EINVAL;
    if (M < 0 || M > 8 || N < 1 || N >= (1ll << 30) || (K != 2048 && K != 4096)) return LQ_EUNSUPPORTED;
    if (M == 0) return LQ_OK;
    { int rc = ensure_device_for(x); if (rc) return rc; }
    return K == 2048 ? launch_linear_rows<4>(x, w, y, M, N, (cudaStream_t)stream) : launch_linear_rows<8>(x, w, y, M, N, (cudaStream_t)stream);
}

int lq_silu_mul(const void* gate_up, void* act, int64_t M, int64_t I, int hf_rounding, lq_stream_t stream) {
    if (!gate_up || !act || !al16p(gate_up) || !al16p(act)) return LQ_EINVAL;
    if (M < 0 || I <= 0 || (I % 8) != 0 || I >= (1ll << 30)) return LQ_EUNSUPPORTED;
    if (M == 0) return LQ_OK;
    { int rc = ensure_device_for(gate_up); if (rc) return rc; }
    const int64_t total = M * (I / 8);
    int64_t g = (total + 255) / 256;
    const int64_t cap = (int64_t)sm_count() * 8;
    if (g > cap) g = cap;
    launch_pdl(k_silu_mul, dim3((unsigned)g), 256u, 0, (cudaStream_t)stream, (const __nv_bfloat16*)gate_up, (__nv_bfloat16*)act, M, (int)I, hf_rounding);
    return check_launch("k_silu_mul");
}

}  // extern "C"
