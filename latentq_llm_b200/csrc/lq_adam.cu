// Fused optimizer step of the latent fine-tune path: one HBM pass per quantized weight instead of the ~40
// tensor-op passes of MyAdam.update_step (utils/quant.py:1052-1148), and one launch for all the small dense
// parameters.  Every intermediate is rounded where the reference's torch ops round it (each op computes in fp32
// and stores in the tensor dtype), so codes, residual words and optimizer states come out bit-identical to the
// op-by-op route.
//
// Where torch's CUDA functors are single expressions (`a + alpha * b`, `a + alpha * (b / c)`), nvcc contracts the
// multiply-add into an FMA in torch's own build; the same contraction is spelled out here with __fmaf_rn
// (checked on the GPU against torch's add_/addcmul_/addcdiv_ on 2^24-element bf16 tensors: the separately
// rounded forms of add_(alpha) and addcdiv_ differ from torch in a few elements per million, the fused ones never).
#include <type_traits>
#include <cstdlib>

#include "lq_requant.cuh"

namespace lq {

struct AdamParams {
    RequantParams rq;
    const void* grad; int grad_dtype;
    uint8_t* st1; float* sc1; float* tm1;
    uint8_t* st2; float* sc2; float* tm2;
    int opt_shift;                 // log2(elements per optimizer-state block): 11 or 7
    int64_t n_tiles;               // tiles of 256 words
    lq_adam_hyper h;
};

// m <- m*b1 ; m <- m + (1-b1)*g ; v <- v*b2 ; v <- v + (1-b2)*(g*g) ; d <- sqrt(v) ; d <- d + eps ; each stored in
// the chain dtype (utils/quant.py:1098-1101).  Returns m and d = sqrt(v)+eps.
template <bool BF>
__device__ __forceinline__ void adam_moments(const lq_adam_hyper& h, float g, float& m, float& v_to_d) {
    m = rb<BF>(__fmul_rn(m, h.beta1));
    m = rb<BF>(__fmaf_rn(h.one_minus_beta1, g, m));
    float v = rb<BF>(__fmul_rn(v_to_d, h.beta2));
    v = rb<BF>(__fmaf_rn(h.one_minus_beta2, __fmul_rn(g, g), v));
    float d = rb<BF>(__fsqrt_rn(v));
    v_to_d = rb<BF>(__fadd_rn(d, h.eps));
}
// p <- p + (-step_size) * (m / d)   (addcdiv_, utils/quant.py:1105)
template <bool BF>
__device__ __forceinline__ float adam_apply(const lq_adam_hyper& h, float p, float m, float d) {
    return rb<BF>(__fmaf_rn(h.neg_step_size, __fdiv_rn(m, d), p));
}

__device__ __forceinline__ uint8_t opt8_encode1(float x, float mx, float s) {
    const float t = rne(div_rn(__fsub_rn(mx, x), div_by(s)));
    return (uint8_t)(f2bits(fminf(fmaxf(t, 0.0f), 255.0f)) & 0xffu);
}
__device__ __forceinline__ uint2 opt8_encode8(const float (&x)[8], float mx, float s) {
    const DivBy by_s = div_by(s);
    uint32_t b[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        float t = rne(div_rn(__fsub_rn(mx, x[k]), by_s));
        t = fminf(fmaxf(t, 0.0f), 255.0f);
        b[k] = f2bits(t) & 0xffu;
    }
    uint2 o;
    o.x = b[0] | (b[1] << 8) | (b[2] << 16) | (b[3] << 24);
    o.y = b[4] | (b[5] << 8) | (b[6] << 16) | (b[7] << 24);
    return o;
}

// One thread per word of 8 elements; a CTA covers 256 words = one 2048-element optimizer-state block, or sixteen
// 128-element blocks (16 lanes each).
template <int WBITS, int CODEC, int DITHER, bool BF>
__global__ void __launch_bounds__(256) k_adam_quant(const AdamParams p) {
    __shared__ float s_red[4][8];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int64_t tile = blockIdx.x; tile < p.n_tiles; tile += gridDim.x) {
        const int64_t w = tile * 256 + tid;
        const bool active = w < p.rq.n_words;
        const int64_t e0 = w * 8;
        float lat[8], m[8], d[8];
        float s = 1.0f, z = 0.0f;
        float mn1 = INFINITY, mx1 = -INFINITY, mn2 = INFINITY, mx2 = -INFINITY;
        int64_t ob = 0;
        if (active) {
            const int64_t g = p.rq.group_shift >= 0 ? (e0 >> p.rq.group_shift) : (e0 / p.rq.group);
            s = load1(p.rq.scales, p.rq.qp_dtype, g);
            z = (WBITS == 4) ? load1(p.rq.zeros, p.rq.qp_dtype, g) : 0.0f;
            ob = e0 >> p.opt_shift;
            const float s1 = p.sc1[ob], t1 = p.tm1[ob], s2 = p.sc2[ob], t2 = p.tm2[ob];   // rewritten below: plain loads
            const uint2 q1 = *reinterpret_cast<const uint2*>(p.st1 + e0);
            const uint2 q2 = *reinterpret_cast<const uint2*>(p.st2 + e0);
            float gr[8];
            load8(p.grad, p.grad_dtype, e0, gr);
            latent_load<WBITS, CODEC, BF>(p.rq, w, s, z, lat);
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const float c1 = u2f(((k < 4 ? q1.x : q1.y) >> (8 * (k & 3))) & 0xffu);
                const float c2 = u2f(((k < 4 ? q2.x : q2.y) >> (8 * (k & 3))) & 0xffu);
                m[k] = rb<BF>(__fsub_rn(t1, __fmul_rn(c1, s1)));           // DeQfunc_8bit_opt(...).to(dtype)
                const float r2 = __fsub_rn(t2, __fmul_rn(c2, s2));
                d[k] = rb<BF>(__fmul_rn(r2, r2));                          // (s2 * s2).to(dtype)
                adam_moments<BF>(p.h, gr[k], m[k], d[k]);
                lat[k] = adam_apply<BF>(p.h, lat[k], m[k], d[k]);
                mn1 = fminf(mn1, m[k]); mx1 = fmaxf(mx1, m[k]);
                mn2 = fminf(mn2, d[k]); mx2 = fmaxf(mx2, d[k]);
            }
        }
        // min/max over the optimizer-state block: 16 lanes, then (2048-element blocks) the whole CTA
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) {
            mn1 = fminf(mn1, __shfl_xor_sync(0xffffffffu, mn1, o)); mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, o));
            mn2 = fminf(mn2, __shfl_xor_sync(0xffffffffu, mn2, o)); mx2 = fmaxf(mx2, __shfl_xor_sync(0xffffffffu, mx2, o));
        }
        if (p.opt_shift == 11) {
            mn1 = fminf(mn1, __shfl_xor_sync(0xffffffffu, mn1, 16)); mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 16));
            mn2 = fminf(mn2, __shfl_xor_sync(0xffffffffu, mn2, 16)); mx2 = fmaxf(mx2, __shfl_xor_sync(0xffffffffu, mx2, 16));
            __syncthreads();                                               // previous tile's readers are done
            if (lane == 0) { s_red[0][warp] = mn1; s_red[1][warp] = mx1; s_red[2][warp] = mn2; s_red[3][warp] = mx2; }
            __syncthreads();
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                mn1 = fminf(mn1, s_red[0][i]); mx1 = fmaxf(mx1, s_red[1][i]);
                mn2 = fminf(mn2, s_red[2][i]); mx2 = fmaxf(mx2, s_red[3][i]);
            }
        }
        if (active) {
            const float ns1 = __fadd_rn(__fdiv_rn(__fsub_rn(mx1, mn1), 255.0f), 1e-10f);
            const float ns2 = __fadd_rn(__fdiv_rn(__fsub_rn(mx2, mn2), 255.0f), 1e-10f);
            *reinterpret_cast<uint2*>(p.st1 + e0) = opt8_encode8(m, mx1, ns1);
            *reinterpret_cast<uint2*>(p.st2 + e0) = opt8_encode8(d, mx2, ns2);
            const bool leader = p.opt_shift == 11 ? (tid == 0) : ((tid & 15) == 0);
            if (leader) { p.sc1[ob] = ns1; p.tm1[ob] = mx1; p.sc2[ob] = ns2; p.tm2[ob] = mx2; }
            latent_store<WBITS, CODEC, DITHER, BF>(p.rq, w, s, z, lat);
        }
    }
}

// ---------------------------------------------------------------------------------------------------------------
// Fast variant of the production configuration (bf16 chain, bf16 qparams and gradient, 3-fold codec, hash dither, group a
// power of two >= 8).  Same results as k_adam_quant, bit for bit.  The kernel is bound by instruction issue, not by its
// 8 bytes per weight, so every step is the cheapest form that provably rounds the same way:
//   states    decoded from two 256-entry tables per 2048-element block (one entry of each per thread): code -> bf16(m) * beta1
//             and bf16(s2^2) * beta2, both already rounded.  128-element blocks have too few elements per table and decode
//             in registers (LUT = false).
//   sqrt      sqrt.approx (relative error <= 2^-23): the root of an 8-bit significand is at least 2^-19 (relative) away from
//             every bf16 rounding boundary (the boundary's square has odd quarters, the operand is an integer on that scale),
//             so the bf16 result is that of the exactly rounded root.
//   m / d     rcp.approx and one residual correction: the quotient of two 8-bit significands is at least 2^-33 away from
//             every midpoint of two fp32 numbers, the corrected quotient is 2^-44 off before its rounding.
//   states    encoded with a quotient from a two-term reciprocal and one residual correction (Markstein's theorem, see div_by), as is
//             the division of the block's range by 255.
//   fp32      two elements per instruction (fma / mul / add .f32x2) for int4 codes: 83 -> 74 instructions per weight, 157 -> 149 us for 4096 x
//             11008.  The int8 kernel has no registers left for the pairs (64, two teams of 256 threads): 11008 x 4096 172 -> 178 us, so it keeps
//             one element per instruction.
//   requantize  everything after Z = w/scale + zero from the table of the requantize fast path (int4: a byte per bf16 pattern,
//             |Z| < 64; int8: two bytes, |Z| < 256); the kernel keeps the two runs of it that can be looked up and puts its other
//             tables into the gap between them.
// int4 codes: 50 KB and 256 threads per CTA, three CTAs per SM (four would fit, but at 64 registers the loop spills: 176 instead of
// 157 us for 4096 x 11008); int8 codes: 100 KB, so two teams of 256 threads share the tables of a CTA and two CTAs fit.
// Measured, a whole optimizer step of one 4096 x 11008 weight: int4 268 -> 149 us (2.4 TB/s), int8 586 -> 177 us.
// A word whose Z leaves the table's range or is not finite, and every word of a block whose moments are not all finite, is
// recomputed with IEEE operations (adam_word_generic).
// ---------------------------------------------------------------------------------------------------------------
constexpr int ADAM_TRES_REPL = 8;
template <int WBITS> struct AdamFast {
    static constexpr int TEAMS = WBITS == 8 ? 2 : 1;
    static constexpr int THREADS = TEAMS * 256;
    static constexpr int MIN_CTAS = WBITS == 8 ? 2 : 3;
    static constexpr int ENTRY = WBITS == 8 ? 2 : 1;                     // bytes per table entry
    static constexpr int RUN = (WBITS == 8 ? 0x4380 : 0x4280) * ENTRY;   // bf16 patterns of [0, 256) / [0, 64)
    static constexpr int NEG = 0x8000 * ENTRY;                           // the run of the negative patterns
    static constexpr int TRES = (RUN + 1023) / 1024 * 1024;              // residual decode table
    static constexpr int LUT = TRES + 256 * ADAM_TRES_REPL * 4;          // per team: [256] first state, [256] second state
    static constexpr int RED = LUT + TEAMS * 2 * 256 * 4;                // per team: block extrema of the 8 warps
    static constexpr int PRM = RED + TEAMS * 64;                         // per team: (s1, t1, s2, t2) of this tile and the next
    static constexpr int SMEM = NEG + RUN;
    static constexpr uint32_t Z_LIMIT = WBITS == 8 ? 0x3c803c80u : 0x3d803d80u;    // carries into bit 15 from |Z| = 256 / 64 on
    static_assert(PRM + TEAMS * 32 <= NEG && RUN % 16 == 0, "tables in the gap of the encode table");
};

__device__ __forceinline__ uint32_t pack2(float a, float b) {       // bf16 roundings of two values, one conversion
    const __nv_bfloat162 q = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&q);
}
__device__ __forceinline__ float lo2f(uint32_t u) { return __uint_as_float(u << 16); }
__device__ __forceinline__ float hi2f(uint32_t u) { return __uint_as_float(u & 0xffff0000u); }
__device__ __forceinline__ __nv_bfloat162 asbf2(uint32_t u) { return *reinterpret_cast<const __nv_bfloat162*>(&u); }
__device__ __forceinline__ uint32_t asu32(__nv_bfloat162 v) { return *reinterpret_cast<const uint32_t*>(&v); }
__device__ __forceinline__ uint32_t min2(uint32_t a, uint32_t b) { return asu32(__hmin2(asbf2(a), asbf2(b))); }
__device__ __forceinline__ uint32_t max2(uint32_t a, uint32_t b) { return asu32(__hmax2(asbf2(a), asbf2(b))); }
__device__ __forceinline__ float sqrt_approx(float x) { float r; asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
__device__ __forceinline__ float rcp_approx(float x) { float r; asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
// Two fp32 values.  f32x2: in one 64-bit register pair, each operation one instruction for two IEEE results; float2: one by one.
typedef unsigned long long f32x2;
template <typename V> __device__ __forceinline__ V f2(float a, float b);
template <> __device__ __forceinline__ f32x2 f2<f32x2>(float a, float b) { f32x2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r; }
template <> __device__ __forceinline__ float2 f2<float2>(float a, float b) { return make_float2(a, b); }
template <typename V> __device__ __forceinline__ V f2(float a) { return f2<V>(a, a); }
template <typename V> __device__ __forceinline__ V bf2f(uint32_t u) { return f2<V>(lo2f(u), hi2f(u)); }            // the two values of a bf16 pair
__device__ __forceinline__ float2 of2(f32x2 v) { float2 r; asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v)); return r; }
__device__ __forceinline__ float2 of2(float2 v) { return v; }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) { f32x2 r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return make_float2(__fmaf_rn(a.x, b.x, c.x), __fmaf_rn(a.y, b.y, c.y)); }
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) { f32x2 r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return make_float2(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)); }
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) { f32x2 r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return make_float2(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y)); }
template <typename V> __device__ __forceinline__ uint32_t packv(V v) { const float2 f = of2(v); return pack2(f.x, f.y); }
// -(a / b) for pairs of bf16-valued a and b, 2^-64 <= b <= 2^64: see above (the residual's sign keeps that of a zero quotient)
template <typename V> __device__ __forceinline__ V neg_div_bf16(V a, V b) {
    const float2 bb = of2(b);
    const V ny = f2<V>(rcp_approx(-bb.x), rcp_approx(-bb.y)), nq = mul2(a, ny);
    return fma2(fma2(nq, b, a), ny, nq);
}
// (scale, its reciprocal as RN(1/s) + remainder) of one 8-bit state block: s = (mx - mn) / 255 + 1e-10
struct OptScale { float s, r, rl; };
__device__ __forceinline__ OptScale opt8_scale(float mx, float mn) {
    constexpr float r255 = 1.0f / 255.0f, r255l = (float)(1.0 / 255.0 - (double)r255);
    const float a = __fsub_rn(mx, mn);
    float q = __fmaf_rn(a, r255, __fmul_rn(a, r255l));               // a / 255, correctly rounded (below 2^-100 the 1e-10 hides it)
    q = __fmaf_rn(__fmaf_rn(-q, 255.0f, a), r255, q);
    OptScale o;
    o.s = __fadd_rn(q, 1e-10f);
    o.r = __frcp_rn(o.s);
    o.rl = __fmul_rn(__fmaf_rn(-o.s, o.r, 1.0f), o.r);
    return o;
}
template <typename V>
__device__ __forceinline__ uint32_t opt8_codes2(uint32_t x, float mx, const OptScale& o) {        // codes of a bf16 pair in bytes 0 and 1
    const V r = f2<V>(o.r), a = fma2(bf2f<V>(x), f2<V>(-1.0f), f2<V>(mx));
    V q = fma2(a, r, mul2(a, f2<V>(o.rl)));
    q = fma2(fma2(q, f2<V>(-o.s), a), r, q);
    const float2 c = of2(add2(q, f2<V>(MAGIC_RNE)));                 // 0 <= q <= 255 (1 + 2^-22)
    return __byte_perm(__float_as_uint(c.x), __float_as_uint(c.y), 0x0040);
}
template <typename V>
__device__ __forceinline__ uint32_t opt8_codes4(uint32_t p01, uint32_t p23, float mx, const OptScale& o) {
    return __byte_perm(opt8_codes2<V>(p01, mx, o), opt8_codes2<V>(p23, mx, o), 0x5410);
}

// One word from its inputs in memory (nothing of it has been written yet) and the block parameters of its states before (s, t) and
// after (ns, mx) the step, with IEEE divisions and roots and the generic requantize.  Elements come one at a time through memory:
// the cold path must not cost the hot one registers.
template <int WBITS>
__device__ __forceinline__ void adam_word_generic(const AdamParams& p, const int64_t w, const float s1, const float t1, const float s2, const float t2,
                                                  const float mx1, const float ns1, const float mx2, const float ns2) {
    const int64_t e0 = w * 8;
    const int64_t g = p.rq.group_shift >= 0 ? (e0 >> p.rq.group_shift) : (e0 / p.rq.group);
    const float s = load1(p.rq.scales, p.rq.qp_dtype, g), z = (WBITS == 4) ? load1(p.rq.zeros, p.rq.qp_dtype, g) : 0.0f;
    float lat[8];
    latent_load<WBITS, LQ_CODEC_THREEFOLD, true>(p.rq, w, s, z, lat);
    const __nv_bfloat16* grad = reinterpret_cast<const __nv_bfloat16*>(p.grad) + e0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const float gr = __bfloat162float(grad[k]);
        float m = bf16r(__fsub_rn(t1, __fmul_rn((float)p.st1[e0 + k], s1)));
        m = bf16r(__fmaf_rn(p.h.one_minus_beta1, gr, bf16r(__fmul_rn(m, p.h.beta1))));
        const float r2 = __fsub_rn(t2, __fmul_rn((float)p.st2[e0 + k], s2));
        float d = bf16r(__fmul_rn(bf16r(__fmul_rn(r2, r2)), p.h.beta2));
        d = bf16r(__fmaf_rn(p.h.one_minus_beta2, __fmul_rn(gr, gr), d));
        d = bf16r(__fadd_rn(bf16r(__fsqrt_rn(d)), p.h.eps));
        lat[k] = bf16r(__fmaf_rn(p.h.neg_step_size, __fdiv_rn(m, d), lat[k]));
        p.st1[e0 + k] = opt8_encode1(m, mx1, ns1);
        p.st2[e0 + k] = opt8_encode1(d, mx2, ns2);
    }
    latent_store<WBITS, LQ_CODEC_THREEFOLD, LQ_DITHER_HASH, true>(p.rq, w, s, z, lat);
}

// row_magic (int8 codes): ceil(2^64 / words per weight row)
template <int WBITS, bool USE_RES, bool LUT>
__global__ void __launch_bounds__(AdamFast<WBITS>::THREADS, AdamFast<WBITS>::MIN_CTAS)
k_adam_fast(const __grid_constant__ AdamParams p, const int enc_slot, const uint64_t row_magic) {
    using AF = AdamFast<WBITS>;
    constexpr bool W8 = WBITS == 8;
    using V = typename std::conditional<W8, float2, f32x2>::type;
    extern __shared__ __align__(16) uint8_t asm_[];
    const uint8_t* encz = asm_;
    const uint16_t* enc8 = reinterpret_cast<const uint16_t*>(asm_);
    uint32_t* tres = reinterpret_cast<uint32_t*>(asm_ + AF::TRES);
    {
        const uint4* src = W8 ? reinterpret_cast<const uint4*>(g_enc8_table[enc_slot]) : reinterpret_cast<const uint4*>(g_encz_table[enc_slot]);
        uint4* dst = reinterpret_cast<uint4*>(asm_);
        for (int i = threadIdx.x; i < AF::RUN / 16; i += AF::THREADS) { dst[i] = __ldg(src + i); dst[AF::NEG / 16 + i] = __ldg(src + AF::NEG / 16 + i); }
        for (int b = threadIdx.x; b < 256; b += AF::THREADS) {
            const uint32_t lo = f32_to_bf16_bits(bf16r(res3_decode((uint32_t)b >> 4, p.rq.dec)));
            const uint32_t hi = f32_to_bf16_bits(bf16r(res3_decode((uint32_t)b & 15u, p.rq.dec)));
            for (int r = 0; r < ADAM_TRES_REPL; ++r) tres[b * ADAM_TRES_REPL + r] = lo | (hi << 16);
        }
    }
    __syncthreads();
    const int team = AF::TEAMS == 1 ? 0 : (int)(threadIdx.x >> 8), tid = threadIdx.x & 255, lane = tid & 31, warp = tid >> 5;
    float* lut = reinterpret_cast<float*>(asm_ + AF::LUT) + team * 512;
    uint2* red = reinterpret_cast<uint2*>(asm_ + AF::RED) + team * 8;
    float4* prm = reinterpret_cast<float4*>(asm_ + AF::PRM) + team * 2;       // for the cold path: keeps four registers free
    int parity = 0;
    auto team_sync = [&] {
        if (AF::TEAMS == 1) __syncthreads();
        else asm volatile("bar.sync %0, 256;" ::"r"(team + 1) : "memory");
    };
    const uint32_t tres_lane = tid & (ADAM_TRES_REPL - 1);
    const unsigned short* scales = reinterpret_cast<const unsigned short*>(p.rq.scales);
    const unsigned short* zeros = reinterpret_cast<const unsigned short*>(p.rq.zeros);
    const uint32_t n_words = (uint32_t)p.rq.n_words;
    const int gsh = p.rq.group_shift - 3;                     // word index -> group index
    const int osh = p.opt_shift - 3;                          // word index -> optimizer-state block
    const uint32_t c128u = 0x43004300u;
    // the loads of the next tile are in flight while the current one is computed
    struct In { uint2 q1, q2, pk; uint4 gv; uint32_t rw, sb, zb; float s1, t1, s2, t2; };
    auto load_in = [&](uint32_t w) -> In {
        In in;
        const uint32_t g = W8 ? (uint32_t)__umul64hi((uint64_t)w, row_magic) : w >> gsh, ob = w >> osh;
        in.q1 = *reinterpret_cast<const uint2*>(p.st1 + (size_t)w * 8);
        in.q2 = *reinterpret_cast<const uint2*>(p.st2 + (size_t)w * 8);
        in.gv = __ldg(reinterpret_cast<const uint4*>(p.grad) + w);
        if (W8) in.pk = __ldg(reinterpret_cast<const uint2*>(p.rq.codes_in) + w);
        else in.pk = make_uint2(__ldg(reinterpret_cast<const uint32_t*>(p.rq.codes_in) + w), 0u);
        in.rw = USE_RES ? (uint32_t)__ldg(p.rq.words_in + w) : 0u;
        in.sb = __ldg(scales + g); in.zb = W8 ? 0u : __ldg(zeros + g);
        in.s1 = p.sc1[ob]; in.t1 = p.tm1[ob]; in.s2 = p.sc2[ob]; in.t2 = p.tm2[ob];
        return in;
    };
    In nxt;
    nxt.q1 = nxt.q2 = nxt.pk = make_uint2(0u, 0u); nxt.gv = make_uint4(0u, 0u, 0u, 0u); nxt.rw = nxt.zb = 0u; nxt.sb = 0x3f80u;
    nxt.s1 = nxt.t1 = nxt.s2 = nxt.t2 = 0.0f;
    const uint32_t tile0 = blockIdx.x * AF::TEAMS + team, tile_step = gridDim.x * AF::TEAMS;
    if (tile0 < (uint32_t)p.n_tiles && tile0 * 256u + (uint32_t)tid < n_words) nxt = load_in(tile0 * 256u + (uint32_t)tid);
    for (uint32_t tile = tile0; tile < (uint32_t)p.n_tiles; tile += tile_step) {
        const uint32_t w = tile * 256u + (uint32_t)tid;
        const bool active = LUT || w < n_words;               // LUT: whole 2048-element blocks only
        const In in = nxt;
        {
            const uint32_t wn = w + tile_step * 256u;
            if (tile + tile_step < (uint32_t)p.n_tiles && wn < n_words) nxt = load_in(wn);
        }
        auto dec1 = [&](float c) { return bf16r(__fmul_rn(bf16r(__fsub_rn(in.t1, __fmul_rn(c, in.s1))), p.h.beta1)); };     // m * beta1
        auto dec2 = [&](float c) { const float r = __fsub_rn(in.t2, __fmul_rn(c, in.s2)); return bf16r(__fmul_rn(bf16r(__fmul_rn(r, r)), p.h.beta2)); };
        if (LUT) {
            const float c = u2f((uint32_t)tid);
            lut[tid] = dec1(c); lut[256 + tid] = dec2(c);
            if (tid == 0) prm[parity] = make_float4(in.s1, in.t1, in.s2, in.t2);
            team_sync();
        }
        uint32_t lat[4], m[4], d[4];
        uint32_t mn1 = 0x7f807f80u, mx1 = 0xff80ff80u, mn2 = 0x7f807f80u, mx2 = 0xff80ff80u;
        if (active) {
            // latent weights: bf16((q - z) * s) (+ bf16(bf16(res * s) + that)), packed
            const __nv_bfloat162 s2 = asbf2(in.sb * 0x00010001u);
            const __nv_bfloat162 z128 = __hadd2_rn(asbf2(in.zb * 0x00010001u), asbf2(c128u));
            const uint32_t lo_n = in.pk.x & 0x0F0F0F0Fu, hi_n = (in.pk.x >> 4) & 0x0F0F0F0Fu;
            const uint32_t c03 = __byte_perm(hi_n, lo_n, 0x5140), c47 = __byte_perm(hi_n, lo_n, 0x7362);
            const uint32_t gw[4] = {in.gv.x, in.gv.y, in.gv.z, in.gv.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                __nv_bfloat162 v;
                if (W8) {
                    // byte ^ 0x80 = code + 128 in the mantissa of fp16 1024.0, minus 1152: exact, as is the integer in bf16
                    const uint32_t h2 = __byte_perm(((j < 2) ? in.pk.x : in.pk.y) ^ 0x80808080u, 0x64646464u, (j & 1) ? 0x4342 : 0x4140);
                    const float2 cf = __half22float2(__hsub2(*reinterpret_cast<const __half2*>(&h2), __floats2half2_rn(1152.0f, 1152.0f)));
                    v = __hmul2_rn(__floats2bfloat162_rn(cf.x, cf.y), s2);
                } else {
                    const uint32_t pair = __byte_perm((j < 2) ? c03 : c47, 0x43434343u, (j & 1) ? 0x4342 : 0x4140);
                    v = __hmul2_rn(__hsub2_rn(asbf2(pair), z128), s2);
                }
                if (USE_RES) {
                    const uint32_t b = (in.rw >> (24 - 8 * j)) & 0xffu;
                    v = __hadd2_rn(__hmul2_rn(asbf2(tres[b * ADAM_TRES_REPL + tres_lane]), s2), v);
                }
                const uint32_t vu = asu32(v);
                // the two elements of the pair through the optimizer chain (every intermediate rounded to bf16)
                const uint32_t w1 = (j < 2) ? in.q1.x : in.q1.y, w2 = (j < 2) ? in.q2.x : in.q2.y;
                const uint32_t a0 = (w1 >> (16 * (j & 1))) & 0xffu, a1 = (w1 >> (16 * (j & 1) + 8)) & 0xffu;
                const uint32_t b0 = (w2 >> (16 * (j & 1))) & 0xffu, b1 = (w2 >> (16 * (j & 1) + 8)) & 0xffu;
                const V m01 = LUT ? f2<V>(lut[a0], lut[a1]) : f2<V>(dec1(u2f(a0)), dec1(u2f(a1)));
                const V v01 = LUT ? f2<V>(lut[256 + b0], lut[256 + b1]) : f2<V>(dec2(u2f(b0)), dec2(u2f(b1)));
                const V gr = bf2f<V>(gw[j]);
                m[j] = packv(fma2(f2<V>(p.h.one_minus_beta1), gr, m01));
                const uint32_t vv = packv(fma2(f2<V>(p.h.one_minus_beta2), mul2(gr, gr), v01));
                const uint32_t t = pack2(sqrt_approx(lo2f(vv)), sqrt_approx(hi2f(vv)));
                d[j] = packv(add2(bf2f<V>(t), f2<V>(p.h.eps)));                                      // sqrt(v) + eps
                lat[j] = packv(fma2(f2<V>(-p.h.neg_step_size), neg_div_bf16(bf2f<V>(m[j]), bf2f<V>(d[j])), bf2f<V>(vu)));
                mn1 = min2(mn1, m[j]); mx1 = max2(mx1, m[j]);
                mn2 = min2(mn2, d[j]); mx2 = max2(mx2, d[j]);
            }
        }
        // block extrema of both states in two registers: (min m, min d) and (-max m, -max d)
        uint32_t lo, hi;
        {
            mn1 = min2(mn1, __byte_perm(mn1, 0u, 0x1032)); mx1 = max2(mx1, __byte_perm(mx1, 0u, 0x1032));
            mn2 = min2(mn2, __byte_perm(mn2, 0u, 0x1032)); mx2 = max2(mx2, __byte_perm(mx2, 0u, 0x1032));
            lo = __byte_perm(mn1, mn2, 0x5410); hi = __byte_perm(mx1, mx2, 0x5410) ^ 0x80008000u;
#pragma unroll
            for (int o = LUT ? 16 : 8; o > 0; o >>= 1) {
                lo = min2(lo, __shfl_xor_sync(0xffffffffu, lo, o)); hi = min2(hi, __shfl_xor_sync(0xffffffffu, hi, o));
            }
            if (LUT) {
                if (lane == 0) red[warp] = make_uint2(lo, hi);
                team_sync();                                  // also: every read of this tile's state tables is done
                const uint4* r4 = reinterpret_cast<const uint4*>(red);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint4 r = r4[i];
                    lo = min2(min2(lo, r.x), r.z); hi = min2(min2(hi, r.y), r.w);
                }
            }
        }
        if (active) {
            const float fmn1 = lo2f(lo), fmn2 = hi2f(lo), fmx1 = -lo2f(hi), fmx2 = -hi2f(hi);
            OptScale o1 = opt8_scale(fmx1, fmn1), o2 = opt8_scale(fmx2, fmn2);
            // requantize: Z = bf16(bf16(lat / s) + z), then one table byte per element
            const float sf = __uint_as_float(in.sb << 16);
            const float rs = __frcp_rn(sf);
            const __nv_bfloat162 z2 = asbf2(in.zb * 0x00010001u);
            uint32_t zbits[4], zmax = 0u;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                __nv_bfloat162 Zp = asbf2(packv(mul2(bf2f<V>(lat[j]), f2<V>(rs))));
                if (!W8) Zp = __hadd2_rn(Zp, z2);
                zbits[j] = asu32(Zp);
                __nv_bfloat162 az = __habs2(Zp);
                if (j) az = __hmax2_nan(asbf2(zmax), az);                                            // NaN-propagating max of the magnitudes
                zmax = asu32(az);
            }
            // |Z| beyond the table or not finite, an extreme scale, or extrema that are not finite (exponent field all ones)
            const uint32_t inf_lo = (lo & 0x7fff7fffu) + 0x00800080u, inf_hi = (hi & 0x7fff7fffu) + 0x00800080u;
            const bool bad = ((((zmax & 0x7fff7fffu) + AF::Z_LIMIT) | inf_lo | inf_hi) & 0x80008000u) != 0u || !fastdiv_ok_scale(sf);
            if (__builtin_expect(bad, 0)) {
                o1.s = __fadd_rn(__fdiv_rn(__fsub_rn(fmx1, fmn1), 255.0f), 1e-10f);      // (the fast division is for finite extrema)
                o2.s = __fadd_rn(__fdiv_rn(__fsub_rn(fmx2, fmn2), 255.0f), 1e-10f);
                const float4 q = LUT ? prm[parity] : make_float4(in.s1, in.t1, in.s2, in.t2);
                adam_word_generic<WBITS>(p, (int64_t)w, q.x, q.y, q.z, q.w, fmx1, o1.s, fmx2, o2.s);
            } else {
                *reinterpret_cast<uint2*>(p.st1 + (size_t)w * 8) = make_uint2(opt8_codes4<V>(m[0], m[1], fmx1, o1), opt8_codes4<V>(m[2], m[3], fmx1, o1));
                *reinterpret_cast<uint2*>(p.st2 + (size_t)w * 8) = make_uint2(opt8_codes4<V>(d[0], d[1], fmx2, o2), opt8_codes4<V>(d[2], d[3], fmx2, o2));
                uint32_t ev[4], od[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    ev[j] = W8 ? (uint32_t)enc8[zbits[j] & 0xffffu] : (uint32_t)encz[zbits[j] & 0xffffu];
                    od[j] = W8 ? (uint32_t)enc8[zbits[j] >> 16] : (uint32_t)encz[zbits[j] >> 16];
                }
                if (W8) {
                    // code in byte 0, nibble in byte 1; residual element k at bits 28 - 4k
                    const uint32_t p01 = __byte_perm(ev[0], od[0], 0x5140), p23 = __byte_perm(ev[1], od[1], 0x5140);   // (c0 c1 n0 n1)
                    const uint32_t p45 = __byte_perm(ev[2], od[2], 0x5140), p67 = __byte_perm(ev[3], od[3], 0x5140);
                    reinterpret_cast<uint2*>(p.rq.codes_out)[w] = make_uint2(__byte_perm(p01, p23, 0x5410), __byte_perm(p45, p67, 0x5410));
                    const uint32_t hi = __byte_perm(__byte_perm(ev[3], ev[2], 0x0051), __byte_perm(ev[1], ev[0], 0x0051), 0x5410);   // n6 n4 n2 n0
                    const uint32_t lo4 = __byte_perm(__byte_perm(od[3], od[2], 0x0051), __byte_perm(od[1], od[0], 0x0051), 0x5410);  // n7 n5 n3 n1
                    p.rq.words_out[w] = (int32_t)((hi << 4) | lo4);
                } else {
                    const uint32_t e_even = __byte_perm(__byte_perm(ev[0], ev[1], 0x4040), __byte_perm(ev[2], ev[3], 0x4040), 0x5410);
                    const uint32_t e_odd = __byte_perm(__byte_perm(od[0], od[1], 0x4040), __byte_perm(od[2], od[3], 0x4040), 0x5410);
                    reinterpret_cast<uint32_t*>(p.rq.codes_out)[w] = (e_even & 0xF0F0F0F0u) | ((e_odd >> 4) & 0x0F0F0F0Fu);
                    p.rq.words_out[w] = (int32_t)__byte_perm(((e_even << 4) & 0xF0F0F0F0u) | (e_odd & 0x0F0F0F0Fu), 0u, 0x0123);
                }
            }
            const uint32_t ob = w >> osh;
            const bool leader = LUT ? (tid == 0) : ((tid & 15) == 0);
            if (leader) { p.sc1[ob] = o1.s; p.tm1[ob] = fmx1; p.sc2[ob] = o2.s; p.tm2[ob] = fmx2; }
        }
        parity ^= 1;
    }
}

// What the fast variant's arithmetic relies on beside finite moments: eps hides a root that sqrt.approx flushes to zero (below
// 2^-63) and keeps denominators normal; a sane step size keeps updates from moments below 2^-117, whose division residual is not
// exact any more, far below the resolution of the codes.
static inline bool adam_fast_hyper_ok(const lq_adam_hyper& h) {
    return h.eps >= 4e-12f && h.eps <= 1.0f && h.neg_step_size >= -1e3f && h.neg_step_size <= 1e3f;
}

template <int WBITS>
static int launch_adam_fast(const AdamParams& p, int enc_slot, int opt_block, uint64_t row_magic, cudaStream_t st) {
    using AF = AdamFast<WBITS>;
    const int v = (p.rq.has_residual ? 2 : 0) + (opt_block == 2048 ? 1 : 0);
    auto* const kernel = v == 3 ? k_adam_fast<WBITS, true, true> : v == 2 ? k_adam_fast<WBITS, true, false>
                         : v == 1 ? k_adam_fast<WBITS, false, true> : k_adam_fast<WBITS, false, false>;
    static bool attr_done[64][4] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !attr_done[dev][v]) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, AF::SMEM);
        if (e != cudaSuccess) { set_cuda_error(e, "cudaFuncSetAttribute(k_adam_fast)"); return LQ_ECUDA; }
        attr_done[dev][v] = true;
    }
    const int64_t cap = (int64_t)sm_count() * AF::MIN_CTAS, want = (p.n_tiles + AF::TEAMS - 1) / AF::TEAMS;
    kernel<<<(int)(want < cap ? want : cap), AF::THREADS, AF::SMEM, st>>>(p, enc_slot, row_magic);
    return check_launch("k_adam_fast");
}

template <int WBITS, int CODEC, int DITHER>
static int launch_adam(const AdamParams& p, bool bf, cudaStream_t st) {
    const int64_t cap = (int64_t)sm_count() * 8;
    const int grid = (int)(p.n_tiles < cap ? p.n_tiles : cap);
    if (bf) k_adam_quant<WBITS, CODEC, DITHER, true><<<grid, 256, 0, st>>>(p);
    else k_adam_quant<WBITS, CODEC, DITHER, false><<<grid, 256, 0, st>>>(p);
    return check_launch("k_adam_quant");
}

// ---- the statistic behind the residual-curve refresh (utils/quant.py:1107-1111) ---------------------------------
// abs(exp_avg) / denom of the step ABOUT to be taken (the reference evaluates it after the moment update and before
// the requantize, whose curve level it may change), summed in fp32 over runs of 128 elements: 16 adjacent threads, fixed
// order.  Reads the gradient and both 8-bit states, writes only the sums.
template <bool BF>
__global__ void __launch_bounds__(256) k_adam_moment_stat(const AdamParams p, float* __restrict__ stat_out) {
    for (int64_t w = (int64_t)blockIdx.x * 256 + threadIdx.x; w < p.n_tiles * 256; w += (int64_t)gridDim.x * 256) {
        const bool active = w < p.rq.n_words;
        float t = 0.0f;
        if (active) {
            const int64_t e0 = w * 8, ob = e0 >> p.opt_shift;
            const float s1 = p.sc1[ob], t1 = p.tm1[ob], s2 = p.sc2[ob], t2 = p.tm2[ob];
            const uint2 q1 = *reinterpret_cast<const uint2*>(p.st1 + e0);
            const uint2 q2 = *reinterpret_cast<const uint2*>(p.st2 + e0);
            float gr[8];
            load8(p.grad, p.grad_dtype, e0, gr);
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const float c1 = u2f(((k < 4 ? q1.x : q1.y) >> (8 * (k & 3))) & 0xffu);
                const float c2 = u2f(((k < 4 ? q2.x : q2.y) >> (8 * (k & 3))) & 0xffu);
                float m = rb<BF>(__fsub_rn(t1, __fmul_rn(c1, s1)));
                const float r2 = __fsub_rn(t2, __fmul_rn(c2, s2));
                float d = rb<BF>(__fmul_rn(r2, r2));
                adam_moments<BF>(p.h, gr[k], m, d);
                t = __fadd_rn(t, rb<BF>(__fdiv_rn(fabsf(m), d)));
            }
        }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) t = __fadd_rn(t, __shfl_xor_sync(0xffffffffu, t, o));
        if (active && (threadIdx.x & 15) == 0) stat_out[w >> 4] = t;
    }
}

// ---- many small dense bf16 tensors ---------------------------------------------------------------
__global__ void __launch_bounds__(256) k_adam_dense_multi(const lq_dense_slot* __restrict__ table, const lq_adam_hyper h) {
    const lq_dense_slot t = table[blockIdx.y];
    __nv_bfloat16* pw = reinterpret_cast<__nv_bfloat16*>(t.param);
    const __nv_bfloat16* pg = reinterpret_cast<const __nv_bfloat16*>(t.grad);
    __nv_bfloat16* p1 = reinterpret_cast<__nv_bfloat16*>(t.state1);
    __nv_bfloat16* p2 = reinterpret_cast<__nv_bfloat16*>(t.state2);
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < t.numel; i += (int64_t)gridDim.x * blockDim.x) {
        float m = __bfloat162float(p1[i]);
        const float s2 = __bfloat162float(p2[i]);
        float d = rb<true>(__fmul_rn(s2, s2));                             // state2 * state2 (utils/quant.py:1092)
        adam_moments<true>(h, __bfloat162float(pg[i]), m, d);
        const float w = adam_apply<true>(h, __bfloat162float(pw[i]), m, d);
        p1[i] = __float2bfloat16_rn(m);
        p2[i] = __float2bfloat16_rn(d);
        pw[i] = __float2bfloat16_rn(w);
    }
}

// ---- 8-bit stochastic gradient accumulator: GradientQTensor (utils/quant.py:846-921) ----------------------------
// One CTA per weight row.  FIRST (set_value): scale = clamp(4 * absmax(row), 1e-5) / 127 in the gradient's dtype, then
// q = clamp(round_half_even(f / scale + noise), -128, 127).  Otherwise (add_): f <- q * scale + f first, scale kept.
// noise: explicit fp32 buffer, or the library's Philox stream (one block per 8 elements), rounded to the chain dtype
// like the reference's noise tensor.
template <bool BF, bool FIRST, int DITHER>
__global__ void __launch_bounds__(256) k_gradq(const void* __restrict__ f, int dtype, int cols, int8_t* __restrict__ q,
                                               void* __restrict__ scale, const float* __restrict__ noise, uint64_t seed,
                                               uint64_t stream_id) {
    __shared__ float red[8];
    const int64_t row = blockIdx.x;
    const int words = cols >> 3;
    float s;
    if (FIRST) {
        float am = 0.0f;
        for (int w = threadIdx.x; w < words; w += 256) {
            float v[8];
            load8(f, dtype, row * cols + (int64_t)w * 8, v);
#pragma unroll
            for (int k = 0; k < 8; ++k) am = fmaxf(am, fabsf(v[k]));
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, o));
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = am;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 8; ++i) am = fmaxf(am, red[i]);
        const float vmax = rb<BF>(__fmul_rn(am, 4.0f));
        s = rb<BF>(__fdiv_rn(fmaxf(vmax, rb<BF>(1e-5f)), 127.0f));
        if (threadIdx.x == 0) {
            if (dtype == LQ_BF16) reinterpret_cast<__nv_bfloat16*>(scale)[row] = __float2bfloat16_rn(s);
            else reinterpret_cast<float*>(scale)[row] = s;
        }
    } else {
        s = load1(scale, dtype, row);
    }
    for (int w = threadIdx.x; w < words; w += 256) {
        const int64_t e0 = row * cols + (int64_t)w * 8;
        float v[8], u[8];
        load8(f, dtype, e0, v);
        if (DITHER == LQ_DITHER_EXPLICIT) load8(noise, LQ_F32, e0, u);
        else philox_dither8(seed, stream_id, (uint64_t)(e0 >> 3), u);
        uint2 old = make_uint2(0u, 0u);
        if (!FIRST) old = *reinterpret_cast<const uint2*>(q + e0);
        uint32_t b[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            float x = v[k];
            if (!FIRST) {
                const uint32_t byte = ((k < 4 ? old.x : old.y) >> (8 * (k & 3))) & 0xffu;
                const float c = __fsub_rn(u2f(byte ^ 0x80u), 128.0f);                 // signed byte
                x = rb<BF>(__fadd_rn(rb<BF>(__fmul_rn(c, s)), x));                    // dequant() + fdata
            }
            float t = rb<BF>(__fadd_rn(rb<BF>(__fdiv_rn(x, s)), rb<BF>(u[k])));
            t = fminf(fmaxf(rne(t), -128.0f), 127.0f);
            b[k] = f2bits(t) & 0xffu;
        }
        *reinterpret_cast<uint2*>(q + e0) = make_uint2(b[0] | (b[1] << 8) | (b[2] << 16) | (b[3] << 24),
                                                      b[4] | (b[5] << 8) | (b[6] << 16) | (b[7] << 24));
    }
}
// The same for bf16 gradients and the Philox stream (words below 2^31), with packed arithmetic and the generator's word-independent part
// from the host.  The division by the row's scale is a product with its rounded reciprocal: gradient and scale have 8-bit significands,
// so their quotient is at least 2^-17 (relative) away from every bf16 rounding boundary and never on one (scales beyond 2^+-40: division).
// Clamped to whole numbers first, then rounded by the addition that leaves the code in the low byte.
// Bound by instruction issue (the Philox block is half of it).  2048 x 8192, first / later micro-batch: 35.6 / 41.3 -> 17.2 / 18.0 us (2.9 / 3.7 TB/s).
template <bool FIRST>
__global__ void __launch_bounds__(256) k_gradq_fast(const uint4* __restrict__ f, int words, uint2* __restrict__ q, __nv_bfloat16* __restrict__ scale,
                                                    const __grid_constant__ PhiloxConsts px) {
    using V = f32x2;
    __shared__ uint32_t red[8];
    const uint32_t row = blockIdx.x, w0 = row * (uint32_t)words;
    float s;
    if (FIRST) {
        uint32_t am = 0u;
        for (int w = threadIdx.x; w < words; w += 256) {
            const uint4 v = __ldg(f + w0 + w);
            am = max2(max2(am, max2(v.x & 0x7fff7fffu, v.y & 0x7fff7fffu)), max2(v.z & 0x7fff7fffu, v.w & 0x7fff7fffu));
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) am = max2(am, __shfl_xor_sync(0xffffffffu, am, o));
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = am;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 8; ++i) am = max2(am, red[i]);
        const float vmax = bf16r(__fmul_rn(fmaxf(lo2f(am), hi2f(am)), 4.0f));
        s = bf16r(__fdiv_rn(fmaxf(vmax, bf16r(1e-5f)), 127.0f));
        if (threadIdx.x == 0) scale[row] = __float2bfloat16_rn(s);
    } else {
        s = __bfloat162float(scale[row]);
    }
    const bool fast = fastdiv_ok_scale(s);
    const V rs = f2<V>(__frcp_rn(s));
    for (int w = threadIdx.x; w < words; w += 256) {
        const uint4 v = __ldg(f + w0 + w);
        uint32_t x[4] = {v.x, v.y, v.z, v.w}, c[4], t[4];
        philox4x32_10_word(w0 + (uint32_t)w, px, c);
        if (!FIRST) {
            const uint2 old = q[w0 + w];
#pragma unroll
            for (int j = 0; j < 4; ++j) {                                            // dequant() + fdata
                const uint32_t h2 = __byte_perm(((j < 2) ? old.x : old.y) ^ 0x80808080u, 0x64646464u, (j & 1) ? 0x4342 : 0x4140);   // fp16 1152 + code
                const float2 cf = __half22float2(__hsub2(*reinterpret_cast<const __half2*>(&h2), __floats2half2_rn(1152.0f, 1152.0f)));
                x[j] = asu32(__hadd2_rn(asbf2(pack2(__fmul_rn(cf.x, s), __fmul_rn(cf.y, s))), asbf2(x[j])));
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t qt = fast ? packv(mul2(bf2f<V>(x[j]), rs)) : pack2(__fdiv_rn(lo2f(x[j]), s), __fdiv_rn(hi2f(x[j]), s));
            // (2^23 + h) 2^-16 - 128.5 = h / 65536 - 0.5, the two halves of c[j]
            const V h = f2<V>(__uint_as_float(__byte_perm(c[j], 0x4B000000u, 0x7610)), __uint_as_float(__byte_perm(c[j], 0x4B000000u, 0x7632)));
            const uint32_t u = packv(fma2(h, f2<V>(1.0f / 65536.0f), f2<V>(-128.5f)));
            const __nv_bfloat162 sum = __hadd2_rn(asbf2(qt), asbf2(u));
            const uint32_t k = min2(max2(asu32(sum) & __heq2_mask(sum, sum), 0xC300C300u), 0x42FE42FEu);          // NaN: 0, as in the generic kernel; -128 .. 127
            const float2 b = of2(add2(bf2f<V>(k), f2<V>(MAGIC_RNE)));
            t[j] = __byte_perm(__float_as_uint(b.x), __float_as_uint(b.y), 0x0040);
        }
        q[w0 + w] = make_uint2(__byte_perm(t[0], t[1], 0x5410), __byte_perm(t[2], t[3], 0x5410));
    }
}
// get_value(): qdata.to(dtype) * scale
__global__ void __launch_bounds__(256) k_gradq_dequant(const int8_t* __restrict__ q, const void* __restrict__ scale, int dtype,
                                                       int cols, int64_t n_words, void* __restrict__ out) {
    for (int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < n_words; w += (int64_t)gridDim.x * blockDim.x) {
        const int64_t e0 = w * 8;
        const float s = load1(scale, dtype, e0 / cols);
        const uint2 pk = *reinterpret_cast<const uint2*>(q + e0);
        float v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const uint32_t byte = ((k < 4 ? pk.x : pk.y) >> (8 * (k & 3))) & 0xffu;
            v[k] = __fmul_rn(__fsub_rn(u2f(byte ^ 0x80u), 128.0f), s);                // store8 rounds to the dtype
        }
        store8(out, dtype, e0, v);
    }
}

}  // namespace lq

using namespace lq;

extern "C" {

int lq_adam_a16w4_step(int8_t* codes, int32_t* words, const void* grad, int grad_dtype, const void* scales,
                       const void* zeros, int qp_dtype, int64_t numel, int group, uint8_t* state1, float* scale1,
                       float* tmax1, uint8_t* state2, float* scale2, float* tmax2, int opt_block,
                       const lq_adam_hyper* hyper, const lq_requant_opts* opts, lq_stream_t stream) {
    if (numel == 0) return LQ_OK;
    AdamParams p{};
    int rc = fill_requant(p.rq, opts, numel, group);
    if (rc) return rc;
    if (!hyper || !codes || !words || !grad || !scales || !zeros || !state1 || !scale1 || !tmax1 || !state2 || !scale2 ||
        !tmax2 || !dtype_ok(grad_dtype) || !dtype_ok(qp_dtype) || !aligned(codes, 4) || !aligned(words, 4) ||
        !aligned(grad, 16) || !aligned(state1, 8) || !aligned(state2, 8))
        return LQ_EINVAL;
    if ((opt_block != 2048 && opt_block != 128) || numel % opt_block != 0) return LQ_EINVAL;
    // the chain dtype is the gradient's; mixed gradient / qparam dtypes promote differently op by op in torch
    if (grad_dtype != qp_dtype || opts->math_dtype != grad_dtype) return LQ_EUNSUPPORTED;
    if ((rc = ensure_device_for(codes)) != LQ_OK) return rc;
    p.rq.codes_in = codes; p.rq.words_in = words; p.rq.codes_out = codes; p.rq.words_out = words;
    p.rq.scales = scales; p.rq.zeros = zeros; p.rq.qp_dtype = qp_dtype;
    p.grad = grad; p.grad_dtype = grad_dtype;
    p.st1 = state1; p.sc1 = scale1; p.tm1 = tmax1; p.st2 = state2; p.sc2 = scale2; p.tm2 = tmax2;
    p.opt_shift = opt_block == 2048 ? 11 : 7;
    p.n_tiles = (p.rq.n_words + 255) / 256;
    p.h = *hyper;
    const bool bf = grad_dtype == LQ_BF16;
    cudaStream_t st = LQ_ST(stream);
    if (opts->codec == LQ_CODEC_THREEFOLD && opts->dither == LQ_DITHER_HASH) {
        if (bf && p.rq.group_shift >= 3 && p.rq.n_words < ((int64_t)1 << 31) && opts->mu_enc >= 0 && opts->mu_enc <= 3 &&
            opts->mu_dec >= 0 && opts->mu_dec <= 3 && adam_fast_hyper_ok(*hyper) && !getenv("LQ_REQUANT_GENERIC")) {
            int table = 0;
            rc = ensure_encz_table(opts->mu_enc, opts->v0, st, table);
            if (rc == LQ_OK) return launch_adam_fast<4>(p, table, opt_block, 0, st);
            if (rc != LQ_EUNSUPPORTED) return rc;
        }
        return launch_adam<4, LQ_CODEC_THREEFOLD, LQ_DITHER_HASH>(p, bf, st);
    }
    if (opts->codec == LQ_CODEC_THREEFOLD && opts->dither == LQ_DITHER_PHILOX) return launch_adam<4, LQ_CODEC_THREEFOLD, LQ_DITHER_PHILOX>(p, bf, st);
    if (opts->codec == LQ_CODEC_UNIFORM16 && opts->dither == LQ_DITHER_PHILOX) return launch_adam<4, LQ_CODEC_UNIFORM16, LQ_DITHER_PHILOX>(p, bf, st);
    return LQ_EUNSUPPORTED;
}

int lq_adam_a8w8_step(int8_t* codes, int32_t* words, const void* grad, int grad_dtype, const void* qscales, int qp_dtype,
                      int64_t rows, int64_t cols, uint8_t* state1, float* scale1, float* tmax1, uint8_t* state2, float* scale2,
                      float* tmax2, int opt_block, const lq_adam_hyper* hyper, const lq_requant_opts* opts, lq_stream_t stream) {
    if (rows == 0 || cols == 0) return LQ_OK;
    if (rows < 0 || cols < 0) return LQ_EINVAL;
    AdamParams p{};
    const int64_t numel = rows * cols;
    int rc = fill_requant(p.rq, opts, numel, cols);          // one scale per weight row: the "group" is the row
    if (rc) return rc;
    if (!hyper || !codes || !words || !grad || !qscales || !state1 || !scale1 || !tmax1 || !state2 || !scale2 || !tmax2 ||
        !dtype_ok(grad_dtype) || !dtype_ok(qp_dtype) || !aligned(codes, 8) || !aligned(words, 4) || !aligned(grad, 16) ||
        !aligned(state1, 8) || !aligned(state2, 8))
        return LQ_EINVAL;
    if ((opt_block != 2048 && opt_block != 128) || numel % opt_block != 0) return LQ_EINVAL;
    if (grad_dtype != qp_dtype || opts->math_dtype != grad_dtype) return LQ_EUNSUPPORTED;
    if ((rc = ensure_device_for(codes)) != LQ_OK) return rc;
    p.rq.codes_in = codes; p.rq.words_in = words; p.rq.codes_out = codes; p.rq.words_out = words;
    p.rq.scales = qscales; p.rq.zeros = nullptr; p.rq.qp_dtype = qp_dtype;
    p.grad = grad; p.grad_dtype = grad_dtype;
    p.st1 = state1; p.sc1 = scale1; p.tm1 = tmax1; p.st2 = state2; p.sc2 = scale2; p.tm2 = tmax2;
    p.opt_shift = opt_block == 2048 ? 11 : 7;
    p.n_tiles = (p.rq.n_words + 255) / 256;
    p.h = *hyper;
    const bool bf = grad_dtype == LQ_BF16;
    cudaStream_t st = LQ_ST(stream);
    if (opts->codec == LQ_CODEC_THREEFOLD && opts->dither == LQ_DITHER_HASH) {
        const uint64_t wpr = (uint64_t)(cols / 8);               // words per weight row; the row of a word by multiply-high, exact below 2^24 words
        if (bf && wpr > 1 && wpr < (1u << 24) && p.rq.n_words < ((int64_t)1 << 31) && opts->mu_enc >= 0 && opts->mu_enc <= 3 &&
            opts->mu_dec >= 0 && opts->mu_dec <= 3 && adam_fast_hyper_ok(*hyper) && !getenv("LQ_REQUANT_GENERIC")) {
            int table = 0;
            rc = ensure_enc8_table(opts->mu_enc, opts->v0, st, table);
            if (rc == LQ_OK) return launch_adam_fast<8>(p, table, opt_block, ~(uint64_t)0 / wpr + 1, st);
            if (rc != LQ_EUNSUPPORTED) return rc;
        }
        return launch_adam<8, LQ_CODEC_THREEFOLD, LQ_DITHER_HASH>(p, bf, st);
    }
    if (opts->codec == LQ_CODEC_THREEFOLD && opts->dither == LQ_DITHER_PHILOX) return launch_adam<8, LQ_CODEC_THREEFOLD, LQ_DITHER_PHILOX>(p, bf, st);
    return LQ_EUNSUPPORTED;
}

int lq_adam_moment_stat(const void* grad, int grad_dtype, int64_t numel, const uint8_t* state1, const float* scale1,
                        const float* tmax1, const uint8_t* state2, const float* scale2, const float* tmax2, int opt_block,
                        const lq_adam_hyper* hyper, float* stat_out, lq_stream_t stream) {
    if (numel == 0) return LQ_OK;
    if (!grad || !state1 || !scale1 || !tmax1 || !state2 || !scale2 || !tmax2 || !hyper || !stat_out || !dtype_ok(grad_dtype) ||
        numel < 0 || (numel % 128) != 0 || !aligned(grad, 16) || !aligned(state1, 8) || !aligned(state2, 8))
        return LQ_EINVAL;
    if ((opt_block != 2048 && opt_block != 128) || numel % opt_block != 0) return LQ_EINVAL;
    int rc = ensure_device_for(grad);
    if (rc != LQ_OK) return rc;
    AdamParams p{};
    p.rq.n_words = numel / 8;
    p.grad = grad; p.grad_dtype = grad_dtype;
    p.st1 = const_cast<uint8_t*>(state1); p.sc1 = const_cast<float*>(scale1); p.tm1 = const_cast<float*>(tmax1);
    p.st2 = const_cast<uint8_t*>(state2); p.sc2 = const_cast<float*>(scale2); p.tm2 = const_cast<float*>(tmax2);
    p.opt_shift = opt_block == 2048 ? 11 : 7;
    p.n_tiles = (p.rq.n_words + 255) / 256;
    p.h = *hyper;
    const int grid = grid_for(p.rq.n_words, 256, 8);
    if (grad_dtype == LQ_BF16) k_adam_moment_stat<true><<<grid, 256, 0, LQ_ST(stream)>>>(p, stat_out);
    else k_adam_moment_stat<false><<<grid, 256, 0, LQ_ST(stream)>>>(p, stat_out);
    return check_launch("k_adam_moment_stat");
}

int lq_gradq_accumulate(const void* fdata, int dtype, int64_t rows, int64_t cols, int8_t* qdata, void* scale, int first,
                        const lq_requant_opts* opts, lq_stream_t stream) {
    if (rows == 0 || cols == 0) return LQ_OK;
    if (!fdata || !qdata || !scale || !opts || !dtype_ok(dtype) || rows < 0 || cols < 0 || (cols % 8) != 0 || cols >= (1ll << 31) ||
        rows >= (1ll << 31) || !aligned(fdata, 16) || !aligned(qdata, 8))
        return LQ_EINVAL;
    if (opts->dither == LQ_DITHER_EXPLICIT && (!opts->dither_buf || !aligned(opts->dither_buf, 16))) return LQ_EINVAL;
    if (opts->dither != LQ_DITHER_EXPLICIT && opts->dither != LQ_DITHER_PHILOX) return LQ_EUNSUPPORTED;
    int rc = ensure_device_for(fdata);
    if (rc != LQ_OK) return rc;
    const bool bf = dtype == LQ_BF16, ex = opts->dither == LQ_DITHER_EXPLICIT;
    cudaStream_t st = LQ_ST(stream);
    if (bf && !ex && rows * (cols / 8) < (1ll << 31)) {
        const PhiloxConsts px = philox_consts(opts->seed, opts->stream_id);
        const uint4* f = reinterpret_cast<const uint4*>(fdata);
        uint2* qd = reinterpret_cast<uint2*>(qdata);
        __nv_bfloat16* sc = reinterpret_cast<__nv_bfloat16*>(scale);
        if (first) k_gradq_fast<true><<<(unsigned)rows, 256, 0, st>>>(f, (int)(cols / 8), qd, sc, px);
        else k_gradq_fast<false><<<(unsigned)rows, 256, 0, st>>>(f, (int)(cols / 8), qd, sc, px);
        return check_launch("k_gradq_fast");
    }
#define LQ_GRADQ(BFv, FIRSTv, DITHv) k_gradq<BFv, FIRSTv, DITHv><<<(unsigned)rows, 256, 0, st>>>(fdata, dtype, (int)cols, qdata, scale, opts->dither_buf, opts->seed, opts->stream_id)
    if (bf) { if (first) { if (ex) LQ_GRADQ(true, true, LQ_DITHER_EXPLICIT); else LQ_GRADQ(true, true, LQ_DITHER_PHILOX); }
              else { if (ex) LQ_GRADQ(true, false, LQ_DITHER_EXPLICIT); else LQ_GRADQ(true, false, LQ_DITHER_PHILOX); } }
    else { if (first) { if (ex) LQ_GRADQ(false, true, LQ_DITHER_EXPLICIT); else LQ_GRADQ(false, true, LQ_DITHER_PHILOX); }
           else { if (ex) LQ_GRADQ(false, false, LQ_DITHER_EXPLICIT); else LQ_GRADQ(false, false, LQ_DITHER_PHILOX); } }
#undef LQ_GRADQ
    return check_launch("k_gradq");
}

int lq_gradq_dequant(const int8_t* qdata, const void* scale, int dtype, int64_t rows, int64_t cols, void* out, lq_stream_t stream) {
    if (rows == 0 || cols == 0) return LQ_OK;
    if (!qdata || !scale || !out || !dtype_ok(dtype) || rows < 0 || cols < 0 || (cols % 8) != 0 || cols >= (1ll << 31) ||
        !aligned(qdata, 8) || !aligned(out, 16))
        return LQ_EINVAL;
    int rc = ensure_device_for(qdata);
    if (rc != LQ_OK) return rc;
    const int64_t n_words = rows * cols / 8;
    k_gradq_dequant<<<grid_for(n_words, 256, 8), 256, 0, LQ_ST(stream)>>>(qdata, scale, dtype, (int)cols, n_words, out);
    return check_launch("k_gradq_dequant");
}

int lq_adam_dense_multi(const lq_dense_slot* table, int n_tensors, int64_t max_numel, const lq_adam_hyper* hyper,
                        lq_stream_t stream) {
    if (n_tensors == 0 || max_numel == 0) return LQ_OK;
    if (!table || !hyper || n_tensors < 0 || n_tensors > 65535 || max_numel < 0) return LQ_EINVAL;
    int rc = ensure_device_for(table);
    if (rc != LQ_OK) return rc;
    int64_t bx = (max_numel + 255) / 256;
    if (bx > 64) bx = 64;
    dim3 grid((unsigned)bx, (unsigned)n_tensors);
    k_adam_dense_multi<<<grid, 256, 0, LQ_ST(stream)>>>(table, *hyper);
    return check_launch("k_adam_dense_multi");
}

}  // extern "C"
