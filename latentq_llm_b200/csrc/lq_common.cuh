// Shared device/host helpers for liblatentq (sm_100a only).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "latentq.h"

#if defined(__CUDA_ARCH__) && (__CUDA_ARCH__ < 1000)
#error "liblatentq targets sm_100a only"
#endif

namespace lq {

// ---- host-side error plumbing ------------------------------------------------
void set_cuda_error(cudaError_t e, const char* where);
int check_launch(const char* where);  // cudaGetLastError -> LQ_OK / LQ_ECUDA
int sm_count();                       // cached per current device
// Makes the device that owns `device_ptr` current on the calling thread if the thread has no CUDA context yet
// (worker threads such as an autograd engine thread start without one; launching from them would otherwise
// target device 0, and tensor-map encoding fails outright).  No-op when a context is already current.
int ensure_device_for(const void* device_ptr);

// ---- programmatic dependent launch (decode chain) -------------------------------------------------
// A decode step is a chain of short launches in which every kernel consumes its predecessor's output.  Inside such a
// chain (lq_decode_chain(1)) kernels are launched with programmatic stream serialization: a kernel signals
// launch_dependents early, so that its successor's launch latency (and, for the GEMMs, the first round of weight loads)
// overlaps its own run, and every kernel reads what a predecessor may have written only after pdl_wait(), which returns
// once the predecessor grid has completed and its writes are visible.  Outside a chain the attribute is off and both
// instructions are no-ops: a caller whose previous kernel wrote the WEIGHTS (an optimizer step followed by a forward)
// must not have those read early.
bool decode_chain_enabled();
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
template <typename... KArgs, typename... Args>
static inline void launch_pdl(void (*kern)(KArgs...), dim3 grid, unsigned block, size_t smem, cudaStream_t st, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid; cfg.blockDim = dim3(block); cfg.dynamicSmemBytes = smem; cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = decode_chain_enabled() ? 1 : 0;
    cfg.attrs = attr; cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kern, KArgs(args)...);
}

// ---- numeric helpers ------------------------------------------------------------
__device__ __forceinline__ float bf16r(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }
template <bool BF> __device__ __forceinline__ float rnd(float x) { return BF ? bf16r(x) : x; }
__device__ __forceinline__ float bf16_bits_to_f32(uint32_t h) { return __uint_as_float(h << 16); }
__device__ __forceinline__ uint32_t f32_to_bf16_bits(float x) {
    return (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(x));
}

// three_fold_curve_4bit (utils/quant.py:708-716) as the constants the reference launchers derive
// (utils/cuda_src/multi_random_quant_kernel.cu:345-351, 384-389).
struct Curve {
    float c1, c2, c3, ic1, ic2, ic3, b1, b2, t1, t2;
};
inline Curve make_curve(int k1, float b1, int k2, float b2, int k3) {
    Curve c;
    c.c1 = (float)k1 / b1;
    c.c2 = (float)k2 / (b2 - b1);
    c.c3 = (float)((double)k3 / (0.5 - (double)b2));
    c.ic1 = b1 / (float)k1;
    c.ic2 = (b2 - b1) / (float)k2;
    c.ic3 = (float)((0.5 - (double)b2) / (double)k3);
    c.b1 = b1; c.b2 = b2; c.t1 = (float)k1; c.t2 = (float)(k1 + k2);
    return c;
}
inline Curve curve_for_level(int mu) {
    switch (mu) {
        case 3: return make_curve(2, 0.4330623539159437f, 2, 0.46875f, 4);
        case 2: return make_curve(2, 0.37272211741724515f, 2, 0.4375f, 4);
        case 1: return make_curve(2, 0.2666300266320331f, 2, 0.375f, 4);
        default: return make_curve(2, 0.125f, 2, 0.25f, 4);
    }
}

// |x|*499 + v0, minus its round-half-away integer part (.cu:49-51); `a*b+c` is an FMA under nvcc defaults.
__device__ __forceinline__ float hash_dither(float x, float v0) {
    float v = __fmaf_rn(fabsf(x), 499.0f, v0);
    return __fsub_rn(v, roundf(v));
}
// 3-fold encode of one residual (.cu:52-63). Returns the nibble, sets carry.
__device__ __forceinline__ uint32_t res3_encode(float x, float v, const Curve& c, float& carry) {
    float S = fabsf(x), q;
    if (S < c.b1) {
        q = roundf(__fmaf_rn(x, c.c1, v));
    } else if (S < c.b2) {
        float r = __fadd_rn(roundf(__fmaf_rn(__fsub_rn(S, c.b1), c.c2, v)), c.t1);
        q = (x < 0.0f) ? -r : r;
    } else {
        float r = __fadd_rn(roundf(__fmaf_rn(__fsub_rn(S, c.b2), c.c3, v)), c.t2);
        q = (x < 0.0f) ? -r : r;
    }
    if (q > 7.5f) { carry = 1.0f; return 1u; }
    carry = 0.0f;
    float t = q + 8.0f;
    return (t <= 0.0f) ? 0u : (uint32_t)t;
}
// 3-fold decode of one nibble (.cu:160-169).
__device__ __forceinline__ float res3_decode(uint32_t nib, const Curve& c) {
    float s = (float)((int)nib - 8);
    if (s < -c.t2) return __fmaf_rn(s + c.t2, c.ic3, -c.b2);
    if (s < -c.t1) return __fmaf_rn(s + c.t1, c.ic2, -c.b1);
    if (s <= c.t1) return __fmul_rn(s, c.ic1);
    if (s <= c.t2) return __fmaf_rn(s - c.t1, c.ic2, c.b1);
    return __fmaf_rn(s - c.t2, c.ic3, c.b2);
}

// Philox4x32-10 (Salmon et al., SC'11), same constants as cuRAND.
__device__ __forceinline__ void philox4x32_10(uint32_t (&c)[4], uint32_t k0, uint32_t k1) {
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        const uint64_t p0 = (uint64_t)0xD2511F53u * c[0], p1 = (uint64_t)0xCD9E8D57u * c[2];   // one wide multiply each
        const uint32_t h0 = (uint32_t)(p0 >> 32), l0 = (uint32_t)p0, h1 = (uint32_t)(p1 >> 32), l1 = (uint32_t)p1;
        uint32_t n0 = h1 ^ c[1] ^ k0, n2 = h0 ^ c[3] ^ k1;
        c[0] = n0; c[1] = l1; c[2] = n2; c[3] = l0;
        k0 += 0x9E3779B9u; k1 += 0xBB67AE85u;
    }
}
// The same generator for counters (word, 0, stream) with word < 2^32: what does not depend on the word - the round keys, one of
// the two products of the first two rounds and the words they leave - is computed once on the host and read as kernel constants.
// 18 instead of 20 wide multiplies, 19 logic instructions, no key additions.  Requantize of 134 M weights, which instruction issue
// bounds: 166 -> 152 us (3.57 TB/s) together with the conditional shift of its selection.
struct PhiloxConsts { uint32_t x1, y0, y2, l0; uint32_t k0[8], k1[8]; };
inline PhiloxConsts philox_consts(uint64_t seed, uint64_t stream_id) {
    const uint32_t M0 = 0xD2511F53u, M1 = 0xCD9E8D57u, W0 = 0x9E3779B9u, W1 = 0xBB67AE85u;
    const uint32_t s0 = (uint32_t)seed, s1 = (uint32_t)(seed >> 32), c2 = (uint32_t)stream_id, c3 = (uint32_t)(stream_id >> 32);
    const uint64_t p1 = (uint64_t)M1 * c2;                                        // round 1: the product of the stream word
    const uint64_t p0 = (uint64_t)M0 * ((uint32_t)(p1 >> 32) ^ s0);               // round 2: the product of what it leaves in c[0]
    PhiloxConsts c;
    c.x1 = c3 ^ s1;
    c.y0 = (uint32_t)p1 ^ (s0 + W0);
    c.y2 = (uint32_t)(p0 >> 32) ^ (s1 + W1);
    c.l0 = (uint32_t)p0;
    for (uint32_t r = 0; r < 8; ++r) { c.k0[r] = s0 + (r + 2) * W0; c.k1[r] = s1 + (r + 2) * W1; }
    return c;
}
__device__ __forceinline__ void philox4x32_10_word(uint32_t word, const PhiloxConsts& k, uint32_t (&c)[4]) {
    const uint64_t p = (uint64_t)0xD2511F53u * word;
    const uint64_t q = (uint64_t)0xCD9E8D57u * ((uint32_t)(p >> 32) ^ k.x1);
    c[0] = (uint32_t)(q >> 32) ^ k.y0; c[1] = (uint32_t)q; c[2] = (uint32_t)p ^ k.y2; c[3] = k.l0;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const uint64_t p0 = (uint64_t)0xD2511F53u * c[0], p1 = (uint64_t)0xCD9E8D57u * c[2];
        const uint32_t n0 = (uint32_t)(p1 >> 32) ^ c[1] ^ k.k0[r], n2 = (uint32_t)(p0 >> 32) ^ c[3] ^ k.k1[r];
        c[0] = n0; c[1] = (uint32_t)p1; c[2] = n2; c[3] = (uint32_t)p0;
    }
}
// Dither of the 8 elements of residual word `word`: 16 random bits each, u = h/65536 - 0.5 (exact).
__device__ __forceinline__ void philox_dither8(uint64_t seed, uint64_t stream_id, uint64_t word, float (&u)[8]) {
    uint32_t c[4] = {(uint32_t)word, (uint32_t)(word >> 32), (uint32_t)stream_id, (uint32_t)(stream_id >> 32)};
    philox4x32_10(c, (uint32_t)seed, (uint32_t)(seed >> 32));
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        uint32_t h = (k & 1) ? (c[k >> 1] >> 16) : (c[k >> 1] & 0xffffu);
        // (2^23 + h) * 2^-16 - 128.5 == h/65536 - 0.5 with no rounding
        u[k] = __fmaf_rn(__uint_as_float(0x4B000000u | h), 1.0f / 65536.0f, -128.5f);
    }
}

// Correctly rounded quotients by a divisor that several elements share.  Method: Markstein's theorem (P. Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34(1), 1990): with y = RN(1/s) and q within one unit
// in the last place of a/s, the remainder a - q s is exact in one FMA and RN(q + y (a - q s)) = RN(a/s).  The first quotient q comes from a
// reciprocal in two terms, y + yl = (1/s)(1 + e) with |e| < 2^-46: q = RN(a y + RN(a yl)) is off by half a unit (its rounding) and less than
// 2^-20 units more.  Everything stays normal, and the remainder exact, for divisors and dividends in the ranges tested below;
// outside them __fdiv_rn divides.
__device__ __forceinline__ bool fastdiv_ok_scale(float s) {
    float a = fabsf(s);
    return a >= 9.094947e-13f && a <= 1.0995116e12f;  // 2^-40 .. 2^40
}
struct DivBy { float s, y, yl; bool ok; };
__device__ __forceinline__ DivBy div_by(float s) {
    DivBy d;
    d.s = s; d.y = __frcp_rn(s); d.ok = fastdiv_ok_scale(s);
    d.yl = __fmul_rn(__fmaf_rn(-s, d.y, 1.0f), d.y);
    return d;
}
__device__ __forceinline__ float markstein_div(float a, const DivBy& d) {
    const float q = __fmaf_rn(a, d.y, __fmul_rn(a, d.yl));
    return __fmaf_rn(__fmaf_rn(-q, d.s, a), d.y, q);
}
__device__ __forceinline__ float div_rn(float a, const DivBy& d) {
    const float m = fabsf(a);
    if (d.ok && (m == 0.0f || (m >= 8.6736174e-19f && m <= 1.1529215e18f))) return markstein_div(a, d);  // 2^-60 .. 2^60
    return __fdiv_rn(a, d.s);
}

}  // namespace lq
