// SiLU(gate) * up of the MLP (flh/quantized_model/modeling_llama.py:522-526: act_fn(gate_proj(x)) * up_proj(x)), defined
// so that the CPU restatement gives the same bits: every step is one IEEE binary32 operation in a fixed order.
//   e      = exp32(-g)                    g, u: the two 16-bit inputs widened to binary32
//   s      = round16(g / (1 + e))         (torch rounds silu's result to the 16-bit type too)
//   result = round16(s * u)               (the product of two 16-bit values is exact in binary32)
//   exp32(t), t clamped to [-87, 88]:  n = rint(t * log2(e));  r = t - n ln2 (two fma, ln2 split in two);
//   y = 1 + r + r^2 P(r) with the degree-5 polynomial of the Cephes expf (Horner, fma);  exp32 = y * 2^n.
#pragma once
#include "common.cuh"

namespace flh {

__device__ __forceinline__ float exp32(float t) {
    t = fminf(fmaxf(t, -87.0f), 88.0f);
    const float n = rintf(__fmul_rn(t, 1.44269504088896341f));
    float r = __fmaf_rn(n, -0.693359375f, t);
    r = __fmaf_rn(n, 2.12194440e-4f, r);
    const float z = __fmul_rn(r, r);
    float y = 1.9875691500e-4f;
    y = __fmaf_rn(y, r, 1.3981999507e-3f);
    y = __fmaf_rn(y, r, 8.3334519073e-3f);
    y = __fmaf_rn(y, r, 4.1665795894e-2f);
    y = __fmaf_rn(y, r, 1.6666665459e-1f);
    y = __fmaf_rn(y, r, 5.0000001201e-1f);
    y = __fmaf_rn(y, z, r);
    y = __fadd_rn(y, 1.0f);
    return __fmul_rn(y, __int_as_float(((int)n + 127) << 23));
}

// The same values for two gates at once in packed binary32, for finite gates of magnitude 2^-90 and up and, in bfloat16, above
// -80 (silu_mul_8 looks; float16 has no smaller ones, and its quotients below -80 round to -0 either way).  There no step of exp32
// rounds to a subnormal or overflows:
//   * rint by adding 1.5 * 2^23, whose low bits then are n for the exponent;
//   * the quotient by Newton-Raphson on a reciprocal estimate and a final fused residual step (Markstein, IBM J. Res. Dev. 34,
//     1990): rounded like the division it replaces.  s is a function of one 16-bit value, and the test compares every one.
// Half the issue slots of the scalar form: the kernel was bound by issue (0.54 of the copy bandwidth), not by memory.
__device__ __forceinline__ uint64_t dup2(float v) { return pack2(v, v); }
__device__ __forceinline__ float rcp_estimate(float d) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    return r;
}
__device__ __forceinline__ uint64_t silu2(uint64_t g) {
    float g0, g1;
    unpack2(g, g0, g1);
    const uint64_t t = pack2(fminf(fmaxf(-g0, -87.0f), 80.0f), fminf(fmaxf(-g1, -87.0f), 80.0f));
    const uint64_t nb = add2(mul2(t, dup2(1.44269504088896341f)), dup2(12582912.0f));
    const uint64_t n = add2(nb, dup2(-12582912.0f));
    uint64_t r = fma2(n, dup2(-0.693359375f), t);
    r = fma2(n, dup2(2.12194440e-4f), r);
    const uint64_t z = mul2(r, r);
    uint64_t y = fma2(dup2(1.9875691500e-4f), r, dup2(1.3981999507e-3f));
    y = fma2(y, r, dup2(8.3334519073e-3f));
    y = fma2(y, r, dup2(4.1665795894e-2f));
    y = fma2(y, r, dup2(1.6666665459e-1f));
    y = fma2(y, r, dup2(5.0000001201e-1f));
    y = fma2(y, z, r);
    y = add2(y, dup2(1.0f));
    // y * 2^n: n goes straight into the exponent (the bits above n of nb leave the word)
    const uint32_t e0 = (uint32_t)y + ((uint32_t)nb << 23), e1 = (uint32_t)(y >> 32) + ((uint32_t)(nb >> 32) << 23);
    const uint64_t d = add2(((uint64_t)e1 << 32) | e0, dup2(1.0f));
    float d0, d1;
    unpack2(d, d0, d1);
    uint64_t q = pack2(rcp_estimate(d0), rcp_estimate(d1));
    const uint64_t nd = mul2(d, dup2(-1.0f));
    q = fma2(q, fma2(nd, q, dup2(1.0f)), q);                // reciprocal of d
    const uint64_t a = mul2(g, q);
    return fma2(fma2(nd, a, g), q, a);
}
// two neighbouring elements at once: g2, u2 hold two 16-bit values each (low half = the lower index)
template <bool BF16>
__device__ __forceinline__ uint32_t silu_mul_pair(uint32_t g2, uint32_t u2) {
    float g0, g1, u0, u1;
    if (BF16) {
        g0 = __uint_as_float(g2 << 16); g1 = __uint_as_float(g2 & 0xffff0000u);
        u0 = __uint_as_float(u2 << 16); u1 = __uint_as_float(u2 & 0xffff0000u);
    } else {
        const float2 gf = __half22float2(*reinterpret_cast<const __half2 *>(&g2));
        const float2 uf = __half22float2(*reinterpret_cast<const __half2 *>(&u2));
        g0 = gf.x; g1 = gf.y; u0 = uf.x; u1 = uf.y;
    }
    const float s0 = __fdiv_rn(g0, __fadd_rn(1.0f, exp32(-g0)));
    const float s1 = __fdiv_rn(g1, __fadd_rn(1.0f, exp32(-g1)));
    if (BF16) {
        const float a0 = __bfloat162float(__float2bfloat16_rn(s0)), a1 = __bfloat162float(__float2bfloat16_rn(s1));
        const __nv_bfloat162 o = __floats2bfloat162_rn(__fmul_rn(a0, u0), __fmul_rn(a1, u1));
        return *reinterpret_cast<const uint32_t *>(&o);
    }
    const float a0 = __half2float(__float2half_rn(s0)), a1 = __half2float(__float2half_rn(s1));
    const __half2 o = __floats2half2_rn(__fmul_rn(a0, u0), __fmul_rn(a1, u1));
    return *reinterpret_cast<const uint32_t *>(&o);
}

template <bool BF16>
__device__ __noinline__ uint4 silu_mul_8_any(uint4 g, uint4 u) {
    return make_uint4(silu_mul_pair<BF16>(g.x, u.x), silu_mul_pair<BF16>(g.y, u.y), silu_mul_pair<BF16>(g.z, u.z),
                      silu_mul_pair<BF16>(g.w, u.w));
}

// Eight elements: one look at all gates, then the packed form for every pair or (a zero, an infinity, a bfloat16 far below zero
// among them) the scalar one out of line: a branch and both forms per pair overflowed the instruction cache.
template <bool BF16>
__device__ __forceinline__ uint4 silu_mul_8(const uint4 g, const uint4 u) {
    const uint32_t gw[4] = {g.x, g.y, g.z, g.w}, uw[4] = {u.x, u.y, u.z, u.w};
    float gf[8];
    float lo = 3.0e38f, hi = 0.0f, least = 0.0f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (BF16) {
            gf[2 * k] = __uint_as_float(gw[k] << 16); gf[2 * k + 1] = __uint_as_float(gw[k] & 0xffff0000u);
            least = fminf(least, fminf(gf[2 * k], gf[2 * k + 1]));
        } else {
            const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&gw[k]));
            gf[2 * k] = f.x; gf[2 * k + 1] = f.y;
        }
        lo = fminf(lo, fminf(fabsf(gf[2 * k]), fabsf(gf[2 * k + 1])));
        hi = fmaxf(hi, fmaxf(fabsf(gf[2 * k]), fabsf(gf[2 * k + 1])));
    }
    if (!(lo > (BF16 ? 8.0e-28f : 0.0f) && hi < 3.0e38f && (!BF16 || least > -80.0f))) return silu_mul_8_any<BF16>(g, u);
    uint32_t o[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        float s0, s1;
        unpack2(silu2(pack2(gf[2 * k], gf[2 * k + 1])), s0, s1);
        if (BF16) {
            const float a0 = __bfloat162float(__float2bfloat16_rn(s0)), a1 = __bfloat162float(__float2bfloat16_rn(s1));
            const __nv_bfloat162 h = __floats2bfloat162_rn(__fmul_rn(a0, __uint_as_float(uw[k] << 16)), __fmul_rn(a1, __uint_as_float(uw[k] & 0xffff0000u)));
            o[k] = *reinterpret_cast<const uint32_t *>(&h);
        } else {
            // the product of two float16 values is exact in binary32: one rounding, as float16 multiplies
            const __half2 h = __hmul2(__floats2half2_rn(s0, s1), *reinterpret_cast<const __half2 *>(&uw[k]));
            o[k] = *reinterpret_cast<const uint32_t *>(&h);
        }
    }
    return make_uint4(o[0], o[1], o[2], o[3]);
}

}  // namespace flh
