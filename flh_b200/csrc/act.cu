// Element-wise pieces of the decoder wiring that sit either side of the quantised linears
// (flh/quantized_model/modeling_llama.py:389-470, 522-526):
//   * silu_mul_kernel     SiLU(gate) * up from the merged gate/up GEMM output into a 16-bit matrix (the form the fused
//                         quantiser entry falls back to for widths its tensor-core kernel does not take);
//   * rope_kv_kernel      rotary embedding of q and k (half-split convention) straight from the merged QKV GEMM output:
//                         q goes to a [B, heads, S, D] tensor for the attention call, k and v are written into the KV cache
//                         at the step's position — one pass instead of split / rope / transpose / two cache copies.
#include "act_common.cuh"

namespace flh {
namespace {

// A thread keeps its 16-byte column and walks down the rows, two at a time: four loads in flight and no division per piece.
constexpr int kSiluThreads = 128;
template <bool BF16>
__global__ void __launch_bounds__(kSiluThreads) silu_mul_kernel(const uint8_t *__restrict__ gu, long M, long F, long ld_bytes, uint8_t *__restrict__ out) {
    const long c = (long)blockIdx.x * kSiluThreads + threadIdx.x;
    pdl_wait();
    pdl_trigger();
    if (c >= F / 8) return;
    const long step = gridDim.y;
    for (long m = blockIdx.y; m < M; m += 2 * step) {
        const bool two = m + step < M;
        const uint8_t *r0 = gu + m * ld_bytes + c * 16, *r1 = two ? r0 + step * ld_bytes : r0;
        const uint4 g0 = ldg_nc_v4(r0), u0 = ldg_nc_v4(r0 + F * 2), g1 = ldg_nc_v4(r1), u1 = ldg_nc_v4(r1 + F * 2);
        *reinterpret_cast<uint4 *>(out + (m * F + c * 8) * 2) = silu_mul_8<BF16>(g0, u0);
        if (two) *reinterpret_cast<uint4 *>(out + ((m + step) * F + c * 8) * 2) = silu_mul_8<BF16>(g1, u1);
    }
}

// out = x * x in binary32 of 16-bit values: what the final norm averages.  As tensor operations (a copy to binary32, then its
// square) 8,192 x 8,192 values took 280 us and 940 MB; here they are 403 MB.
template <bool BF16>
__global__ void __launch_bounds__(256) square_kernel(const uint4 *__restrict__ x, uint8_t *__restrict__ out, long n8) {
    pdl_wait();
    pdl_trigger();
    const long stride = (long)gridDim.x * 256;
    for (long i = (long)blockIdx.x * 256 + threadIdx.x; i < n8; i += 2 * stride) {
        const bool two = i + stride < n8;
        const uint4 a = ldg_nc_v4(x + i), b = two ? ldg_nc_v4(x + i + stride) : a;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            if (k && !two) break;
            const uint4 v = k ? b : a;
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
            uint32_t o[8];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float lo, hi;
                if (BF16) { lo = __uint_as_float(w[j] << 16); hi = __uint_as_float(w[j] & 0xffff0000u); }
                else { const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&w[j])); lo = f.x; hi = f.y; }
                o[2 * j] = __float_as_uint(__fmul_rn(lo, lo));
                o[2 * j + 1] = __float_as_uint(__fmul_rn(hi, hi));
            }
            stg_v8(out + (i + k * stride) * 32, make_uint4(o[0], o[1], o[2], o[3]), make_uint4(o[4], o[5], o[6], o[7]));
        }
    }
}

struct RopeParams {
    const __half *qkv;         // [B * S, (nh + 2 nkv) * D]
    const float *cos, *sin;    // [S, D / 2] for the S positions of this step
    __half *q_out;             // [B, nh, S, D], or [B, S, nh, D]
    __half *k_cache, *v_cache; // [B, nkv, T, D]
    int B, S, nh, nkv, D, T, cur;
    int q_by_token;            // q_out is [B, S, nh, D]
};

// One block per token (and part of its heads); a thread takes W elements of the first half of a head and their W rotation
// partners.  The token is the block's, so that a piece costs one small division; W = 8 (16-byte accesses) when D % 16 == 0:
// 335 MB of the 8,192-token, 80-head case in 88 us before, with W = 4 and five 64-bit divisions per piece.
template <int W>
__global__ void __launch_bounds__(256) rope_kv_kernel(const RopeParams p) {
    const int half = p.D / 2, vec = half / W;                      // pieces of W elements per half head
    const int heads = p.nh + 2 * p.nkv, items = heads * vec;
    const long token = blockIdx.x;
    pdl_wait();
    pdl_trigger();
    const int b = (int)(token / p.S), s = (int)(token - (long)b * p.S);
    for (int i = blockIdx.y * 256 + threadIdx.x; i < items; i += gridDim.y * 256) {
        const int h = i / vec, v = i - h * vec;
        const __half *src = p.qkv + (token * heads + h) * p.D + v * W;
        alignas(16) __half a[W], bb[W];
        if (W == 8) {
            *reinterpret_cast<uint4 *>(a) = ldg_nc_v4(src);
            *reinterpret_cast<uint4 *>(bb) = ldg_nc_v4(src + half);
        } else {
            *reinterpret_cast<uint2 *>(a) = *reinterpret_cast<const uint2 *>(src);
            *reinterpret_cast<uint2 *>(bb) = *reinterpret_cast<const uint2 *>(src + half);
        }
        if (h < p.nh + p.nkv) {                                    // q and k rotate; v passes through
#pragma unroll
            for (int e4 = 0; e4 < W; e4 += 4) {
                const float4 c = *reinterpret_cast<const float4 *>(p.cos + (long)s * half + v * W + e4);
                const float4 sn = *reinterpret_cast<const float4 *>(p.sin + (long)s * half + v * W + e4);
                const float cc[4] = {c.x, c.y, c.z, c.w}, ss[4] = {sn.x, sn.y, sn.z, sn.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float x1 = __half2float(a[e4 + e]), x2 = __half2float(bb[e4 + e]);
                    // x1 cos - x2 sin and x2 cos + x1 sin, every product and sum rounded on its own (as separate tensor operations do)
                    a[e4 + e] = __float2half_rn(__fsub_rn(__fmul_rn(x1, cc[e]), __fmul_rn(x2, ss[e])));
                    bb[e4 + e] = __float2half_rn(__fadd_rn(__fmul_rn(x2, cc[e]), __fmul_rn(x1, ss[e])));
                }
            }
        }
        __half *dst;
        if (h < p.nh) dst = p.q_out + (p.q_by_token ? token * p.nh + h : ((long)b * p.nh + h) * p.S + s) * p.D;
        else if (h < p.nh + p.nkv) dst = p.k_cache + (((long)b * p.nkv + (h - p.nh)) * p.T + p.cur + s) * p.D;
        else dst = p.v_cache + (((long)b * p.nkv + (h - p.nh - p.nkv)) * p.T + p.cur + s) * p.D;
        dst += v * W;
        if (W == 8) {
            *reinterpret_cast<uint4 *>(dst) = *reinterpret_cast<const uint4 *>(a);
            *reinterpret_cast<uint4 *>(dst + half) = *reinterpret_cast<const uint4 *>(bb);
        } else {
            *reinterpret_cast<uint2 *>(dst) = *reinterpret_cast<const uint2 *>(a);
            *reinterpret_cast<uint2 *>(dst + half) = *reinterpret_cast<const uint2 *>(bb);
        }
    }
}

}  // namespace

int launch_silu_mul(const void *gu, int in_dtype, long M, long F, long ld, void *out, cudaStream_t stream) {
    if (M == 0 || F == 0) return 0;
    // enough blocks for 2,048 threads on every SM
    const long cols = (F / 8 + kSiluThreads - 1) / kSiluThreads;
    long rows = (16L * kNumSMs + cols - 1) / cols;
    if (rows > M) rows = M;
    const dim3 grid((unsigned)cols, (unsigned)rows);
    if (in_dtype == FLH_B200_BF16)
        return cuda_status(launch_pdl(silu_mul_kernel<true>, grid, kSiluThreads, 0, stream, static_cast<const uint8_t *>(gu), M, F, ld * 2, static_cast<uint8_t *>(out)), "silu_mul launch");
    return cuda_status(launch_pdl(silu_mul_kernel<false>, grid, kSiluThreads, 0, stream, static_cast<const uint8_t *>(gu), M, F, ld * 2, static_cast<uint8_t *>(out)), "silu_mul launch");
}

int launch_square(const void *x, int in_dtype, long n, void *out, cudaStream_t stream) {
    if (n == 0) return 0;
    long grid = (n / 8 + 255) / 256;
    if (grid > 8L * kNumSMs) grid = 8L * kNumSMs;
    return cuda_status(launch_pdl(in_dtype == FLH_B200_BF16 ? square_kernel<true> : square_kernel<false>, dim3((unsigned)grid), 256, 0, stream,
                                  static_cast<const uint4 *>(x), static_cast<uint8_t *>(out), n / 8), "square launch");
}

int launch_rope_kv(const void *qkv, const float *cos, const float *sin, void *q_out, void *k_cache, void *v_cache,
                   int B, int S, int nh, int nkv, int D, int T, int cur, int q_by_token, cudaStream_t stream) {
    RopeParams p;
    p.qkv = static_cast<const __half *>(qkv);
    p.cos = cos; p.sin = sin;
    p.q_out = static_cast<__half *>(q_out);
    p.k_cache = static_cast<__half *>(k_cache);
    p.v_cache = static_cast<__half *>(v_cache);
    p.B = B; p.S = S; p.nh = nh; p.nkv = nkv; p.D = D; p.T = T; p.cur = cur; p.q_by_token = q_by_token;
    const long tokens = (long)B * S;
    if (tokens == 0) return 0;
    const int w = D % 16 == 0 ? 8 : 4;
    const long items = (long)(nh + 2 * nkv) * (D / 2 / w), parts = (items + 255) / 256;
    // a token's heads are spread over several blocks only while the tokens alone do not fill the GPU
    const dim3 grid((unsigned)tokens, (unsigned)(tokens >= 4L * kNumSMs ? 1 : parts));
    return cuda_status(launch_pdl(w == 8 ? rope_kv_kernel<8> : rope_kv_kernel<4>, grid, 256, 0, stream, p), "rope_kv launch");
}

}  // namespace flh
