// Decode GEMM (M <= 64 tokens): the packed weights stream through a TMA ring, mma.sync.m16n8k32 multiplies them.
//
// Bound by the weight bytes; what has to be kept down is the instructions a warp spends per kilobyte of them (the cp.async
// kernel of gemm_mma.cu: 269 at 16 tokens, two thirds of all issue slots at 2.5 TB/s) and the launch's fixed cost (about
// 9 us in the tcgen05 form of gemm_decode_tc.cu).  So:
//   * one thread issues the copies (warp 8), no warp computes an address of global memory in the main loop;
//   * a warp owns 32 channels x 256 K of a stage: 94 instructions per 2 KB at 16 tokens, the tokens' expansion shared by
//     both 16-row tiles;
//   * the eight warps of a CTA split K (WK of them; 8 / WK share the tokens), so that a stage is a kilobyte of every row and
//     there are N / 32 tiles to spread over the GPU; their partial sums meet in shared memory in a fixed order: int32
//     without group scales (exact), a binary32 chain per warp with them;
//   * the kernel is persistent: the ring runs on into the next tile while the outputs of this one are written.
// Both operands are expanded as in gemm_mma.cu (nibble x 16, even elements then odd ones), the product comes out x 256.
// With group scales the accumulators start at 1.5 * 2^23 as bits: what the tensor core leaves IS the binary32 number
// 1.5 * 2^23 + 256 I (|256 I| < 2^22), so the conversion costs one subtraction.
//
// Shared memory: 16-byte chunk c of a row r lies at chunk c ^ (r & 7) (TMA's 128-byte swizzle).  The eight lanes of a quarter
// read chunks 4h .. 4h + 3 of two rows; rows that differ in bit 2 hit different banks, so row g of the MMA is row
// rho(g) = g / 2 + 4 (g & 1) of the tile, and the same for the tokens.
//
// Measured (B200, weights from HBM, 16 tokens without group scales, us; what AUTO ran before -> this): 4096 -> 4096 8.7 -> 5.1,
// 11008 -> 4096 13.5 -> 7.8, 4096 -> 22016 15.7 -> 13.3 (3.4 TB/s), 8192 -> 28672 35.5 -> 26.3 (4.5 TB/s).  Above 32 tokens the rate of
// mma.sync bounds it (64 per 2 KB of weights).
//
// Every wait is bounded (two seconds) and reports through a status word.
#include "tc_common.cuh"
#include "tc_pair.cuh"

namespace flh {
namespace {

constexpr int kWarps = 8;                // consumer warps; warp 8 produces
constexpr int kThreadsRing = 32 * (kWarps + 1);
constexpr int MT = 2;                    // 16-row tiles of a warp

__device__ int g_status_ring[4];

__device__ __forceinline__ bool wait_ring(uint32_t bar, uint32_t parity, volatile int *abort_flag, int code) {
    return mbar_wait_status(g_status_ring, bar, parity, abort_flag, code);
}

struct RingParams {
    const __half *a_scale, *a_zero, *b_scale, *bias;
    const int32_t *b_rowsum;
    void *D;
    int M, N, KB, chunks, steps, tiles;  // KB groups of 128, chunks of 256, steps of WK chunks
    int ga_cols, gb_cols, out_bf16;
};

constexpr int kMaxChunksGrouped = 128;   // token scales of all K-groups are kept in shared memory: K <= 32768
template <int NT, int WK, bool GROUPED>
struct RingPlan {
    static constexpr int WR = kWarps / WK, BR = 32 * WR, TOK = 8 * NT;
    static constexpr int kW = BR * 128, kX = TOK * 128;           // bytes of one 256-K chunk
    static constexpr int kStage = WK * (kW + kX);
    static constexpr int kPart = kWarps * 32 * TOK * 4;
    static constexpr int kScales = GROUPED ? TOK * 4 * kMaxChunksGrouped : 2 * 64 * 4;
    static constexpr int kFit = (227 * 1024 - 1024 - 256 - kPart - kScales) / kStage;
    static constexpr int kStages = kFit > 5 ? 5 : kFit;
    static constexpr int kPartOff = kStages * kStage;
    static constexpr int kBarOff = kPartOff + kPart;
    static constexpr int kAuxOff = kBarOff + 256;                 // token scales f32 and zero-points s32, or pairs of f16 scales [chunk][token]
    static constexpr int kBytes = kAuxOff + kScales + 1024;
};

template <bool U>
__device__ __forceinline__ void mma_w_tok(int32_t (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    if (U)
        asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.u8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                     : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
    else
        asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                     : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// the scales of two neighbouring groups of one row, as bits (low half = group g0); cols == 1: one scale for all of K
__device__ __forceinline__ uint32_t scale_pair(const __half *s, long row, int cols, int g0) {
    const unsigned short *p = reinterpret_cast<const unsigned short *>(s) + row * cols;
    if (cols == 1) return (uint32_t)__ldg(p) * 0x10001u;
    if ((cols & 1) == 0) return __ldg(reinterpret_cast<const uint32_t *>(p + g0));
    return (uint32_t)__ldg(p + g0) | (uint32_t)__ldg(p + (g0 + 1 < cols ? g0 + 1 : g0)) << 16;
}
__device__ __forceinline__ float half_of(uint32_t pair, int h) {
    return __half2float(__ushort_as_half((unsigned short)(h ? pair >> 16 : pair & 0xFFFFu)));
}

template <int NT, int WK, bool GROUPED, bool ZERO>
__global__ void __launch_bounds__(kThreadsRing, 1)
gemm_decode_ring_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const RingParams p) {
    static_assert(!(GROUPED && ZERO), "zero-points come without group scales here");
    using Plan = RingPlan<NT, WK, GROUPED>;
    constexpr int S = Plan::kStages, BR = Plan::BR, TOK = Plan::TOK;
    static_assert(S >= 2, "the ring needs two stages");
    extern __shared__ uint8_t smem_dyn[];
    const uint32_t raw = smem_u32(smem_dyn);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t *sm = smem_dyn + (base - raw);
    const uint32_t bars = base + Plan::kBarOff;
    auto full = [&](int s) { return bars + 8u * s; };
    auto empty = [&](int s) { return bars + 8u * (8 + s); };
    volatile int *abort_flag = reinterpret_cast<volatile int *>(sm + Plan::kBarOff + 128);
    float *sa_s = reinterpret_cast<float *>(sm + Plan::kAuxOff);
    int *za_s = reinterpret_cast<int *>(sa_s + 64);
    uint32_t *sap_s = reinterpret_cast<uint32_t *>(sa_s);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int s = 0; s < S; ++s) { mbar_init(full(s), 1); mbar_init(empty(s), kWarps); }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_proxy_async();
    }
    if (!GROUPED && tid >= 64 && tid < 64 + TOK) {
        const int j = tid - 64;
        pdl_wait();
        sa_s[j] = j < p.M ? __half2float(p.a_scale[j]) : 0.0f;
        za_s[j] = ZERO && j < p.M ? (int)__half2float(p.a_zero[j]) : 0;
    }
    __syncthreads();                         // the barriers exist: the producer starts

    if (warp == kWarps) {
        // ------------------------------------------------------------ TMA producer
        if (lane == 0) {
            int it = 0;
            bool ok = true;
            // With group scales the first stages of weights come into the L2 cache while the kernel that makes the tokens still runs
            // (a prefetch reads no value, so it needs no order with whatever wrote them).  Without them the barrier above waits
            // for the threads that fetch the token scales behind their own wait, and the prefetch overlaps nothing.
            for (int st = 0; st < S && st < p.steps && (int)blockIdx.x < p.tiles; ++st)
#pragma unroll
                for (int k = 0; k < WK; ++k) tma_prefetch_2d(&map_w, (st * WK + k) * 128, blockIdx.x * BR);
            pdl_wait();
            pdl_trigger();
            for (int tile = blockIdx.x; tile < p.tiles && ok; tile += gridDim.x) {
                for (int st = 0; st < p.steps; ++st, ++it) {
                    const int s = it % S;
                    if (!wait_ring(empty(s), ((it / S) & 1) ^ 1, abort_flag, 61)) { ok = false; break; }
                    mbar_expect_tx(full(s), Plan::kStage);
                    const uint32_t w = base + s * Plan::kStage, x = w + WK * Plan::kW;
#pragma unroll
                    for (int k = 0; k < WK; ++k) tma_load_2d(w + k * Plan::kW, &map_w, (st * WK + k) * 128, tile * BR, full(s));
#pragma unroll
                    for (int k = 0; k < WK; ++k) tma_load_2d(x + k * Plan::kX, &map_x, (st * WK + k) * 128, 0, full(s));
                }
            }
            if (*abort_flag) {               // let the copies already issued land before the CTA leaves
                for (int j = it > S ? it - S : 0; j < it; ++j) {
                    const uint64_t t0 = gtimer();
                    while (!mbar_try(full(j % S), (j / S) & 1) && gtimer() - t0 < 100000000ull) {}
                }
            }
        }
    } else {
        // ------------------------------------------------------------ consumers
        pdl_wait();
        const int kg = warp % WK, wr = warp / WK;
        const int g = lane >> 2, t = lane & 3, rho = (g >> 1) | ((g & 1) << 2);
        const int frag = rho * 128 + ((t ^ rho) << 4);                // chunk t of row rho; chunk 4 + t is at ^ 64
        uint32_t *part = reinterpret_cast<uint32_t *>(sm + Plan::kPartOff);
        const int o_row = tid % BR, o_tok = tid / BR;                 // outputs this thread finishes: one channel, every (256 / BR)-th token
        constexpr int kTokStep = 256 / BR;
        int it = 0;
        bool ok = true;
        if (GROUPED) {                       // token scales of the whole K, while the first tiles are on their way
            for (int i = tid; i < p.chunks * TOK; i += 32 * kWarps) {
                const int tok = i / p.chunks, ch = i - tok * p.chunks;
                sap_s[ch * TOK + tok] = tok < p.M ? scale_pair(p.a_scale, tok, p.ga_cols, 2 * ch) : 0u;
            }
            bar_sync_named(1, 32 * kWarps);
        }
        uint32_t sbn[2 * MT];                                         // channel scales of the next chunk (GROUPED), two groups each
        auto load_scales = [&](int tile, int chunk) {
#pragma unroll
            for (int j = 0; j < 2 * MT; ++j) sbn[j] = scale_pair(p.b_scale, (long)tile * BR + wr * 32 + rho + 8 * j, p.gb_cols, 2 * chunk);
        };
        if (GROUPED && kg < p.chunks && (int)blockIdx.x < p.tiles) load_scales(blockIdx.x, kg);

        // A wait that runs out must not split the warps: they meet at named barriers.  Its outcome is made warp-uniform by a
        // vote, and a warp that gave up keeps walking (no waits, no stores).
        for (int tile = blockIdx.x; tile < p.tiles; tile += gridDim.x) {
            const int n = tile * BR + o_row;
            const float sb_o = GROUPED ? 0.0f : __half2float(p.b_scale[n]) * (1.0f / 256.0f);
            const int rs_o = ZERO ? p.b_rowsum[n] : 0;
            const float bias_o = p.bias ? __half2float(p.bias[n]) : 0.0f;
            int32_t sum[MT][NT][4];                                   // int32 sums, or the bits of binary32 chains (GROUPED)
#pragma unroll
            for (int m = 0; m < MT; ++m)
#pragma unroll
                for (int j = 0; j < NT; ++j)
#pragma unroll
                    for (int e = 0; e < 4; ++e) sum[m][j][e] = 0;
#pragma unroll 1
            for (int st = 0; st < p.steps; ++st, ++it) {
                const int s = it % S, chunk = st * WK + kg;
                uint32_t sbc[2 * MT];
                if (GROUPED) {
#pragma unroll
                    for (int j = 0; j < 2 * MT; ++j) sbc[j] = sbn[j];
                    if (chunk + WK < p.chunks) load_scales(tile, chunk + WK);
                    else if (kg < p.chunks && tile + (int)gridDim.x < p.tiles && st == p.steps - 1) load_scales(tile + gridDim.x, kg);
                }
                ok = __all_sync(0xffffffffu, ok && wait_ring(full(s), (it / S) & 1, abort_flag, 62));
                if (ok && chunk < p.chunks) {
                    const uint8_t *ws = sm + s * Plan::kStage + kg * Plan::kW + wr * 32 * 128 + frag;
                    const uint8_t *xs = sm + s * Plan::kStage + WK * Plan::kW + kg * Plan::kX + frag;
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        uint4 w[2 * MT];
#pragma unroll
                        for (int j = 0; j < 2 * MT; ++j)
                            w[j] = *reinterpret_cast<const uint4 *>(sm + (((uint32_t)(ws - sm) ^ (h << 6)) + j * 1024));
                        uint32_t a[MT][4][4];
#pragma unroll
                        for (int m = 0; m < MT; ++m) {
                            const uint32_t lo[4] = {w[2 * m].x, w[2 * m].y, w[2 * m].z, w[2 * m].w};
                            const uint32_t hi[4] = {w[2 * m + 1].x, w[2 * m + 1].y, w[2 * m + 1].z, w[2 * m + 1].w};
#pragma unroll
                            for (int q = 0; q < 4; ++q) {
                                a[m][q][0] = (lo[q] << 4) & 0xF0F0F0F0u; a[m][q][1] = (hi[q] << 4) & 0xF0F0F0F0u;
                                a[m][q][2] = lo[q] & 0xF0F0F0F0u; a[m][q][3] = hi[q] & 0xF0F0F0F0u;
                            }
                        }
#pragma unroll
                        for (int j = 0; j < NT; ++j) {
                            const uint4 xv = *reinterpret_cast<const uint4 *>(sm + (((uint32_t)(xs - sm) ^ (h << 6)) + j * 1024));
                            const uint32_t xw[4] = {xv.x, xv.y, xv.z, xv.w};
                            int32_t c[MT][4];
#pragma unroll
                            for (int m = 0; m < MT; ++m)
#pragma unroll
                                for (int e = 0; e < 4; ++e) c[m][e] = GROUPED ? 0x4B400000 : sum[m][j][e];
#pragma unroll
                            for (int q = 0; q < 4; ++q) {
                                const uint32_t b0 = (xw[q] << 4) & 0xF0F0F0F0u, b1 = xw[q] & 0xF0F0F0F0u;
#pragma unroll
                                for (int m = 0; m < MT; ++m) mma_w_tok<ZERO>(c[m], a[m][q], b0, b1);
                            }
                            if (!GROUPED) {
#pragma unroll
                                for (int m = 0; m < MT; ++m)
#pragma unroll
                                    for (int e = 0; e < 4; ++e) sum[m][j][e] = c[m][e];
                            } else if (2 * chunk + h < p.KB) {
                                // c[m][2 hh + e]: channel rho + 16 m + 8 hh, token 8 j + t + 4 e
#pragma unroll
                                for (int e = 0; e < 2; ++e) {
                                    const float sa = half_of(sap_s[chunk * TOK + 8 * j + t + 4 * e], h) * (1.0f / 256.0f);
#pragma unroll
                                    for (int m = 0; m < MT; ++m)
#pragma unroll
                                        for (int hh = 0; hh < 2; ++hh) {
                                            const float I = __fsub_rn(__int_as_float(c[m][2 * hh + e]), 12582912.0f);
                                            int32_t &v = sum[m][j][2 * hh + e];
                                            v = __float_as_int(__fmaf_rn(I, __fmul_rn(sa, half_of(sbc[2 * m + hh], h)), __int_as_float(v)));
                                        }
                                }
                            }
                        }
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(empty(s));
            }
            // partial sums: [warp][token][channel], channel ^ 8 (token & 3) so that the four token columns of a warp store use
            // different banks
            uint32_t *mine = part + warp * (32 * TOK);
#pragma unroll
            for (int m = 0; m < MT; ++m)
#pragma unroll
                for (int j = 0; j < NT; ++j)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int tok = 8 * j + t + 4 * (e & 1), row = rho + 16 * m + 8 * (e >> 1);
                        mine[tok * 32 + (row ^ (8 * (tok & 3)))] = (uint32_t)sum[m][j][e];
                    }
            bar_sync_named(1, 32 * kWarps);
            const int prow = o_row & 31;
            const uint32_t *src = part + (o_row >> 5) * WK * (32 * TOK);
            if (ok) {
                for (int tok = o_tok; tok < p.M; tok += kTokStep) {
                    const int off = tok * 32 + (prow ^ (8 * (tok & 3)));
                    float o;
                    if (GROUPED) {
                        o = __uint_as_float(src[off]);
#pragma unroll
                        for (int k = 1; k < WK; ++k) o = __fadd_rn(o, __uint_as_float(src[k * (32 * TOK) + off]));
                    } else {
                        int I = (int)src[off];
#pragma unroll
                        for (int k = 1; k < WK; ++k) I += (int)src[k * (32 * TOK) + off];
                        if (ZERO) I -= (za_s[tok] * rs_o) << 8;
                        o = __fmaf_rn((float)I, __fmul_rn(sa_s[tok], sb_o), 0.0f);
                    }
                    if (p.bias) o = __fadd_rn(o, bias_o);
                    if (p.out_bf16) static_cast<__nv_bfloat16 *>(p.D)[(long)tok * p.N + n] = __float2bfloat16_rn(o);
                    else static_cast<__half *>(p.D)[(long)tok * p.N + n] = __float2half_rn(o);
                }
            }
            bar_sync_named(1, 32 * kWarps);              // the partial sums are rewritten for the next tile
        }
    }
}

template <int NT, int WK, bool GROUPED, bool ZERO>
int launch_ring(const CUtensorMap &mw, const CUtensorMap &mx, RingParams p, cudaStream_t stream) {
    using Plan = RingPlan<NT, WK, GROUPED>;
    auto kern = gemm_decode_ring_kernel<NT, WK, GROUPED, ZERO>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Plan::kBytes);
    if (e != cudaSuccess) return cuda_status(e, "gemm_decode_ring attribute");
    p.steps = (p.chunks + WK - 1) / WK;
    p.tiles = p.N / Plan::BR;
    const int sms = tc_device_sms();
    return cuda_status(launch_pdl(kern, dim3(p.tiles < sms ? p.tiles : sms), kThreadsRing, Plan::kBytes, stream, mw, mx, p), "gemm_decode_ring launch");
}

// packed matrix of rows x K / 2 bytes; box = box_rows x 128 bytes with the 128-byte swizzle, zeros outside
int make_map_packed(CUtensorMap *map, const uint8_t *ptr, long rows, long K, int box_rows) { return make_map_bytes(map, ptr, rows, K / 2, box_rows); }

}  // namespace

// group scales with zero-points stay with the kernels that stage the row sums of every group, and so do the widest rows
bool gemm_decode_ring_supported(long M, long N, long K, bool grouped, bool zero) {
    return M >= 1 && M <= 64 && N % 64 == 0 && K % 128 == 0 && (!grouped || (!zero && K <= 256 * kMaxChunksGrouped));
}

int launch_gemm_decode_ring(const uint8_t *A, const uint8_t *B, const void *a_scale, const void *a_zero, const void *b_scale,
                            const int32_t *b_rowsum, const void *bias, void *D, long M, long N, long K, long a_group, long b_group,
                            int out_dtype, cudaStream_t stream) {
    RingParams p;
    p.a_scale = static_cast<const __half *>(a_scale);
    p.a_zero = static_cast<const __half *>(a_zero);
    p.b_scale = static_cast<const __half *>(b_scale);
    p.bias = static_cast<const __half *>(bias);
    p.b_rowsum = b_rowsum; p.D = D;
    p.M = (int)M; p.N = (int)N; p.KB = (int)(K / 128); p.chunks = (int)((K + 255) / 256);
    p.ga_cols = (int)(K / a_group); p.gb_cols = (int)(K / b_group);
    p.out_bf16 = out_dtype == FLH_B200_BF16;
    const int nt = M <= 8 ? 1 : M <= 16 ? 2 : M <= 32 ? 4 : 8;
    const bool grouped = a_group < K || b_group < K;
    CUtensorMap mw, mx;
    int rc = make_map_packed(&mw, B, N, K, nt == 8 ? 64 : 32);
    if (rc) return rc;
    rc = make_map_packed(&mx, A, M, K, 8 * nt);
    if (rc) return rc;
#define FLH_RING(NT_, WK_) (grouped ? launch_ring<NT_, WK_, true, false>(mw, mx, p, stream) \
                            : a_zero ? launch_ring<NT_, WK_, false, true>(mw, mx, p, stream) : launch_ring<NT_, WK_, false, false>(mw, mx, p, stream))
    switch (nt) {
        case 1: return FLH_RING(1, 8);
        case 2: return FLH_RING(2, 8);
        case 4: return FLH_RING(4, 8);
        default: return FLH_RING(8, 4);
    }
#undef FLH_RING
}

int gemm_decode_ring_status(int *out4) {
    return cuda_status(cudaMemcpyFromSymbol(out4, g_status_ring, sizeof(int) * 4), "status read");
}
int gemm_decode_ring_status_clear() {
    int z[4] = {0, 0, 0, 0};
    return cuda_status(cudaMemcpyToSymbol(g_status_ring, z, sizeof(z)), "status clear");
}

}  // namespace flh
