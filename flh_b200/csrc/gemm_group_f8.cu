// int4 x int4 GEMM with group-128 scales for prefill batches, on the fp8 tensor cores (tcgen05 kind::f8f6f4).
//
// The contract is acc = fmaf(float(I_g), sa * sb, acc) for every 128-K group g ascending, I_g the exact integer dot product
// of the group: a binary32 multiply and a multiply-add per output element and group on the CUDA cores, 512 clocks per
// 128 x 256 x 128 block — exactly what the tensor core needs for the block.  So nothing else may be left on the CUDA cores:
//   * I_g must arrive as binary32.  An e4m3 byte 0x00 .. 0x08 is the number 0 .. 8 times 2^-9 (the subnormals and the first
//     normal lie on one line), so a signed int4 code is sign | magnitude, products are exact, |I_g| <= 2^13 units of 2^-18
//     is exact in the binary32 accumulator, and there is no int -> float conversion.  The 2^18 rides in sa (a power of two:
//     exact).
//   * the expansion of the codes is a pass of its own in front (prep_group_f8_kernel), as are the scales, which are laid out
//     [group][row] in binary32, so that a block's 256 + 128 scales are two bulk copies into a ring in shared memory.
// A pair of CTAs (cta_group::2) shares one 256 x BN tile, as in gemm_i8.cu: 64 KB of shared-memory traffic per CTA and
// block instead of 96.  Per block the MMA thread fills one of two TMEM buffers while the epilogue warps fold the other.
//
// Measured (B200, expansion included, operands from HBM): 2048 x 4096 -> 12288 149 us, 4096 -> 22016 243 us, 11008 -> 4096 132 us; the
// converting kernel of gemm_tcgen05.cu, which has the same results, 272, 445 and 256 us.  The epilogue is the limit, and of its time what
// it spends on barriers counts most.  For the first shape, the same operands call after call: eight epilogue warps and issue loops walked by one lane 183; sixteen warps 179; their
// wait and arrival for the scales of every fourth K-block in place of each 157; waits with one outcome for the warp (mbar_wait_warp)
// and the leader's barrier mapped once 146.
//
//   warp 0   TMA: 128 rows of A and BN / 2 rows of B per stage        warp 1   MMA issuer (the leader's)
//   warp 2   bulk copies of the scales                                warps 4-19 epilogue, 32 rows x 64 columns each
//
// Every wait is bounded (two seconds) and reports through a status word, as in the other GEMM kernels.
#include "tc_common.cuh"
#include "tc_pair.cuh"

namespace flh {
namespace {

constexpr int BM = 128;
constexpr int BK = 128;                  // K of a block = one group = one 128-byte swizzle row of e4m3
constexpr int kRing = 3;                 // scale slots
constexpr int kSB = 4;                   // K-blocks of a scale slot: a wait and an arrival of every epilogue warp per slot
constexpr int EW = 16;                   // epilogue warps, 32 rows x 64 columns each
constexpr int BN = 256;                  // columns of a tile

__device__ int g_status_f8[4];

__device__ __forceinline__ bool wait_f8(uint32_t bar, uint32_t parity, volatile int *abort_flag, int code) {
    return mbar_wait_warp(g_status_f8, bar, parity, abort_flag, code);
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void mma_f8_pair(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accum) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accum) : "memory");
}

// ---- preparation ------------------------------------------------------------------------------
// four two's-complement nibbles (one per byte) -> e4m3 bytes sign | |q|
__device__ __forceinline__ uint32_t nibbles_to_f8(uint32_t x) {
    const uint32_t s = x & 0x08080808u, one = s >> 3;
    return ((((x & 0x07070707u) ^ (s - one)) + one)) | (s << 4);
}
// Where the scale of a row or column lies within its group's line: so that what one epilogue thread needs is 16 bytes.  It holds
// rows r, r + 8, r + 16, r + 24 of 32 and, of every 16 columns, 2 q, 2 q + 1, 8 + 2 q and 9 + 2 q.
__device__ __forceinline__ int row_slot(int r) { return (r & ~31) | ((r & 7) << 2) | ((r >> 3) & 3); }
__device__ __forceinline__ int col_slot(int c) { return (c & ~15) | ((c & 6) << 1) | ((c >> 2) & 2) | (c & 1); }
// bound by memory: 1.5 bytes per code of A and B; the scales are a few per cent of that
struct PrepParams {
    const uint4 *a, *b;
    uint4 *ea, *eb;
    long a16, b16;                       // 16-byte packed chunks of A, of B
    const __half *a_scale, *b_scale;
    float *sa, *sb;                      // [G][Mp], [G][N]
    int M, Mp, N, G, ga_cols, gb_cols;
};
__global__ void __launch_bounds__(256) prep_group_f8_kernel(const PrepParams p) {
    const long stride = (long)gridDim.x * blockDim.x, t0 = (long)blockIdx.x * blockDim.x + threadIdx.x;
    const long total = p.a16 + p.b16;
    pdl_trigger();
    constexpr int U = 4;                                 // loads in flight
    for (long i0 = t0; i0 < total; i0 += stride * U) {
        uint4 wv[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const long i = i0 + u * stride;
            if (i < total) wv[u] = ldg_nc_v4(i >= p.a16 ? p.b + (i - p.a16) : p.a + i);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const long i = i0 + u * stride;
            if (i >= total) break;
            const bool isb = i >= p.a16;
            const long j = isb ? i - p.a16 : i;
            const uint4 w = wv[u];
            uint4 e, o;
            e.x = nibbles_to_f8(w.x & 0x0F0F0F0Fu); e.y = nibbles_to_f8(w.y & 0x0F0F0F0Fu);
            e.z = nibbles_to_f8(w.z & 0x0F0F0F0Fu); e.w = nibbles_to_f8(w.w & 0x0F0F0F0Fu);
            o.x = nibbles_to_f8((w.x >> 4) & 0x0F0F0F0Fu); o.y = nibbles_to_f8((w.y >> 4) & 0x0F0F0F0Fu);
            o.z = nibbles_to_f8((w.z >> 4) & 0x0F0F0F0Fu); o.w = nibbles_to_f8((w.w >> 4) & 0x0F0F0F0Fu);
            stg_v8((isb ? p.eb : p.ea) + 2 * j, e, o);
        }
    }
    // scales: a thread takes one row and eight consecutive groups, so that its 2-byte reads share a sector
    const int G8 = (p.G + 7) / 8;
    const long na = (long)p.Mp * G8, nb = (long)p.N * G8;
    for (long i = t0; i < na + nb; i += stride) {
        const bool isb = i >= na;
        const long j = isb ? i - na : i;
        const int rows = isb ? p.N : p.Mp;
        const int g0 = (int)(j / rows) * 8, r = (int)(j - (long)(j / rows) * rows);
        const int cols = isb ? p.gb_cols : p.ga_cols;
        const __half *src = (isb ? p.b_scale : p.a_scale) + (long)r * cols;
        float *dst = (isb ? p.sb : p.sa) + (isb ? col_slot(r) : row_slot(r));
        const bool live = isb || r < p.M;
        const float unit = isb ? 1.0f : 262144.0f;       // the 2^18 of the two e4m3 operands
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (g0 + k < p.G) dst[(long)(g0 + k) * rows] = live ? __half2float(src[cols > 1 ? g0 + k : 0]) * unit : 0.0f;
    }
}

// ---- the GEMM ---------------------------------------------------------------------------------
struct F8Params {
    const float *sa, *sb;                // [G][Mp] (times 2^18), [G][N]
    const __half *bias;
    void *D;
    int M, Mp, N, KB;
    int out_bf16;
    int num_tiles, m_blocks;             // tiles of 256 x BN, row blocks fastest
};

struct F8Plan {
    static constexpr int kStageBytes = (BM + BN / 2) * BK;
    static constexpr int kStages = 6;
    static constexpr int kRingOff = kStages * kStageBytes;
    static constexpr int kScales = (BN + BM) * 4;         // of a K-block: weight scales, then token scales
    static constexpr int kSlot = kSB * kScales;
    static constexpr int kBarOff = kRingOff + kRing * kSlot;
    static constexpr int kBytes = kBarOff + 512 + 1024;   // barriers, then slack to align the base to 1024
    static constexpr int kThreads = 128 + 32 * EW;
};

__global__ void __launch_bounds__(F8Plan::kThreads, 1)
gemm_group_f8_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const F8Params p) {
    using Plan = F8Plan;
    constexpr int S = Plan::kStages, COLS = 64;             // COLS: columns of an epilogue warp
    extern __shared__ uint8_t smem_dyn[];
    const uint32_t raw = smem_u32(smem_dyn);
    const uint32_t base = (raw + 1023u) & ~1023u;         // the same offset in both CTAs of a pair
    uint8_t *sm = smem_dyn + (base - raw);

    const uint32_t bars = base + Plan::kBarOff;
    auto full = [&](int s) { return bars + 8u * s; };                  // both CTAs' tiles of stage s, counted by the leader
    auto empty = [&](int s) { return bars + 8u * (8 + s); };
    auto sfull = [&](int s) { return bars + 8u * (16 + s); };          // the scales of a block have landed
    auto sempty = [&](int s) { return bars + 8u * (24 + s); };
    auto acc_full = [&](int b) { return bars + 8u * (32 + b); };
    auto acc_empty = [&](int b) { return bars + 8u * (34 + b); };      // leader only
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(sm + Plan::kBarOff + 8 * 40);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(sm + Plan::kBarOff + 8 * 40 + 8);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int KB = p.KB;
    const uint32_t rank = cluster_rank();
    const int first = (int)(blockIdx.x >> 1), step = (int)(gridDim.x >> 1);

    if (tid == 0) {
        for (int s = 0; s < S; ++s) { mbar_init(full(s), 1); mbar_init(empty(s), 1); }
        for (int s = 0; s < kRing; ++s) { mbar_init(sfull(s), 1); mbar_init(sempty(s), EW); }
        for (int b = 0; b < 2; ++b) { mbar_init(acc_full(b), 1); mbar_init(acc_empty(b), 2 * EW); }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_proxy_async();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();                      // both CTAs' barriers exist before anyone signals across
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 32;" ::);     // 128 x 32 + 512 x 112 = 640 x 96, what the block is launched with
        if (warp == 0) {
            // -------------------------------------------------------- TMA producer (own halves)
            pdl_wait();                      // the operands are made by the kernel before; the set-up above overlapped it
            int it = 0, s = 0;
            uint32_t ph = 1;
            bool ok = true;
            for (int tile = first; tile < p.num_tiles; tile += step) {
                const int m0 = (tile % p.m_blocks) * 2 * BM + (int)rank * BM;
                const int n0 = (tile / p.m_blocks) * BN + (int)rank * (BN / 2);
                for (int kb = 0; kb < KB; ++kb) {
                    ok = ok && wait_f8(empty(s), ph, abort_flag, 41);
                    const uint32_t dst = base + s * Plan::kStageBytes;
                    if (ok && elect_one()) {
                        if (rank == 1) {
                            tma_load_2d_to_leader(dst, &map_a, kb * BK, m0, full(s));
                            tma_load_2d_to_leader(dst + BM * BK, &map_b, kb * BK, n0, full(s));
                        } else {
                            mbar_expect_tx(full(s), 2 * Plan::kStageBytes);
                            tma_load_2d(dst, &map_a, kb * BK, m0, full(s));
                            tma_load_2d(dst + BM * BK, &map_b, kb * BK, n0, full(s));
                        }
                    }
                    __syncwarp();
                    it += ok;
                    if (++s == S) { s = 0; ph ^= 1; }
                }
            }
            if (*abort_flag && rank == 0) {      // let the copies already issued land before the CTA leaves
                for (int j = it > S ? it - S : 0; j < it; ++j) {
                    const uint64_t t0 = gtimer();
                    while (!mbar_try(full(j % S), (j / S) & 1) && gtimer() - t0 < 100000000ull) {}
                }
            }
        } else if (warp == 2) {
            // -------------------------------------------------------- scales of every block
            pdl_wait();
            int it = 0, slot = 0;
            uint32_t ph = 1;
            bool ok = true;
            for (int tile = first; tile < p.num_tiles; tile += step) {
                const float *sa = p.sa + (tile % p.m_blocks) * 2 * BM + (int)rank * BM, *sb = p.sb + (tile / p.m_blocks) * BN;
                for (int kb = 0; kb < KB; kb += kSB) {
                    const int nb = min(kSB, KB - kb);
                    ok = ok && wait_f8(sempty(slot), ph, abort_flag, 44);
                    const uint32_t dst = base + Plan::kRingOff + slot * Plan::kSlot;
                    if (ok && elect_one()) {
                        mbar_expect_tx(sfull(slot), nb * Plan::kScales);
                        for (int b = 0; b < nb; ++b) {
                            bulk_load(dst + b * Plan::kScales, sb + (long)b * p.N, BN * 4, sfull(slot));
                            bulk_load(dst + b * Plan::kScales + BN * 4, sa + (long)b * p.Mp, BM * 4, sfull(slot));
                        }
                    }
                    __syncwarp();
                    sa += (long)kSB * p.Mp; sb += (long)kSB * p.N;
                    it += ok;
                    if (++slot == kRing) { slot = 0; ph ^= 1; }
                }
            }
            if (*abort_flag) {
                for (int j = it > kRing ? it - kRing : 0; j < it; ++j) {
                    const uint64_t t0 = gtimer();
                    while (!mbar_try(sfull(j % kRing), (j / kRing) & 1) && gtimer() - t0 < 100000000ull) {}
                }
            }
        } else if (warp == 1 && rank == 0) {
            // -------------------------------------------------------- MMA issuer (the whole warp walks the loop, see elect_one)
            // D binary32, A and B e4m3 (format 0), N = BN, M = 256
            const uint32_t idesc = (1u << 4) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)((2 * BM) >> 4) << 24);
            int it = 0, s = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int tile = first; tile < p.num_tiles; tile += step) {
                for (int kb = 0; kb < KB; ++kb, ++it) {
                    const int buf = it & 1;
                    ok = ok && wait_f8(full(s), ph, abort_flag, 43) && wait_f8(acc_empty(buf), ((it >> 1) & 1) ^ 1, abort_flag, 42);
                    tc_fence_after();
                    const uint32_t a_addr = base + s * Plan::kStageBytes;
                    const uint64_t adesc = make_smem_desc(a_addr), bdesc = make_smem_desc(a_addr + BM * BK);
                    if (ok && elect_one()) {
#pragma unroll
                        for (int k4 = 0; k4 < BK / 32; ++k4)
                            mma_f8_pair(tmem + buf * 256, adesc + 2 * k4, bdesc + 2 * k4, idesc, k4 > 0 ? 1u : 0u);
                        tc_commit_pair(acc_full(buf));
                        tc_commit_pair(empty(s));
                    }
                    __syncwarp();
                    if (++s == S) { s = 0; ph ^= 1; }
                }
            }
        }
    } else {
        // ------------------------------------------------------------ epilogue
        asm volatile("setmaxnreg.inc.sync.aligned.u32 112;" ::);
        const int wq = warp & 3;                         // TMEM lane quarter this warp may read
        const int c0 = ((warp - 4) >> 2) * COLS;         // first tile column of this warp
        const uint32_t tlane = tmem + ((uint32_t)(wq * 32) << 16) + c0;
        const uint32_t leader_empty = map_to_leader(acc_empty(0));
        int it = 0, slot = 0;
        uint32_t sph = 0;
        bool ok = true;
        // The outcome of every wait is made warp-uniform by a vote, and a warp that gave up keeps walking the loops (no
        // waits, no TMEM reads, no stores): warp-wide tcgen05.ld never runs in a diverged warp.
        for (int tile = first; tile < p.num_tiles; tile += step) {
            const int m0 = (tile % p.m_blocks) * 2 * BM + (int)rank * BM;
            const int n0 = (tile / p.m_blocks) * BN;
            const int r0 = wq * 32 + (lane >> 2);            // this thread's rows of the tile: r0, + 8, + 16, + 24
            uint64_t acc[4][COLS / 8];                       // [row][8-column block]: columns 8 n + 2 (lane % 4) and the next
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int n = 0; n < COLS / 8; ++n) acc[r][n] = 0ull;
#pragma unroll 1
            for (int kb = 0; kb < KB; ++kb, ++it) {
                const int buf = it & 1, sub = kb % kSB;
                ok = ok && (sub != 0 || wait_f8(sfull(slot), sph, abort_flag, 45)) && wait_f8(acc_full(buf), (it >> 1) & 1, abort_flag, 46);
                auto release_acc = [&]() {               // the accumulator is in registers: the tensor core may have the buffer
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_cluster(leader_empty + 8u * buf);
                };
                if (ok) {
                    const float *sl = reinterpret_cast<const float *>(sm + Plan::kRingOff + slot * Plan::kSlot + sub * Plan::kScales);
                    const uint32_t src = tlane + buf * 256;
                    tc_fence_after();
                    // the next 16 columns are on their way from TMEM while these are folded
                    uint32_t vv[2][16];
                    tc_ld_frag2(src, vv[0]);
                    tc_ld_frag2(src + (16u << 16), vv[0] + 8);
                    const float4 sa = *reinterpret_cast<const float4 *>(sl + BN + wq * 32 + (lane >> 2) * 4);
                    const uint64_t sa2[4] = {pack2(sa.x, sa.x), pack2(sa.y, sa.y), pack2(sa.z, sa.z), pack2(sa.w, sa.w)};
                    const ulonglong2 *sb = reinterpret_cast<const ulonglong2 *>(sl + c0) + (lane & 3);
#pragma unroll
                    for (int cc = 0; cc < COLS / 16; ++cc) {
                        const ulonglong2 sb2 = sb[cc * 4];
                        tc_wait_ld();
                        if (cc + 1 < COLS / 16) {
                            tc_ld_frag2(src + (cc + 1) * 16, vv[(cc + 1) & 1]);
                            tc_ld_frag2(src + (cc + 1) * 16 + (16u << 16), vv[(cc + 1) & 1] + 8);
                        } else release_acc();
                        const uint32_t (&v)[16] = vv[cc & 1];
#pragma unroll
                        for (int n = 0; n < 2; ++n) {
#pragma unroll
                            for (int r = 0; r < 4; ++r) {
                                const int i = (r >> 1) * 8 + 4 * n + 2 * (r & 1);
                                acc[r][cc * 2 + n] = fma2(((uint64_t)v[i + 1] << 32) | v[i], mul2(sa2[r], n ? sb2.y : sb2.x), acc[r][cc * 2 + n]);
                            }
                        }
                    }
                } else {
                    release_acc();
                }
                if (sub == kSB - 1 || kb == KB - 1) {
                    __syncwarp();
                    if (lane == 0) mbar_arrive(sempty(slot));
                    if (++slot == kRing) { slot = 0; sph ^= 1; }
                }
            }
            // Four lanes hold a row's columns two by two: they exchange 4 x 4 words so that each has eight neighbours (one 16-byte
            // store; four lanes then write 64 bytes of a row).
            const int q = lane & 3;
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int row = m0 + r0 + 8 * r;
#pragma unroll
                for (int n4 = 0; n4 < COLS / 32; ++n4) {
                    uint32_t w[4];
#pragma unroll
                    for (int n = 0; n < 4; ++n) {
                        float lo, hi;
                        unpack2(acc[r][n4 * 4 + n], lo, hi);
                        if (p.bias) {
                            const int col = n0 + c0 + (n4 * 4 + n) * 8 + 2 * q;
                            lo = __fadd_rn(lo, __half2float(p.bias[col]));
                            hi = __fadd_rn(hi, __half2float(p.bias[col + 1]));
                        }
                        if (p.out_bf16) { const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi); w[n] = *reinterpret_cast<const uint32_t *>(&h); }
                        else { const __half2 h = __floats2half2_rn(lo, hi); w[n] = *reinterpret_cast<const uint32_t *>(&h); }
                    }
                    uint32_t a = __shfl_xor_sync(0xffffffffu, q & 1 ? w[0] : w[1], 1), b = __shfl_xor_sync(0xffffffffu, q & 1 ? w[2] : w[3], 1);
                    if (q & 1) { w[0] = a; w[2] = b; } else { w[1] = a; w[3] = b; }
                    a = __shfl_xor_sync(0xffffffffu, q & 2 ? w[0] : w[2], 2); b = __shfl_xor_sync(0xffffffffu, q & 2 ? w[1] : w[3], 2);
                    if (q & 2) { w[0] = a; w[1] = b; } else { w[2] = a; w[3] = b; }
                    if (ok && row < p.M)
                        *reinterpret_cast<uint4 *>(static_cast<uint16_t *>(p.D) + (long)row * p.N + n0 + c0 + (n4 * 4 + q) * 8) = make_uint4(w[0], w[1], w[2], w[3]);
                }
            }
        }
    }

    __syncthreads();
    cluster_sync_all();                      // nobody signals the peer's barriers or reads its tiles after this
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

int launch_f8(const CUtensorMap &ma, const CUtensorMap &mb, F8Params p, cudaStream_t stream) {
    using Plan = F8Plan;
    auto kern = gemm_group_f8_kernel;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Plan::kBytes);
    if (e != cudaSuccess) return cuda_status(e, "gemm_group_f8 attribute");
    p.m_blocks = (p.M + 2 * BM - 1) / (2 * BM);
    p.num_tiles = p.m_blocks * (p.N / BN);
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    cfg.blockDim = dim3(Plan::kThreads);
    cfg.dynamicSmemBytes = Plan::kBytes;
    cfg.stream = stream;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = 2;
    // persistent: no more pairs than can be resident at once
    static int max_pairs = 0;
    if (max_pairs == 0) {
        cfg.gridDim = dim3(tc_device_sms() / 2 * 2);
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n < 1) n = tc_device_sms() / 2;
        max_pairs = n;
    }
    cfg.gridDim = dim3(2 * (p.num_tiles < max_pairs ? p.num_tiles : max_pairs));
    e = cudaLaunchKernelEx(&cfg, kern, ma, mb, p);
    return cuda_status(e, "gemm_group_f8 launch");
}

size_t up256(size_t v) { return (v + 255) & ~(size_t)255; }

}  // namespace

bool gemm_group_f8_supported(long M, long N, long K) { return M > 0 && N % 256 == 0 && K % 128 == 0; }

// e4m3 A, e4m3 B, token scales [G][Mp], weight scales [G][N]
size_t gemm_group_f8_workspace_bytes(long M, long N, long K) {
    const size_t G = (size_t)K / 128, Mp = ((size_t)M + 255) / 256 * 256;
    return up256((size_t)M * K) + up256((size_t)N * K) + G * Mp * 4 + G * (size_t)N * 4;
}

int launch_gemm_group_f8(const uint8_t *A, const uint8_t *B, const void *a_scale, const void *b_scale, const void *bias, void *D,
                         long M, long N, long K, long a_group, long b_group, int out_dtype, void *workspace, cudaStream_t stream) {
    const long G = K / 128, Mp = (M + 255) / 256 * 256;
    uint8_t *ea = static_cast<uint8_t *>(workspace), *eb = ea + up256((size_t)M * K);
    float *sa = reinterpret_cast<float *>(eb + up256((size_t)N * K)), *sb = sa + G * Mp;
    PrepParams q;
    q.a = reinterpret_cast<const uint4 *>(A); q.b = reinterpret_cast<const uint4 *>(B);
    q.ea = reinterpret_cast<uint4 *>(ea); q.eb = reinterpret_cast<uint4 *>(eb);
    q.a16 = M * K / 32; q.b16 = N * K / 32;
    q.a_scale = static_cast<const __half *>(a_scale); q.b_scale = static_cast<const __half *>(b_scale);
    q.sa = sa; q.sb = sb;
    q.M = (int)M; q.Mp = (int)Mp; q.N = (int)N; q.G = (int)G;
    q.ga_cols = (int)(K / a_group); q.gb_cols = (int)(K / b_group);
    long grid = (q.a16 + q.b16 + 255) / 256;
    if (grid > 8L * tc_device_sms()) grid = 8L * tc_device_sms();
    prep_group_f8_kernel<<<(unsigned)grid, 256, 0, stream>>>(q);
    int rc = cuda_status(cudaGetLastError(), "prep_group_f8 launch");
    if (rc) return rc;
    F8Params p;
    p.sa = sa; p.sb = sb;
    p.bias = static_cast<const __half *>(bias);
    p.D = D;
    p.M = (int)M; p.Mp = (int)Mp; p.N = (int)N; p.KB = (int)G;
    p.out_bf16 = out_dtype == FLH_B200_BF16;
    CUtensorMap ma, mb;
    rc = make_map_bytes(&ma, ea, M, K, BM);
    if (rc) return rc;
    rc = make_map_bytes(&mb, eb, N, K, 128);
    if (rc) return rc;
    return launch_f8(ma, mb, p, stream);
}

int gemm_group_f8_status(int *out4) {
    return cuda_status(cudaMemcpyFromSymbol(out4, g_status_f8, sizeof(int) * 4), "status read");
}
int gemm_group_f8_status_clear() {
    int z[4] = {0, 0, 0, 0};
    return cuda_status(cudaMemcpyToSymbol(g_status_f8, z, sizeof(z)), "status clear");
}

}  // namespace flh
