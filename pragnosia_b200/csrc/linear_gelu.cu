// y = act(x W^T + bias) for the up-projection of the MLP block (src/model.py:552-560: Linear(d, 4d) followed by GELU), as one
// persistent tcgen05 GEMM whose epilogue applies the bias and the erf-GELU on the accumulator as it leaves tensor memory.
// As two ops the activation is a second pass over the 4d-wide hidden tensor (read + write of 2 x M x 4d x 2 bytes, about as
// long as the GEMM itself at d = 768); fused it costs nothing but epilogue arithmetic that overlaps the next tile's MMAs.
//
//   x [M][K] bf16 (K contiguous)  -> A operand, K-major;   W [N][K] bf16 (torch.nn.Linear layout) -> B operand, K-major
//   tile 128 x 256 x 64, four TMA stages of 48 KiB (128-byte swizzle), accumulators 128 lanes x 256 fp32 columns in tensor
//   memory, two of them (512 columns) so that the epilogue of tile i runs under the MMAs of tile i + 1.
//   warp 0: TMA producer;  warp 1: MMA issuer (one elected lane of the converged warp), owns the tensor-memory allocation;
//   warps 2-17: epilogue -- warp w reads TMEM lanes 32 (w mod 4) .. +31 (one output row per thread) and column quarter
//   (w-2)/4, 32 columns at a time with the next 32 already on their way from tensor memory: + bias (one packed pair per
//   lane, fetched at the start of the tile and handed round by shuffles), round to bf16 (where the separate Linear would
//   round), GELU in fp32, round, 64-byte stores. The epilogue's arithmetic is as long as the tile's MMAs, so its length
//   per element decides the kernel's speed: see lg_gelu.
//   One CTA per SM walks tiles blockIdx.x, blockIdx.x + gridDim.x, ... (column blocks fastest, so the CTAs running together
//   share rows of x in L2). Every mbarrier wait is bounded; a wait that runs out sets the error flag and the CTA winds down.
#include "tc_common.cuh"

namespace pgb {

constexpr int LG_BM = 128, LG_BK = 64, LG_STAGES = 4;
constexpr int LG_EPI = 16;                                            // epilogue warps: four per tensor-memory subpartition
constexpr int LG_NT = (2 + LG_EPI) * 32;
constexpr int LG_A_BYTES = LG_BM * LG_BK * 2;
// The tile is 128 x BN with BN = 256 (the default) or 192 columns. At N = 3072 on 148 SMs, 768 tiles of 256 are 5.2 rounds
// and pay for 6, 1024 tiles of 192 are 6.9 rounds and pay for 7 three-quarter ones -- and take the same time to within
// 2 % (39.4 vs 39.9 us), as do 24 epilogue warps in place of 16 (slower by 5 %): neither the rounding of the tile count nor
// latency inside the epilogue is what the kernel waits for. An epilogue warp owns BN / 4 columns of 32 rows.
template <int BN, int EPI = LG_EPI>
struct LgCfg {
    static constexpr int NT = (2 + EPI) * 32;
    static constexpr int CW = BN / (EPI / 4);                         // columns per epilogue warp: 64, 48 or 32
    static constexpr int B_BYTES = BN * LG_BK * 2, STAGE = LG_A_BYTES + B_BYTES;
    static constexpr int OUT_BYTES = 32 * (CW == 64 ? 32 : CW) * 2;  // per epilogue warp: 32 rows of the columns it stages at a time
    static constexpr int SMEM = LG_STAGES * STAGE + 1024 + EPI * OUT_BYTES + 1024;   // stages, barriers, output staging, alignment slack
    static_assert(BN == 256 || BN == 192, "tile width");
    static_assert(STAGE % 1024 == 0 && SMEM <= 232448, "shared memory");
};

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, uint32_t bar, int c0, int c1) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
                 ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(0) : "memory");
}
__device__ __forceinline__ void lg_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// GELU(x) = x Phi(x) with Phi(x) = 0.5 (1 + erf(x / sqrt 2)) written as a logistic function of an odd polynomial,
// Phi(x) ~= 1 / (1 + exp(-2 x p(x^2))): p fitted (minimax, |x| <= 6, beyond which Phi is 0 or 1 to 1e-9) so that the result
// is within 3.3e-5 of the erf form everywhere -- a sixtieth of the bf16 rounding of a value near 1. The logistic form has
// no cancellation in either tail (1 + tanh would), and costs a dozen instructions with two special-function issues
// against about twenty for an erf polynomial.
__device__ __forceinline__ float lg_gelu(float x) {
    // the coefficients carry the factor -2 log2(e); the square is clamped, so beyond |x| = 6 the exponent keeps growing with
    // x and the result goes to x or to -0 as it should
    const float z2 = fminf(x * x, 36.0f);
    float p = fmaf(4.6257928e-05f, z2, 4.6197393e-04f);
    p = fmaf(p, z2, -1.0517757e-01f);
    p = fmaf(p, z2, -2.3021175e+00f);
    const float e = fast_exp2(x * p);                                 // exp(-2 x p(x^2))
    return __fdividef(x, 1.0f + e);
}
__device__ __forceinline__ bool elect_one() {
    uint32_t e;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(e));
    return e != 0;
}

// columns of its block an epilogue warp stages at a time: half of a 64-column block, the whole of a 48-column one
template <int CW> struct LgStage { static constexpr int cols = CW == 64 ? 32 : CW; };

// One epilogue warp's share of a tile: 32 accumulator rows (tensor-memory lanes of the warp's subpartition) x CW columns
// starting at tensor-memory address tacc, to y rows row0.. and columns n0.. . bias2: this lane's packed pair of the CW bias
// values (lanes below CW / 2). stage_out: the warp's staging block, 32 rows of LgStage<CW>::cols bf16.
//   16 columns at a time, the next 16 on their way from tensor memory while these are processed: + bias, round to bf16
//   (where the separate Linear would round), GELU in fp32, round; the staged columns then leave as whole row segments
//   (64 or 96 bytes), several rows per store instruction (a thread-per-row store would touch 32 lines per instruction and
//   the load/store unit, not memory, would set the epilogue's pace).
template <int CW>
__device__ __forceinline__ void lg_epilogue_block(uint32_t tacc, uint32_t bias2, uint8_t *stage_out, __nv_bfloat16 *__restrict__ y,
                                                  long long row0, int n0, long long M, int N, int act, int lane) {
    constexpr int SC = LgStage<CW>::cols, NP = SC / 16, RC = SC / 8;   // per staging round: 16-column pieces, 16-byte chunks per row
    // chunk c of row r: with 64-byte rows the chunks are rotated by the row, so that the row-per-lane writes and the
    // chunk-per-lane reads both touch every bank once per 128 bytes; 96-byte rows spread by themselves (two ways at worst)
    auto chunk_at = [&](int r, int c) { return stage_out + r * (2 * SC) + ((SC == 32 ? (c ^ ((r >> 1) & 3)) : c) << 4); };
    float v[2][16];
    tmem_ld16_nowait(tacc, v[0]);
#pragma unroll
    for (int h = 0; h < CW / SC; ++h) {
#pragma unroll
        for (int q = 0; q < NP; ++q) {
            constexpr int TOTAL = CW / 16;
            const int pc = h * NP + q;                                 // piece of the block
            tmem_ld_wait();
            if (pc + 1 < TOTAL) tmem_ld16_nowait(tacc + 16 * (pc + 1), v[(pc + 1) & 1]);
            const float (&a)[16] = v[pc & 1];
#pragma unroll
            for (int g = 0; g < 2; ++g) {                              // 8 columns = one 16-byte chunk
                uint4 outv;
                __nv_bfloat162 *o2 = reinterpret_cast<__nv_bfloat162 *>(&outv);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint32_t braw = __shfl_sync(0xffffffffu, bias2, 8 * pc + 4 * g + i);
                    const float2 bv = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&braw));
                    // the pre-activation, rounded to bf16 as the separate Linear would hand it on
                    const float2 x = __bfloat1622float2(__floats2bfloat162_rn(a[8 * g + 2 * i] + bv.x, a[8 * g + 2 * i + 1] + bv.y));
                    o2[i] = act == 1 ? __floats2bfloat162_rn(lg_gelu(x.x), lg_gelu(x.y)) : __floats2bfloat162_rn(x.x, x.y);
                }
                *reinterpret_cast<uint4 *>(chunk_at(lane, 2 * q + g)) = outv;
            }
        }
        __syncwarp();
        const int col = n0 + SC * h;
#pragma unroll
        for (int k = 0; k < RC; ++k) {
            const int idx = lane + 32 * k, r = idx / RC, c = idx % RC;
            const uint4 val = *reinterpret_cast<const uint4 *>(chunk_at(r, c));
            const long long grow = row0 + r;
            if (grow < M && col + 8 * c < N) *reinterpret_cast<uint4 *>(y + (size_t)grow * N + col + 8 * c) = val;
        }
        __syncwarp();
    }
}

template <int BN, int EPI>
__global__ void __launch_bounds__((2 + EPI) * 32, 1) linear_gelu_kernel(const __grid_constant__ CUtensorMap mx, const __grid_constant__ CUtensorMap mw,
                                                              const __nv_bfloat16 *__restrict__ bias, __nv_bfloat16 *__restrict__ y,
                                                              long long M, int N, int K, int act) {
    using CF = LgCfg<BN, EPI>;
    constexpr int LG_BN = BN, LG_STAGE = CF::STAGE;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t *sm = smem_raw + (base - smem_u32(smem_raw));
    const uint32_t mb = base + LG_STAGES * LG_STAGE;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(sm + LG_STAGES * LG_STAGE + 128);
    auto bar_full = [&](int s) { return mb + 8 * s; };
    auto bar_empty = [&](int s) { return mb + 32 + 8 * s; };
    auto bar_acc_full = [&](int a) { return mb + 64 + 8 * a; };
    auto bar_acc_empty = [&](int a) { return mb + 80 + 8 * a; };

    const int tid = threadIdx.x, lane = tid & 31, warp = warp_uniform(tid >> 5);
    const int tiles_n = (N + LG_BN - 1) / LG_BN;
    const long long tiles = ((M + LG_BM - 1) / LG_BM) * tiles_n;
    const int KB = (K + LG_BK - 1) / LG_BK;

    if (tid == 0) {
        for (int s = 0; s < LG_STAGES; ++s) { mbar_init(bar_full(s), 1); mbar_init(bar_empty(s), 1); }
        for (int a = 0; a < 2; ++a) { mbar_init(bar_acc_full(a), 1); mbar_init(bar_acc_empty(a), EPI); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tmem_alloc(smem_u32(tmem_slot), 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = warp_uniform(*tmem_slot);
    // Launched as a programmatic dependent: the set-up above overlaps the tail of the kernel that produces x.
    pdl_wait();
    pdl_launch_dependents();

    if (warp == 0) {
        // ------------------------------------------------------------------------------------------ producer
        const bool leader = elect_one();
        uint32_t it = 0;
        bool ok = true;
        for (long long t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
            const int m0 = (int)(t / tiles_n) * LG_BM, n0 = (int)(t % tiles_n) * LG_BN;
            for (int kb = 0; kb < KB && ok; ++kb, ++it) {
                const int s = it % LG_STAGES;
                if (it >= LG_STAGES) ok = __all_sync(0xffffffffu, mbar_wait(bar_empty(s), ((it / LG_STAGES) + 1) & 1, 71));
                if (ok && leader) {
                    const uint32_t sa = base + s * LG_STAGE;
                    mbar_expect_tx(bar_full(s), LG_STAGE);
                    tma_load_2d(sa, &mx, bar_full(s), kb * LG_BK, m0);
                    tma_load_2d(sa + LG_A_BYTES, &mw, bar_full(s), kb * LG_BK, n0);
                }
                __syncwarp();
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------------------------------ MMA issuer
        constexpr uint32_t IDESC = idesc_bf16(LG_BM, LG_BN, 0, 0);
        uint32_t it = 0, ti = 0;
        bool ok = true;
        for (long long t = blockIdx.x; t < tiles && ok; t += gridDim.x, ++ti) {
            const uint32_t a = ti & 1;
            if (ti >= 2) ok = __all_sync(0xffffffffu, mbar_wait(bar_acc_empty(a), ((ti >> 1) + 1) & 1, 72));
            tc_fence_after();
            for (int kb = 0; kb < KB && ok; ++kb, ++it) {
                const int s = it % LG_STAGES;
                ok = __all_sync(0xffffffffu, mbar_wait(bar_full(s), (it / LG_STAGES) & 1, 73));
                if (!ok) break;
                tc_fence_after();
                const uint32_t sa = base + s * LG_STAGE;
                const uint64_t da = smem_desc(sa, 16, 1024), db = smem_desc(sa + LG_A_BYTES, 16, 1024);
#pragma unroll
                for (int k = 0; k < LG_BK / 16; ++k) mma_bf16_elect(tmem + a * LG_BN, da + k * 2, db + k * 2, IDESC, (kb | k) != 0);
                mma_commit_elect(bar_empty(s));                       // the stage is free once these MMAs have read it
            }
            if (ok) mma_commit_elect(bar_acc_full(a));
        }
    } else {
        // ------------------------------------------------------------------------------------------ epilogue
        constexpr int CW = CF::CW;                                     // columns per warp: 64 or 48
        const int sub = warp & 3, part = (warp - 2) >> 2;
        const uint32_t lane_base = (uint32_t)(32 * sub) << 16;
        uint8_t *stage_out = sm + LG_STAGES * LG_STAGE + 1024 + (warp - 2) * CF::OUT_BYTES;
        uint32_t ti = 0;
        bool ok = true;
        for (long long t = blockIdx.x; t < tiles && ok; t += gridDim.x, ++ti) {
            const uint32_t a = ti & 1;
            const long long row0 = (t / tiles_n) * LG_BM + 32 * sub;
            const int n0 = (int)(t % tiles_n) * LG_BN + part * CW;
            // this warp's 64 bias values, two per lane, requested before the accumulator is waited for
            uint32_t bias2 = 0u;
            if (bias != nullptr && 2 * lane < CW && n0 + 2 * lane < N) bias2 = *reinterpret_cast<const uint32_t *>(bias + n0 + 2 * lane);
            ok = __all_sync(0xffffffffu, mbar_wait(bar_acc_full(a), (ti >> 1) & 1, 74));
            if (!ok) break;
            tc_fence_after();
            lg_epilogue_block<CW>(tmem + lane_base + a * LG_BN + part * CW, bias2, stage_out, y, row0, n0, M, N, act, lane);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) lg_arrive(bar_acc_empty(a));
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, 512);
}

// ------------------------------------------------------------------------------------------------ the pair kernel
// The same GEMM on pairs of SMs: a cluster of two CTAs computes one 256 x 256 tile with tcgen05.mma.cta_group::2. Each CTA
// loads its own 128 rows of x and its own 128 rows of W per 64-wide K block (32 KiB instead of the 48 KiB a lone CTA
// needs for a 128 x 256 tile), the tensor cores of both SMs read the two halves of W from either CTA's shared memory, and
// each CTA's tensor memory receives its own 128 rows of the tile. A third less operand traffic from the L2 -- what the
// single-CTA kernel is bound by -- and six 32 KiB stages in flight.
//   The CTA of cluster rank 0 issues every MMA. Its full[] barriers count the bytes of both CTAs' loads (each CTA's TMA
//   names rank 0's barrier); a stage is handed back, and an accumulator handed on, by one tcgen05.commit per CTA (the
//   rank-1 barrier through its cluster address); the epilogue warps of both CTAs arrive on rank 0's acc_empty[] barrier.
//   No load is shared between the CTAs, so there is no multicast anywhere. Roles, epilogue and the bounded waits are those
//   of the kernel above; the cluster meets twice more, after set-up and before tensor memory is freed. Results are those
//   of the kernel above to the bit (the same products accumulated in the same order).
constexpr int LP_BM = 256, LP_STAGES = 6;
constexpr int LP_A_BYTES = (LP_BM / 2) * LG_BK * 2;
template <int BN>
struct LpCfg {
    static constexpr int CW = BN / (LG_EPI / 4);
    static constexpr int B_BYTES = (BN / 2) * LG_BK * 2, STAGE = LP_A_BYTES + B_BYTES;
    static constexpr int OUT_BYTES = 32 * (CW == 64 ? 32 : CW) * 2;
    static constexpr int SMEM = LP_STAGES * STAGE + 1024 + LG_EPI * OUT_BYTES + 1024;
    static_assert(BN == 256 || BN == 192, "tile width");
    static_assert(STAGE % 1024 == 0 && SMEM <= 232448, "shared memory of the pair kernel");
};

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// the address, in the cluster's shared window, of this CTA's shared-memory address `addr` in the CTA of rank `rank`
__device__ __forceinline__ uint32_t cluster_addr(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void lp_arrive_cluster(uint32_t cluster_bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
// bounded wait on a barrier of this CTA whose arrivals come from both CTAs of the pair
__device__ __forceinline__ bool lp_wait_cluster(uint32_t bar, uint32_t parity, int code) {
    for (uint32_t n = WAIT_TRIES; n != 0; --n) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n\tselp.b32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok) : "r"(bar), "r"(parity), "r"(WAIT_HINT) : "memory");
        if (ok) return true;
    }
    atomicExch(&g_tc_error, code);
    return false;
}
// this CTA's half of a stage; the bytes are counted on `cluster_bar`, a barrier of the pair's first CTA
__device__ __forceinline__ void lp_tma_load(uint32_t dst, const CUtensorMap *map, uint32_t cluster_bar, int c0, int c1) {
    asm volatile("cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
                 ::"r"(dst), "l"(map), "r"(cluster_bar), "r"(c0), "r"(c1), "r"(0) : "memory");
}
__device__ __forceinline__ void lp_mma_elect(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p, e;\n\telect.sync _|e, 0xffffffff;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "@e tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n\t}"
                 ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0u) : "memory");
}
// one arrival on `cluster_bar` (any CTA of the pair) once every MMA this thread has issued so far is complete
__device__ __forceinline__ void lp_commit_elect(uint32_t cluster_bar) {
    asm volatile("{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\t"
                 "@e tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(cluster_bar) : "memory");
}

template <int BN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(LG_NT, 1)
linear_gelu_pair_kernel(const __grid_constant__ CUtensorMap mx, const __grid_constant__ CUtensorMap mw, const __nv_bfloat16 *__restrict__ bias,
                        __nv_bfloat16 *__restrict__ y, long long M, int N, int K, int act) {
    using CF = LpCfg<BN>;
    constexpr int LP_BN = BN, LP_STAGE = CF::STAGE;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;      // the same offset in both CTAs: one descriptor serves both
    uint8_t *sm = smem_raw + (base - smem_u32(smem_raw));
    const uint32_t mb = base + LP_STAGES * LP_STAGE;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(sm + LP_STAGES * LP_STAGE + 256);
    auto bar_full = [&](int s) { return mb + 8 * s; };                 // used in the first CTA only
    auto bar_empty = [&](int s) { return mb + 64 + 8 * s; };
    auto bar_acc_full = [&](int a) { return mb + 128 + 8 * a; };
    auto bar_acc_empty = [&](int a) { return mb + 144 + 8 * a; };      // used in the first CTA only

    const int tid = threadIdx.x, lane = tid & 31, warp = warp_uniform(tid >> 5);
    const uint32_t rank = cluster_rank();
    const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    const int tiles_n = (N + LP_BN - 1) / LP_BN;
    const long long tiles = ((M + LP_BM - 1) / LP_BM) * tiles_n;
    const int KB = (K + LG_BK - 1) / LG_BK;

    if (tid == 0) {
        for (int s = 0; s < LP_STAGES; ++s) { mbar_init(bar_full(s), 1); mbar_init(bar_empty(s), 1); }
        for (int a = 0; a < 2; ++a) { mbar_init(bar_acc_full(a), 1); mbar_init(bar_acc_empty(a), 2 * LG_EPI); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {                                                   // the same warp of both CTAs, the same slot address
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();                                                // the partner's barriers and tensor memory exist from here on
    tc_fence_after();
    const uint32_t tmem = warp_uniform(*tmem_slot);
    pdl_wait();
    pdl_launch_dependents();

    if (warp == 0) {
        // ------------------------------------------------------------------------------------------ producer (both CTAs)
        const bool leader = elect_one();
        uint32_t it = 0;
        bool ok = true;
        for (long long t = pair; t < tiles && ok; t += pairs) {
            const int m0 = (int)(t / tiles_n) * LP_BM + (int)rank * (LP_BM / 2), n0 = (int)(t % tiles_n) * LP_BN + (int)rank * (LP_BN / 2);
            for (int kb = 0; kb < KB && ok; ++kb, ++it) {
                const int s = it % LP_STAGES;
                if (it >= LP_STAGES) ok = __all_sync(0xffffffffu, mbar_wait(bar_empty(s), ((it / LP_STAGES) + 1) & 1, 75));
                if (ok && leader) {
                    const uint32_t sa = base + s * LP_STAGE, full0 = cluster_addr(bar_full(s), 0);
                    if (rank == 0) mbar_expect_tx(bar_full(s), 2 * LP_STAGE);      // both CTAs' bytes
                    lp_tma_load(sa, &mx, full0, kb * LG_BK, m0);
                    lp_tma_load(sa + LP_A_BYTES, &mw, full0, kb * LG_BK, n0);
                }
                __syncwarp();
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------------------------------ MMA issuer (first CTA)
        if (rank == 0) {
            constexpr uint32_t IDESC = idesc_bf16(LP_BM, LP_BN, 0, 0);
            uint32_t it = 0, ti = 0;
            bool ok = true;
            for (long long t = pair; t < tiles && ok; t += pairs, ++ti) {
                const uint32_t a = ti & 1;
                if (ti >= 2) ok = __all_sync(0xffffffffu, lp_wait_cluster(bar_acc_empty(a), ((ti >> 1) + 1) & 1, 76));
                tc_fence_after();
                for (int kb = 0; kb < KB && ok; ++kb, ++it) {
                    const int s = it % LP_STAGES;
                    ok = __all_sync(0xffffffffu, lp_wait_cluster(bar_full(s), (it / LP_STAGES) & 1, 77));
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t sa = base + s * LP_STAGE;
                    const uint64_t da = smem_desc(sa, 16, 1024), db = smem_desc(sa + LP_A_BYTES, 16, 1024);
#pragma unroll
                    for (int k = 0; k < LG_BK / 16; ++k) lp_mma_elect(tmem + a * LP_BN, da + k * 2, db + k * 2, IDESC, (kb | k) != 0);
                    lp_commit_elect(bar_empty(s));                     // the stage is free in both CTAs once these MMAs have read it
                    lp_commit_elect(cluster_addr(bar_empty(s), 1));
                }
                if (ok) {
                    lp_commit_elect(bar_acc_full(a));
                    lp_commit_elect(cluster_addr(bar_acc_full(a), 1));
                }
            }
        }
    } else {
        // ------------------------------------------------------------------------------------------ epilogue (both CTAs)
        constexpr int CW = CF::CW;
        const int sub = warp & 3, part = (warp - 2) >> 2;
        const uint32_t lane_base = (uint32_t)(32 * sub) << 16;
        uint8_t *stage_out = sm + LP_STAGES * LP_STAGE + 1024 + (warp - 2) * CF::OUT_BYTES;
        uint32_t ti = 0;
        bool ok = true;
        for (long long t = pair; t < tiles && ok; t += pairs, ++ti) {
            const uint32_t a = ti & 1;
            const long long row0 = (t / tiles_n) * LP_BM + (long long)rank * (LP_BM / 2) + 32 * sub;
            const int n0 = (int)(t % tiles_n) * LP_BN + part * CW;
            uint32_t bias2 = 0u;
            if (bias != nullptr && 2 * lane < CW && n0 + 2 * lane < N) bias2 = *reinterpret_cast<const uint32_t *>(bias + n0 + 2 * lane);
            ok = __all_sync(0xffffffffu, mbar_wait(bar_acc_full(a), (ti >> 1) & 1, 78));
            if (!ok) break;
            tc_fence_after();
            lg_epilogue_block<CW>(tmem + lane_base + a * LP_BN + part * CW, bias2, stage_out, y, row0, n0, M, N, act, lane);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) lp_arrive_cluster(cluster_addr(bar_acc_empty(a), 0));
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();                                                // neither CTA frees tensor memory the other's MMAs may still write
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
}

// 0: one CTA per 128 x BN tile; 1: the pair kernel whenever the problem has more than one 128-row block. Timed at the MLP's
// shape (M 8192, K 768, N 3072; launches back to back over rotating buffers) with 256-wide tiles, the pair is ahead without
// an activation (34.8 vs 36.7 us) and behind with the GELU (40.7 vs 39.7 us): once the pair has made the mainloop cheaper,
// the epilogue -- unchanged, and as long as the mainloop -- is what a tile waits for. The model's only use is the one with
// the GELU, so the single-CTA kernel stays the default.
// Bits 1-2 pick the tile width (0 or 1: 256, 2: 192) for timing and tests.
static int g_lg_variant = 0;
int linear_gelu_variant() { return g_lg_variant; }
int linear_gelu_set_variant(int v) {
    if (v < 0 || v > 5 || (v >> 1) > 2) return PGB_ERR_BAD_SHAPE;
    g_lg_variant = v;
    return PGB_OK;
}

// clusters of two CTAs of the pair kernel that can be resident at once (cached per device); 0 if the query fails
template <int BN>
static int lp_resident_pairs(int dev) {
    static int cached[64];
    static bool have[64];
    if (dev >= 0 && dev < 64 && have[dev]) return cached[dev];
    int n = 0, sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(sms > 1 ? sms & ~1 : 2)); cfg.blockDim = dim3(LG_NT); cfg.dynamicSmemBytes = LpCfg<BN>::SMEM;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    cfg.attrs = at; cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&n, linear_gelu_pair_kernel<BN>, &cfg) != cudaSuccess) { cudaGetLastError(); n = 0; }
    if (dev >= 0 && dev < 64) { cached[dev] = n; have[dev] = true; }
    return n;
}

template <int BN, int EPI>
static int lg_launch_single(const void *x, const void *W, const void *bias, void *y, long long M, int N, int K, int act, int sms,
                            cudaStream_t stream) {
    CUtensorMap mx, mw;
    if (!tc_make_map(&mx, x, 1, M, K, K, (long long)M * K, LG_BM) || !tc_make_map(&mw, W, 1, N, K, K, (long long)N * K, BN)) {
        set_cuda_error(cudaErrorUnknown, "cuTensorMapEncodeTiled");
        return PGB_ERR_CUDA;
    }
    const long long tiles = ((M + LG_BM - 1) / LG_BM) * ((N + BN - 1) / BN);
    const unsigned grid = (unsigned)(tiles < sms ? tiles : sms);
    cudaError_t e = cudaFuncSetAttribute(linear_gelu_kernel<BN, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, LgCfg<BN, EPI>::SMEM);
    if (e != cudaSuccess) { set_cuda_error(e, "linear_gelu smem attribute"); return PGB_ERR_CUDA; }
    e = pdl_launch(linear_gelu_kernel<BN, EPI>, dim3(grid), dim3(LgCfg<BN, EPI>::NT), (size_t)LgCfg<BN, EPI>::SMEM, stream, mx, mw, (const __nv_bfloat16 *)bias,
                   (__nv_bfloat16 *)y, M, N, K, act);
    if (e != cudaSuccess) { set_cuda_error(e, "linear_gelu launch"); return PGB_ERR_CUDA; }
    return check_launch("linear_gelu_kernel");
}

template <int BN>
static int lg_launch_pair(const void *x, const void *W, const void *bias, void *y, long long M, int N, int K, int act, int room,
                          cudaStream_t stream) {
    CUtensorMap mx, mw;
    if (!tc_make_map(&mx, x, 1, M, K, K, (long long)M * K, LP_BM / 2) || !tc_make_map(&mw, W, 1, N, K, K, (long long)N * K, BN / 2)) {
        set_cuda_error(cudaErrorUnknown, "cuTensorMapEncodeTiled");
        return PGB_ERR_CUDA;
    }
    const long long tiles = ((M + LP_BM - 1) / LP_BM) * ((N + BN - 1) / BN);
    const unsigned pairs = (unsigned)(tiles < room ? tiles : room);
    cudaError_t e = pdl_launch(linear_gelu_pair_kernel<BN>, dim3(2 * pairs), dim3(LG_NT), (size_t)LpCfg<BN>::SMEM, stream, mx, mw,
                               (const __nv_bfloat16 *)bias, (__nv_bfloat16 *)y, M, N, K, act);
    if (e != cudaSuccess) { set_cuda_error(e, "linear_gelu pair launch"); return PGB_ERR_CUDA; }
    return check_launch("linear_gelu_pair_kernel");
}

int linear_gelu_launch(const void *x, const void *W, const void *bias, void *y, long long M, int N, int K, int act, cudaStream_t stream) {
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int pin = g_lg_variant >> 1;                                 // 2: tiles 192 columns wide
    if ((g_lg_variant & 1) && M > LG_BM) {
        cudaError_t e = cudaFuncSetAttribute(linear_gelu_pair_kernel<256>, cudaFuncAttributeMaxDynamicSharedMemorySize, LpCfg<256>::SMEM);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(linear_gelu_pair_kernel<192>, cudaFuncAttributeMaxDynamicSharedMemorySize, LpCfg<192>::SMEM);
        if (e != cudaSuccess) { set_cuda_error(e, "linear_gelu pair smem attribute"); return PGB_ERR_CUDA; }
        const int r256 = lp_resident_pairs<256>(dev), r192 = lp_resident_pairs<192>(dev);
        if (r256 > 0 && r192 > 0) {
            if (pin == 2) return lg_launch_pair<192>(x, W, bias, y, M, N, K, act, r192, stream);
            return lg_launch_pair<256>(x, W, bias, y, M, N, K, act, r256, stream);
        }
    }
    if (pin == 2) return lg_launch_single<192, LG_EPI>(x, W, bias, y, M, N, K, act, sms, stream);
    return lg_launch_single<256, LG_EPI>(x, W, bias, y, M, N, K, act, sms, stream);
}

int linear_gelu_error_flag(int *out) { return tc_read_error_flag(out); }

}  // namespace pgb
