// y = act(norm(x) W^T + bias) [+ residual] for one token of up to 64 sequences: the linear layers of a batch's decode step, each with what
// stands around it in one launch, as links of a chain of programmatic dependents.
//
// Such a layer reads its weight once (a few MB) and multiplies next to nothing, so it costs its latency: the kernel ahead, x from the L2, the
// sums, the way out. This kernel keeps all else off that path:
//   * The weights, which no kernel ahead writes, are requested before the wait on the kernel ahead. A CTA is small (its share of x and W at
//     once, 50 to 110 KB up to d 960, and 64 columns of tensor memory), so that it is resident, set up and holding its weights while the kernel ahead still runs.
//   * K is cut over a cluster of S CTAs, so that x (64 rows, all of K) is read once a cluster and not once a CTA: of 64 rows by K 768 a CTA's whole
//     share would be 98 KB, 3 us from the L2. The sums meet by rows: CTA r of the cluster gets its 64 / S rows from all S (st.async into its shared
//     memory, counted by its barrier), adds them in rank order and finishes them.
//   * The RMS norm ahead of a layer costs neither a launch nor a pass: the layer that produced the residual stream x also leaves x w (w the norm's
//     weight; rounded once, as the normalised row would be) and each row's sum of squares by tiles; here x w is multiplied, and the row's
//     1 / rms applied to the fp32 sum.
//
// A token of 12 layers of 768 (graph replay): batch 64 421 -> 317 us, batch 16 383 -> 240, batch 5 372 -> 224, against the library's products with
// separate norms. What bounds it now is the chain, 62 links a token. Linear links that leave early, each variant doing what the one ahead of it does and one thing more, us a
// token at batch 5 / 64: behind the wait on the kernel ahead 143 / 220 (the state steps in full), x landed 147 / 216, products and row sums done 150 / 228, sums exchanged
// 186 / 278, all 227 / 318. So of the 3.6 us a link at batch 5 the launch and the wait are 2.3; the exchange is 0.7 of a linear link and the way out 0.9. Only the batch's rows of x
// are fetched: all 64 took 0.4 a link more. An L2 prefetch of the weights two links ahead gave nothing, one barrier for all blocks of K instead of
// one each 0.4 more a link, two issuing warps 0.2 more.
//
// x [B][K] bf16 is the K-major A operand (64 rows; those past the batch are zero or whatever shared memory holds, each its own row's only), W [N][K] the B operand. Replaces, for T = 1, F.linear with the
// norm, GELU and residual add around it (src/assoc.py:384-512, src/model.py:552-560). Every wait is bounded; one that runs out sets the error flag, and
// the cluster winds down together.
#include "tc_common.cuh"

namespace pgb {

constexpr int DL_NT = 256, DL_ROWS = 64;
constexpr int DL_KB = 16;                                             // K blocks (of 64) of a CTA at most
constexpr int DL_SMEM_MOST = 224 * 1024, DL_SMEM_FIRST = 200 * 1024;

struct DlArgs {
    const __nv_bfloat16 *bias;
    const float *sums; int parts; float eps;                          // [B][parts] sums of squares of the row behind x (NULL: no norm)
    const __nv_bfloat16 *resid, *next_w;                              // residual stream to add to [B][N]; weight of the norm behind it [N]
    __nv_bfloat16 *y, *yw; float *logits, *sums_out;                  // y [B][N], or logits in fp32; with resid: y next_w and [B][tiles] sums of squares
    long long *pos; float *shift; int window;                         // the last layer of a token: the next one's position and shift
    int B, N, K, act, xrows;                                          // xrows: rows of x fetched, the batch rounded up
};

template <int BN> __host__ __device__ constexpr int dl_block() { return DL_ROWS * 128 + BN * 128; }      // bytes of a K block: 64 rows of x, BN of W
template <int BN> __host__ __device__ constexpr int dl_parts() { return DL_ROWS * (BN + 4) * 4; }

__device__ __forceinline__ uint32_t dl_mapa(uint32_t addr, int rank) {
    uint32_t at;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(addr), "r"(rank));
    return at;
}
__device__ __forceinline__ void dl_send4(uint32_t at, uint32_t bar, float a, float b, float c, float d) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];"
                 ::"r"(at), "f"(a), "f"(b), "f"(c), "f"(d), "r"(bar) : "memory");
}
__device__ __forceinline__ void dl_tmem_ld8(uint32_t taddr, float (&v)[8]) {
    uint32_t *r = reinterpret_cast<uint32_t *>(v);
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
}

template <int BN, int S>
__global__ void __launch_bounds__(DL_NT) decode_linear_kernel(const __grid_constant__ CUtensorMap mx, const __grid_constant__ CUtensorMap mw,
                                                             const __grid_constant__ DlArgs a) {
    constexpr int RR = DL_ROWS / S, PROW = BN + 4, G4 = BN / 4;       // rows a CTA finishes; padded row of the sums; groups of four columns
    constexpr int GL = G4 <= 4 ? 4 : (G4 <= 8 ? 8 : (G4 <= 16 ? 16 : 32));              // lanes of a row behind the sums: one a group, rounded up to a power of two
    constexpr int TCOLS = BN <= 32 ? 32 : (BN <= 64 ? 64 : 128);
    extern __shared__ uint8_t dl_smem[];
    __shared__ __align__(8) unsigned long long bars[DL_KB + 2];
    __shared__ uint32_t tmem_slot;
    __shared__ float rstd[RR];
    const uint32_t base = (smem_u32(dl_smem) + 1023u) & ~1023u;
    uint8_t *sm = dl_smem + (base - smem_u32(dl_smem));
    const int tid = threadIdx.x, lane = tid & 31, warp = warp_uniform(tid >> 5);
    const int rank = blockIdx.x % S, tile = blockIdx.x / S, n0 = tile * BN;
    const int KBa = (a.K + 63) >> 6, kb0 = KBa * rank / S, nk = KBa * (rank + 1) / S - kb0;
    const uint32_t bar = smem_u32(bars), bar_acc = bar + 8 * DL_KB, bar_p = bar_acc + 8;
    const uint32_t ws = base + nk * (DL_ROWS * 128), parts = base + (KBa + S - 1) / S * dl_block<BN>();   // the sums: at the same place in every CTA
    const bool live = rank * RR < a.B;                                // this CTA finishes rows

    if (warp == 0) {
        if (lane == 29) asm volatile("prefetch.tensormap [%0];" ::"l"(&mx) : "memory");       // used behind the wait only
        if (lane < nk) mbar_init(bar + 8 * lane, 1);
        if (lane == 30) mbar_init(bar_acc, 1);
        if (lane == 31) mbar_init(bar_p, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        __syncwarp();
        if (lane == 0)
            for (int i = 0; i < nk; ++i) {
                mbar_expect_tx(bar + 8 * i, (a.xrows + BN) * 128);
                tma_load_3d(ws + i * (BN * 128), &mw, bar + 8 * i, (kb0 + i) * 64, n0, 0);
            }
        if (lane == 1 && live) mbar_expect_tx(bar_p, S * RR * BN * 4);
    }
    if (warp == 1) tmem_alloc(smem_u32(&tmem_slot), TCOLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = warp_uniform(tmem_slot);
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");          // this CTA's barriers are set up ...
    pdl_launch_dependents();
    // this thread's outputs: four columns of a row
    constexpr int NG = (RR * GL + DL_NT - 1) / DL_NT;
    uint2 braw[NG], rraw[NG], wraw[NG];
#pragma unroll
    for (int j = 0; j < NG; ++j) {
        const int g = tid + j * DL_NT, col = n0 + 4 * (g % GL);
        braw[j] = wraw[j] = rraw[j] = make_uint2(0u, 0u);
        if (g < RR * GL && g % GL < G4 && col < a.N) {
            if (a.bias != nullptr) braw[j] = *reinterpret_cast<const uint2 *>(a.bias + col);
            if (a.resid != nullptr) wraw[j] = *reinterpret_cast<const uint2 *>(a.next_w + col);
        }
    }
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");            // ... and its peers', before anything is sent to them
    pdl_wait();                                                       // x, its sums and the residual are the work of kernels ahead
    bool ok = true;
    if (warp == 0) {
        if (lane == 0)
            for (int i = 0; i < nk; ++i) tma_load_3d(base + i * (DL_ROWS * 128), &mx, bar + 8 * i, (kb0 + i) * 64, 0, 0);
        __syncwarp();
    } else if (warp == 1) {
        constexpr uint32_t IDESC = idesc_bf16(DL_ROWS, BN, 0, 0);
        for (int i = 0; i < nk && ok; ++i) {
            ok = mbar_wait_warp(bar + 8 * i, 0, 78);
            tc_fence_after();
            const uint64_t da = smem_desc(base + i * (DL_ROWS * 128), 16, 1024), db = smem_desc(ws + i * (BN * 128), 16, 1024);
#pragma unroll
            for (int k = 0; k < 4; ++k) mma_bf16_elect(tmem, da + k * 2, db + k * 2, IDESC, i != 0 || k != 0 ? 1u : 0u);
        }
        mma_commit_elect(bar_acc);
    } else if (a.sums != nullptr) {
        // 1 / rms of this CTA's rows, eight lanes a row, the tiles' sums in a fixed order
        for (int r = (warp - 2) * 4 + (lane >> 3); r < RR; r += 24) {
            float t = 0.f;
            if (rank * RR + r < a.B)
                for (int p = lane & 7; p < a.parts; p += 8) t += a.sums[(size_t)(rank * RR + r) * a.parts + p];
            t += __shfl_xor_sync(0xffffffffu, t, 1);
            t += __shfl_xor_sync(0xffffffffu, t, 2);
            t += __shfl_xor_sync(0xffffffffu, t, 4);
            if ((lane & 7) == 0) rstd[r] = rsqrtf(t / (float)a.K + a.eps);
        }
    }
    if (a.resid != nullptr)
#pragma unroll
        for (int j = 0; j < NG; ++j) {
            const int g = tid + j * DL_NT, col = n0 + 4 * (g % GL), row = rank * RR + g / GL;
            if (g < RR * GL && g % GL < G4 && col < a.N && row < a.B) rraw[j] = *reinterpret_cast<const uint2 *>(a.resid + (size_t)row * a.N + col);
        }
    if (!mbar_wait(bar_acc, 0, 78)) ok = false;
    tc_fence_after();
    // each quarter of the tensor-memory lanes holds 16 rows in its first 16 lanes
    {
        const int row = 16 * (warp & 3) + lane, to = row / RR;
        if (16 * (warp & 3) / RR * RR < a.B) {                        // all rows of a CTA that finishes any
            float v[(BN / 8 + 1) / 2][8];
#pragma unroll
            for (int j = 0; j < (BN / 8 + 1) / 2; ++j)
                if ((warp >> 2) + 2 * j < BN / 8) dl_tmem_ld8(tmem + ((uint32_t)(32 * (warp & 3)) << 16) + 8 * ((warp >> 2) + 2 * j), v[j]);
            tmem_ld_wait();
            if (lane < 16 && to * RR < a.B) {
                const uint32_t at = dl_mapa(parts, to) + ((rank * RR + row % RR) * PROW + 8 * (warp >> 2)) * 4, tobar = dl_mapa(bar_p, to);
#pragma unroll
                for (int j = 0; j < (BN / 8 + 1) / 2; ++j)
                    if ((warp >> 2) + 2 * j < BN / 8) {
                        dl_send4(at + 64 * j, tobar, v[j][0], v[j][1], v[j][2], v[j][3]);
                        dl_send4(at + 64 * j + 16, tobar, v[j][4], v[j][5], v[j][6], v[j][7]);
                    }
            }
        }
    }
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    if (live && !mbar_wait(bar_p, 0, 79)) ok = false;
    tc_fence_before();
    ok = __syncthreads_and(ok);                                       // the rows' factors, too
    if (ok && live) {
#pragma unroll
        for (int j = 0; j < NG; ++j) {
            const int g = tid + j * DL_NT, lr = g / GL, col = n0 + 4 * (g % GL), row = rank * RR + lr;
            const bool in = g < RR * GL && g % GL < G4 && row < a.B && col < a.N;
            float v[4] = {0.f, 0.f, 0.f, 0.f}, sq = 0.f;
            if (in) {
                const float *pp = reinterpret_cast<const float *>(sm + (parts - base)) + lr * PROW + 4 * (g % GL);
#pragma unroll
                for (int r = 0; r < S; ++r) {
                    const float4 t = *reinterpret_cast<const float4 *>(pp + r * RR * PROW);
                    v[0] += t.x; v[1] += t.y; v[2] += t.z; v[3] += t.w;
                }
                const __nv_bfloat162 *b2 = reinterpret_cast<const __nv_bfloat162 *>(&braw[j]);
                const float2 b01 = __bfloat1622float2(b2[0]), b23 = __bfloat1622float2(b2[1]);
                const float bb[4] = {b01.x, b01.y, b23.x, b23.y}, rs = a.sums != nullptr ? rstd[lr] : 1.f;
                // rounded to bf16 where the separate Linear would hand its result on
#pragma unroll
                for (int i = 0; i < 4; ++i) v[i] = __bfloat162float(__float2bfloat16_rn(fmaf(rs, v[i], bb[i])));
                if (a.logits != nullptr) {
                    *reinterpret_cast<float4 *>(a.logits + (size_t)row * a.N + col) = make_float4(v[0], v[1], v[2], v[3]);
                } else {
                    if (a.act == 1)
#pragma unroll
                        for (int i = 0; i < 4; ++i) v[i] = 0.5f * v[i] * (1.0f + erff(v[i] * 0.70710678118654752f));
                    if (a.resid != nullptr) {
                        const __nv_bfloat162 *r2 = reinterpret_cast<const __nv_bfloat162 *>(&rraw[j]), *w2 = reinterpret_cast<const __nv_bfloat162 *>(&wraw[j]);
                        const float2 r01 = __bfloat1622float2(r2[0]), r23 = __bfloat1622float2(r2[1]), w01 = __bfloat1622float2(w2[0]), w23 = __bfloat1622float2(w2[1]);
                        const float rr[4] = {r01.x, r01.y, r23.x, r23.y}, ww[4] = {w01.x, w01.y, w23.x, w23.y};
                        float z[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            v[i] = __bfloat162float(__float2bfloat16_rn(v[i] + rr[i]));
                            sq = fmaf(v[i], v[i], sq);
                            z[i] = v[i] * ww[i];
                        }
                        uint2 o;
                        __nv_bfloat162 *o2 = reinterpret_cast<__nv_bfloat162 *>(&o);
                        o2[0] = __floats2bfloat162_rn(z[0], z[1]); o2[1] = __floats2bfloat162_rn(z[2], z[3]);
                        *reinterpret_cast<uint2 *>(a.yw + (size_t)row * a.N + col) = o;
                    }
                    uint2 o;
                    __nv_bfloat162 *o2 = reinterpret_cast<__nv_bfloat162 *>(&o);
                    o2[0] = __floats2bfloat162_rn(v[0], v[1]); o2[1] = __floats2bfloat162_rn(v[2], v[3]);
                    *reinterpret_cast<uint2 *>(a.y + (size_t)row * a.N + col) = o;
                }
            }
            if (a.sums_out != nullptr && g - lane < RR * GL) {
#pragma unroll
                for (int o = 1; o < GL; o <<= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
                if (in && g % GL == 0) a.sums_out[(size_t)row * (gridDim.x / S) + tile] = sq;
            }
        }
    }
    if (a.window > 0 && blockIdx.x == 0 && tid == 0) {
        a.pos[0] = (a.pos[0] + 1) % a.window;
        a.shift[0] = 1.f;
    }
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");            // everyone has its sums or has given them up: long past where all is well
    if (!ok) __nanosleep(50000);                             // what a peer sent late has landed
    if (warp == 1) tmem_dealloc(tmem, TCOLS);
}

// ------------------------------------------------------------------------------------------------ host
template <int BN, int S>
static int decode_linear_go(const void *x, const void *W, const DlArgs &a, cudaStream_t stream) {
    CUtensorMap mx, mw;
    if (!tc_make_map(&mx, x, 1, a.B, a.K, a.K, (long long)a.B * a.K, a.xrows) || !tc_make_map(&mw, W, 1, a.N, a.K, a.K, (long long)a.N * a.K, BN)) {
        set_cuda_error(cudaErrorUnknown, "cuTensorMapEncodeTiled");
        return PGB_ERR_CUDA;
    }
    const int nk = ((a.K + 63) / 64 + S - 1) / S, smem = nk * dl_block<BN>() + dl_parts<BN>() + 1024;
    cudaError_t e = cudaFuncSetAttribute(decode_linear_kernel<BN, S>, cudaFuncAttributeMaxDynamicSharedMemorySize, DL_SMEM_MOST);
    if (e != cudaSuccess) { set_cuda_error(e, "decode_linear smem attribute"); return PGB_ERR_CUDA; }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((a.N + BN - 1) / BN * S)); cfg.blockDim = dim3(DL_NT); cfg.dynamicSmemBytes = smem; cfg.stream = stream;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization; at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension; at[1].val.clusterDim.x = S; at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
    cfg.attrs = at; cfg.numAttrs = 2;
    e = cudaLaunchKernelEx(&cfg, decode_linear_kernel<BN, S>, mx, mw, a);
    if (e != cudaSuccess) { set_cuda_error(e, "decode_linear launch"); return PGB_ERR_CUDA; }
    return check_launch("decode_linear_kernel");
}

struct DlForm { int bn, s; };
static int dl_bytes(DlForm f, int kb) { return (kb + f.s - 1) / f.s * (DL_ROWS + f.bn) * 128 + DL_ROWS * (f.bn + 4) * 4 + 1024; }
static bool dl_fits(DlForm f, int kb, int most) { return (kb + f.s - 1) / f.s <= DL_KB && dl_bytes(f, kb) <= most; }
// in how many rounds a link's clusters go over the chip: what cudaOccupancyMaxActiveClusters says of 148 SMs at 1, 2, 3, 4 CTAs of this memory an SM
static int dl_rounds(DlForm f, int N, int kb) {
    constexpr int ACTIVE[3][4] = {{74, 148, 222, 296}, {33, 71, 104, 142}, {15, 33, 48, 71}};
    const int per_sm = 233472 / (dl_bytes(f, kb) + 1024 + 512);        // the system's own, and the static share
    const int fit = ACTIVE[f.s == 2 ? 0 : (f.s == 4 ? 1 : 2)][per_sm < 1 ? 0 : (per_sm > 4 ? 3 : per_sm - 1)];
    return ((N + f.bn - 1) / f.bn + fit - 1) / fit;
}
// Columns of a tile and CTAs of a cluster. kind 0: plain or activation, 1: residual, 2: logits. {0, 0}: K too short or too long, at whatever batch and N.
// Two things pull: x is read once a tile (wide tiles, few clusters), and CTAs of neighbouring links must fit an SM together, at best one of each (about
// 100 to 130 CTAs of 80 to 100 KB a link). Batch 64, d 768, dff 3072, us a token, all else equal: projection 48,2 335 (32,2 345, 64,4 341, 16,1 333
// but 276 against 275 at batch 16); output projection 32,4 312 (16,4 344, 32,2 318, 16,1 326); MLP up 48,2 331 (32,2 344, 32,4 347, 64,2 349); MLP
// down 32,8 344 (32,4 350, 16,8 379, 48,8 2 % slower; but at batch 5 223 against 239, at 16 240 against 245, at 32 271 against 276); head the same in
// every form.
// Every CTA keeps at least two blocks of K; shorter K is not taken. The wider tiles of few rows hold K up to 6656, the others up to 7680 in MLP down:
// where the wider do not fit the others are taken, so that whether a layer is taken does not depend on the batch.
static DlForm decode_linear_first_form(int kind, int kb, int B) {
    DlForm f;
    if (kb < 4) return DlForm{0, 0};
    if (kind == 1) f = kb >= 32 ? (B <= 32 && dl_fits(DlForm{48, 8}, kb, DL_SMEM_FIRST) ? DlForm{48, 8} : DlForm{32, 8}) : (kb >= 8 ? DlForm{32, 4} : DlForm{16, 2});
    else f = kind == 2 ? DlForm{64, 2} : DlForm{48, 2};
    while (f.s < 8 && !dl_fits(f, kb, DL_SMEM_FIRST)) f.s *= 2;
    return dl_fits(f, kb, DL_SMEM_FIRST) ? f : DlForm{0, 0};
}
// That is for links of one round. In wider models it takes two to four, and a link's time follows their number (d 2048, batch 16, projection: 633 us a token in two,
// 676 in three, 725 in four): where another form needs fewer, the one with the fewest is taken, of those the smallest cluster, then the least shared memory. The head
// stays: its many rounds go at the memory's rate. Twelve layers, us a token, the first forms / these / the separate kernels:
//   d 1024, dff 4096: batch 16 373 / 296 / 435, batch 64 456 / 406 / 485      d 1536, dff 6144: 569 / 475 / 684, 806 / 627 / 758
//   d 1792, dff 7168: 711 / 653 / 775, 904 / 843 / 874                        d 2048, dff 4096: 722 / 577 / 716, 962 / 759 / 834
static DlForm decode_linear_form(int kind, int N, int K, int B) {
    const int kb = (K + 63) / 64;
    DlForm f = decode_linear_first_form(kind, kb, B);
    if (f.bn == 0 || kind == 2) return f;
    int rounds = dl_rounds(f, N, kb);
    bool first = true;
    for (DlForm c : {DlForm{32, 4}, DlForm{32, 8}, DlForm{48, 2}, DlForm{48, 4}, DlForm{48, 8}, DlForm{64, 2}, DlForm{64, 4}, DlForm{64, 8}, DlForm{96, 4}, DlForm{96, 8}}) {
        if (kb < 2 * c.s || !dl_fits(c, kb, DL_SMEM_MOST)) continue;
        const int r = dl_rounds(c, N, kb);
        if (r > rounds || (r == rounds && (first || c.s > f.s || (c.s == f.s && dl_bytes(c, kb) >= dl_bytes(f, kb))))) continue;
        f = c; rounds = r; first = false;
    }
    return f;
}
// tiles (= sums of squares a row) of a residual layer; 0: not taken
int decode_linear_parts(int N, int K, int B) {
    const DlForm f = decode_linear_form(1, N, K, B);
    return f.bn == 0 ? 0 : (N + f.bn - 1) / f.bn;
}
int decode_linear_rounds(int kind, int N, int K, int B) {
    const DlForm f = decode_linear_form(kind, N, K, B);
    return f.bn == 0 ? 0 : dl_rounds(f, N, (K + 63) / 64);
}
bool decode_linear_takes(int kind, int K) { return decode_linear_first_form(kind, (K + 63) / 64, DL_ROWS).bn != 0; }   // at every batch and N

int decode_linear_launch(const void *x, const void *W, const void *bias, const float *sums, int parts, float eps, int act, const void *resid,
                         const void *next_w, void *y, void *yw, float *sums_out, float *logits, long long *pos, float *shift, int window, int B, int N,
                         int K, cudaStream_t stream) {
    const DlArgs a{(const __nv_bfloat16 *)bias, sums, parts, eps, (const __nv_bfloat16 *)resid, (const __nv_bfloat16 *)next_w, (__nv_bfloat16 *)y,
                   (__nv_bfloat16 *)yw, logits, sums_out, pos, shift, window, B, N, K, act, (B + 7) / 8 * 8};
    const DlForm f = decode_linear_form(resid != nullptr ? 1 : (logits != nullptr ? 2 : 0), N, K, B);
#define PGB_DL(BN_, S_) if (f.bn == BN_ && f.s == S_) return decode_linear_go<BN_, S_>(x, W, a, stream)
    PGB_DL(16, 2); PGB_DL(32, 4); PGB_DL(32, 8);
    PGB_DL(48, 2); PGB_DL(48, 4); PGB_DL(48, 8);
    PGB_DL(64, 2); PGB_DL(64, 4); PGB_DL(64, 8);
    PGB_DL(96, 4); PGB_DL(96, 8);
#undef PGB_DL
    return PGB_ERR_TOO_LARGE;
}

int decode_linear_error_flag(int *out) { return tc_read_error_flag(out); }

}  // namespace pgb
