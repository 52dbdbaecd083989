// Device helpers shared by the tensor-core kernels: mbarrier / TMA / tcgen05 PTX wrappers, shared-memory and
// instruction descriptors, the 128-byte swizzle, bf16 head/tail splitting. sm_100a only.
#pragma once
#include <cuda.h>

#include "common.cuh"

namespace pgb {

constexpr int TC_C = 64;

// Set (to the code of the wait) when a bounded mbarrier wait inside a tensor-core kernel runs out. One copy per
// translation unit (no relocatable device code in this build); each unit exports a reader, the C ABI takes the maximum.
static __device__ int g_tc_error = 0;

// reads and clears this translation unit's flag; synchronises the device
static inline int tc_read_error_flag(int *out) {
    int zero = 0;
    cudaError_t e = cudaMemcpyFromSymbol(out, g_tc_error, sizeof(int));
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_tc_error, &zero, sizeof(int));
    if (e != cudaSuccess) { set_cuda_error(e, "tc_error_flag"); return PGB_ERR_CUDA; }
    return PGB_OK;
}

// ---- host: tiled tensor maps through the driver entry point (no link-time dependency on libcuda)
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                  const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static inline EncodeTiledFn tc_encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (fn == nullptr) {
        void *sym = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(sym);
    }
    return fn;
}

// A thread that has done no CUDA work yet (an autograd worker on its first backward, a server's new thread) has no context
// current, which the encoding wants although the runtime's calls do without: bind the current device's and try once more.
static inline bool tc_encode_map(CUtensorMap *m, CUtensorMapDataType type, const void *ptr, const cuuint64_t *dims, const cuuint64_t *strides,
                                 const cuuint32_t *box, CUtensorMapSwizzle swizzle, CUtensorMapL2promotion promotion) {
    EncodeTiledFn fn = tc_encode_fn();
    if (fn == nullptr) return false;
    const cuuint32_t estr[3] = {1, 1, 1};
    auto encode = [&]() {
        return fn(m, type, 3, const_cast<void *>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, promotion,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    };
    if (encode()) return true;
    int dev = 0;
    return cudaGetDevice(&dev) == cudaSuccess && cudaSetDevice(dev) == cudaSuccess && encode();
}

// bf16 [n2][n1][cols] with the given row / slab strides (elements); box = 64 columns x box_rows x 1, 128-byte swizzle,
// zero fill outside the tensor
static inline bool tc_make_map(CUtensorMap *m, const void *ptr, long long n2, long long n1, long long cols, long long stride_1,
                               long long stride_2, int box_rows = 64) {
    cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)n1, (cuuint64_t)n2};
    cuuint64_t strides[2] = {(cuuint64_t)stride_1 * 2, (cuuint64_t)stride_2 * 2};
    cuuint32_t box[3] = {64, (cuuint32_t)box_rows, 1};
    return tc_encode_map(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, ptr, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B);
}

// [n2][n1][cols] dense, bf16 or fp32; box = box_cols x box_rows x 1, rows packed in shared memory (no swizzle): what a warp
// stores through when a lane owns a column
static inline bool tc_make_store_map(CUtensorMap *m, const void *ptr, bool f32, long long n2, long long n1, long long cols, int box_cols,
                                     int box_rows) {
    const int e = f32 ? 4 : 2;
    cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)n1, (cuuint64_t)n2};
    cuuint64_t strides[2] = {(cuuint64_t)cols * e, (cuuint64_t)(cols * n1) * e};
    cuuint32_t box[3] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows, 1};
    return tc_encode_map(m, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, ptr, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_NONE,
                         CU_TENSOR_MAP_L2_PROMOTION_NONE);
}

// ---------------------------------------------------------------------------------------------- PTX wrappers
__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.b32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// Bounded wait, a handful of instructions a site: the waits of a kernel with many roles are a good part of its code, and the
// roles share the instruction caches (a poll loop with a clock in it, unrolled at every site, made the delta walk 28 % slower).
// Each try suspends the thread for up to WAIT_HINT ns; at most WAIT_TRIES of them: 0.13 s if every one sleeps its full time,
// and still milliseconds, a thousand times a healthy wait, if none does. False (and the error flag set) when used up, so a
// broken pipeline winds down in a fraction of a second.
constexpr uint32_t WAIT_HINT = 1000, WAIT_TRIES = 1u << 17;
__device__ __forceinline__ bool mbar_wait_tries(uint32_t bar, uint32_t parity) {
    uint32_t left;
    asm volatile("{\n\t.reg .pred p;\n\t.reg .u32 n;\n\tmov.u32 n, %4;\n\t"
                 "AGAIN:\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t@p bra DONE;\n\t"
                 "sub.u32 n, n, 1;\n\tsetp.ne.u32 p, n, 0;\n\t@p bra AGAIN;\n\tDONE:\n\tmov.u32 %0, n;\n\t}"
                 : "=r"(left) : "r"(bar), "r"(parity), "r"(WAIT_HINT), "n"(WAIT_TRIES) : "memory");
    return left != 0;
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int code) {
    const bool good = mbar_wait_tries(bar, parity);
    if (!good) atomicExch(&g_tc_error, code);
    return good;
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap *map, uint32_t bar, int c0, int c1, int c2) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
                 ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
// shared -> global; rows outside the tensor are not written. One thread: commit, and wait before the source is reused.
__device__ __forceinline__ void tma_store_3d(const CUtensorMap *map, uint32_t src, int c0, int c1, int c2) {
    asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4}], [%1];"
                 ::"l"(map), "r"(src), "r"(c0), "r"(c1), "r"(c2) : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
__device__ __forceinline__ void tma_store_source_free() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void tma_store_done() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
// plain (untiled) bulk copy global -> shared, completion counted on an mbarrier; addresses and size multiples of 16 B
__device__ __forceinline__ void bulk_load_1d(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_alloc(uint32_t dst_smem, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
template <typename T_> __device__ __forceinline__ T_ warp_uniform(T_ x) { return __shfl_sync(0xffffffffu, x, 0); }
// D[M x N] (+)= A B issued by ONE elected lane of a converged warp: every lane executes the call with identical operands, so the
// descriptors stay warp-uniform values (the instruction takes them from the uniform datapath) instead of being moved
// there lane by lane under a divergent branch.
__device__ __forceinline__ void mma_bf16_elect(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p, e;\n\telect.sync _|e, 0xffffffff;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}"
                 ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0u) : "memory");
}
__device__ __forceinline__ void mma_commit_elect(uint32_t bar) {
    asm volatile("{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\t"
                 "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar) : "memory");
}
// 32 lanes x 32 columns of 32-bit: thread i of the warp gets lane (base lane + i), columns col .. col+31
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
    uint32_t *r = reinterpret_cast<uint32_t *>(v);
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                 "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                   "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                   "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// the same without the wait: the caller overlaps the load with other work and calls tmem_ld_wait() before using v
__device__ __forceinline__ void tmem_ld32_nowait(uint32_t taddr, float (&v)[32]) {
    uint32_t *r = reinterpret_cast<uint32_t *>(v);
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                 "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                   "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                   "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr) : "memory");
}

// 32 lanes x 16 columns of 32-bit, no wait (tmem_ld_wait() before v is used)
__device__ __forceinline__ void tmem_ld16_nowait(uint32_t taddr, float (&v)[16]) {
    uint32_t *r = reinterpret_cast<uint32_t *>(v);
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr) : "memory");
}

// 16 lanes x 256 bits per repetition: thread l of the warp gets, for block j of 8 columns,
//   v[4j+0], v[4j+1] = lane (base + l/4),     columns 8j + 2(l%4), +1
//   v[4j+2], v[4j+3] = lane (base + l/4 + 8), same columns
__device__ __forceinline__ void tmem_ld_frag4(uint32_t taddr, float (&v)[16]) {
    uint32_t *r = reinterpret_cast<uint32_t *>(v);
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x4.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld_frag8(uint32_t taddr, float (&v)[32]) {
    uint32_t *r = reinterpret_cast<uint32_t *>(v);
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x8.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                 "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                   "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                   "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld_frag2(uint32_t taddr, float (&v)[8]) {
    uint32_t *r = reinterpret_cast<uint32_t *>(v);
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr) : "memory");
}
template <int NB>
__device__ __forceinline__ void tmem_ld_frag(uint32_t taddr, float (&v)[4 * NB]) {
    if constexpr (NB == 4) tmem_ld_frag4(taddr, v); else tmem_ld_frag8(taddr, v);
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// four 8 x 8 matrices of 16-bit elements, a register each in fragment order; lane l gives the address of row l & 7 of matrix l >> 3
__device__ __forceinline__ void stmatrix4(uint32_t addr, uint32_t r0, uint32_t r1, uint32_t r2, uint32_t r3) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(r0), "r"(r1), "r"(r2), "r"(r3) : "memory");
}
__device__ __forceinline__ void named_sync(int id, int nthreads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory"); }
// the wait of a converged warp: the verdict is the same for every lane (they leave the chunk loop together)
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, int code) {
    const bool good = __all_sync(0xffffffffu, mbar_wait_tries(bar, parity));
    if (!good) atomicExch(&g_tc_error, code);
    return good;
}
// one arrival per warp, after every lane's shared-memory writes are visible to the async proxy
__device__ __forceinline__ void warp_arrive(uint32_t bar, int lane) {
    fence_proxy_async();
    __syncwarp();
    if (lane == 0) mbar_arrive(bar);
}

// ---------------------------------------------------------------------------------------------- operand A in tensor memory
// D[M x N] (+)= A B with A read from tensor memory: lane = row of A, each 32-bit column two consecutive bf16 along K (the
// even one in the low half), so one K = 16 step is 8 columns. Always K-major. Called by a converged warp; one elected lane
// issues (see mma_bf16_elect).
__device__ __forceinline__ void mma_bf16_ts_elect(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p, e;\n\telect.sync _|e, 0xffffffff;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t}"
                 ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0u) : "memory");
}
// thread i of the warp writes lane (base lane + i), 16 consecutive 32-bit columns; tmem_st_wait() before anyone reads them
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
                 "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                   "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// ---------------------------------------------------------------------------------------------- descriptors
// Shared-memory matrix descriptor, 128-byte swizzle. lbo / sbo in bytes.
//   K-major:  sbo = bytes between 8-row groups (1024); lbo unused (set 16).
//   MN-major: sbo = bytes between 8-row (K) groups (1024); lbo = bytes between 64-element groups along M/N.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = 0;
    d |= (uint64_t)((addr >> 4) & 0x3fff);
    d |= (uint64_t)((lbo >> 4) & 0x3fff) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3fff) << 32;
    d |= (uint64_t)1 << 46;                       // descriptor version (Blackwell)
    d |= (uint64_t)2 << 61;                       // SWIZZLE_128B
    return d;
}
// Instruction descriptor for kind::f16 with bf16 operands and an fp32 accumulator.
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N, int a_mn_major, int b_mn_major) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)a_mn_major << 15) | ((uint32_t)b_mn_major << 16) |
           ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// byte offset of the 16-byte chunk (row r, chunk j) in a [rows][128 B] tile with the 128-byte swizzle
__device__ __forceinline__ uint32_t swz(int r, int j) { return (uint32_t)(r * 128 + ((j ^ (r & 7)) << 4)); }

__device__ __forceinline__ void split_bf16(float x, __nv_bfloat16 &hi, __nv_bfloat16 &lo) {
    hi = __float2bfloat16_rn(x);
    lo = __float2bfloat16_rn(x - __bfloat162float(hi));
}
// 8 fp32 -> one 16-byte chunk of bf16 heads and one of tails
__device__ __forceinline__ void split8(const float (&x)[8], uint4 &hi, uint4 &lo) {
    __nv_bfloat162 h[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        h[i] = __floats2bfloat162_rn(x[2 * i], x[2 * i + 1]);         // one packed convert for two heads
        const float2 hf = __bfloat1622float2(h[i]);
        l[i] = __floats2bfloat162_rn(x[2 * i] - hf.x, x[2 * i + 1] - hf.y);
    }
    hi = *reinterpret_cast<uint4 *>(h);
    lo = *reinterpret_cast<uint4 *>(l);
}

// the same with what both leave over as a third: 24 bits of x in all
__device__ __forceinline__ void split8(const float (&x)[8], uint4 &hi, uint4 &lo, uint4 &rest) {
    split8(x, hi, lo);
    const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&hi), *l = reinterpret_cast<const __nv_bfloat162 *>(&lo);
    __nv_bfloat162 r[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 a = __bfloat1622float2(h[i]), b = __bfloat1622float2(l[i]);
        r[i] = __floats2bfloat162_rn(x[2 * i] - a.x - b.x, x[2 * i + 1] - a.y - b.y);
    }
    rest = *reinterpret_cast<uint4 *>(r);
}

// two fp32 -> packed bf16 heads and packed bf16 tails
__device__ __forceinline__ void split2(float a, float b, uint32_t &hi, uint32_t &lo) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    const float2 hf = __bfloat1622float2(h);
    const __nv_bfloat162 l = __floats2bfloat162_rn(a - hf.x, b - hf.y);
    hi = *reinterpret_cast<const uint32_t *>(&h);
    lo = *reinterpret_cast<const uint32_t *>(&l);
}

// m16n8k8 products of fp32 factors (the warp-level kind: blocks too small for tensor memory). x as a head of eleven bits and a tail rounded to eleven, which
// together miss up to 2^-23 of x: with tail by tail left out, a product is off by up to 2^-21 of itself
__device__ __forceinline__ void tf32_split(float x, uint32_t &hi, uint32_t &lo) {
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(hi) : "f"(x));
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(lo) : "f"(x - __uint_as_float(hi)));
}
__device__ __forceinline__ void mma_tf32(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}


// kernel parameters of the plain-rule tensor-core prefill kernels
struct TcParams {
    const float *la, *S0, *theta, *shift_dev;
    float shift_host;
    void *o; float *S_out; __nv_bfloat16 *sent;
    int H, T, o_is_f32;
    // fused layer pieces (all optional): decay gate logits instead of log-decays, per-head RMS norm of the read,
    // token-major output
    const __nv_bfloat16 *la_raw; long long aux_sb, aux_st; const float *decay_A;
    const float *rms_w; float rms_eps; int o_token_major;
    // RAW mode: write-gate logits (same strides as la_raw) and the rotation table [H][rot_T][D/2] of (cos, sin)
    const __nv_bfloat16 *gate_raw; const float2 *rot; int rot_T;
    // warp-specialised kernel: chains, and their segments (the first is entered with S0, the states entering segments 1, 2, ... are
    // seg_states [nseg - 1][BH][D][D], where seg_rotates rebased like S0 at a piece's beginning)
    int BH; SegCut seg; const float *seg_states; int seg_rotates;
};


}  // namespace pgb
