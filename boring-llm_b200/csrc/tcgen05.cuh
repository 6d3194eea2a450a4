// What the tcgen05 kernels share: thin wrappers around the PTX of mbarriers, TMA loads, tcgen05.mma / ld / fences,
// the shared-memory operand descriptor, and the host side's tensor maps. Each kernel file keeps its own status
// word, into which its bounded waits record, and its own instruction descriptors.
#pragma once
#include "common.cuh"
#include "api.h"
#include <cuda.h>

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// ---- mbarriers (shared memory of this block) ---------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(bar) : "memory");
}
// One try of a wait on the phase of parity `parity`: true once that phase has completed.
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}

// Bounded wait of a block that goes on after a wait has run out: false when the bound did or another thread of the block has given up;
// the first such wait leaves `code` in the file's status word.
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity, uint32_t limit, volatile int* give_up, int* status, int code) {
#pragma unroll 1
    for (uint32_t i = 0; i < limit; ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if (*give_up) return false;
    }
    *give_up = 1;
    atomicCAS(status, 0, code);
    return false;
}
// Bounded wait that does not look at the give-up flag (a block that has given up waits for its own copies).
__device__ __forceinline__ void mbar_wait_landed(uint32_t bar, uint32_t parity, uint32_t limit) {
#pragma unroll 1
    for (uint32_t i = 0; i < limit; ++i)
        if (mbar_try_wait(bar, parity)) return;
}

// All blocks of the cluster; what each has written before is visible to the others behind it.
__device__ __forceinline__ void cluster_meet() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// ---- TMA: one 2-D box into shared memory, its bytes reported to `bar` -----------------------------------------
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                 :: "r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1) : "memory");
}

// Asks for a tensor map to be brought into the TMA unit's descriptor cache (no register, no wait): at the top of a
// kernel, so that its first copy does not wait for the descriptor.
__device__ __forceinline__ void tma_prefetch_map(const CUtensorMap* map) {
    asm volatile("prefetch.tensormap [%0];" :: "l"(map) : "memory");
}

// True in one thread of a converged warp. Code that issues copies and MMAs stands behind this and not behind a test of the
// lane: the compiler then knows that one thread runs it and feeds the instructions' uniform operands directly, where it
// otherwise goes round a loop over the active threads for each (58 cycles of issue an MMA, more than a 256 x 128 x 16
// MMA of a pair takes). Measured on pairs of SMs, 2,048 rows: 896 x 896 10.4 -> 8.8 us, 896 x 4,864 24.3 -> 21.1, 4,864 + 4,864
// x 896 32.8 -> 28.4 (with tensor memory taken before the wait for the kernel before, 1,800 cycles off the path).
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(p));
    return p != 0;
}
// The warp's number as a value that is known to be the same in all its lanes.
__device__ __forceinline__ int uniform_warp() { return __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0); }

// ---- tcgen05 --------------------------------------------------------------------------------------------------
// D (tensor memory) (+)= A . B, both operands in shared memory, one block
__device__ __forceinline__ void umma_bf16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}"
                 :: "r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
// `bar` gets one arrival when every MMA issued so far by this thread has completed
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(bar) : "memory");
}
// 32 columns of this warp's 32 lanes of tensor memory: thread t gets lane t, register j column j
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                 "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                   "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                   "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// 16 columns, waited for
__device__ __forceinline__ void tmem_ld16_wait(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
                 "tcgen05.wait::ld.sync.aligned;"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr) : "memory");
}
__device__ __forceinline__ void fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Operand tile in shared memory with 128-byte swizzle: rows of 128 bytes, groups of 8 rows 1024 bytes apart. The
// same descriptor serves a K-major operand (rows = M or N, 64 elements of K per row) and an MN-major one (rows = K,
// 64 elements of N per row; the instruction descriptor says which).
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
    const uint32_t lo = ((addr >> 4) & 0x3FFFu) | (1u << 16);                 // start address, leading offset 1 (unused: one 64-wide atom)
    const uint32_t hi = (1024u >> 4) | (1u << 14) | (2u << 29);               // stride offset, version 1, SWIZZLE_128B
    return ((uint64_t)hi << 32) | lo;
}

// ---- host: tensor maps ------------------------------------------------------------------------------------------
typedef CUresult (*BlEncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// cuTensorMapEncodeTiled through the runtime (the library does not link the driver); nullptr if the driver has none
inline BlEncodeTiled bl_tensor_map_encoder() {
    static BlEncodeTiled fn = nullptr;
    if (fn == nullptr) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (BlEncodeTiled)p;
    }
    return fn;
}

// A row-major [rows, cols] bfloat16 matrix as a 2-D tensor map with boxes of box_rows x box_cols elements (box_cols
// x 2 bytes = 128: one swizzle atom), 128-byte swizzle. `who` names the caller in the error.
inline int bl_make_map_bf16(const char* who, CUtensorMap* map, const void* ptr, long long rows, long long cols,
                            int box_rows, int box_cols) {
    BlEncodeTiled enc = bl_tensor_map_encoder();
    if (enc == nullptr) BL_FAIL("%s: cuTensorMapEncodeTiled is not available from the driver", who);
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
    cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS)
        BL_FAIL("%s: cuTensorMapEncodeTiled failed with code %d (rows %lld, columns %lld)", who, (int)r, rows, cols);
    return 0;
}
