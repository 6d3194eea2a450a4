// Matrix products of routed experts on the fifth-generation tensor cores: rows of x that lie expert by expert (bl_moe_plan with tiles
// of 16 rows), out[row] = epilogue(x[row] . W[expert of the row]^T), bfloat16 operands, 32-bit accumulation in tensor memory.
//
// An expert has few hundred rows of a prompt and a handful in a decode step, never a multiple of 128, so the rows of x are the N side
// of the MMA, which takes any multiple of 16 (a tile of 128 rows of x computed 35 % padding at 250 rows an expert), and 128 rows of W
// the M side. A chunk is up to NT rows of one expert (more rows: several chunks of even size); a work item is a chunk by a tile of W,
// chunk after chunk, so that W crosses HBM once and the chunks of one expert find its tiles in L2. One block an SM walks items with
// two accumulators: an item's epilogue runs under the next one's products. NT is 256 (128 x 256 products need 96 bytes of operands a
// cycle and SM at the tensor cores' rate, 128 x 128 ones 128) or, for few rows an expert, 64 with a ring of nine stages to stream W.
// SWIGLU: a tile is 64 gate rows of W and the 64 up rows that match, in runs of 16: a warp's lanes 0..15 hold gate rows, lanes 16..31
// the matching up rows, and one exchange of two neighbouring tokens' values gives every lane a pair to gate.
// 16 experts of 2,752 hidden values, two a token, 2,048 wide (gate/up and down, us; tiles of 128 rows -> this): 2,000 tokens 117 -> 102
// and 73 -> 64, 1,000 tokens 81 -> 75 and 54 -> 42, 64 tokens 71 -> 58 and 39 -> 32 (6.3 TB/s of W).
// One thread issues the copies of W, one those of x, one the MMAs, four warps the epilogue. Every wait on an mbarrier is bounded; when
// a bound runs out the block records a code in a status word, lets its own copies land, frees its tensor memory and returns
// (bl_gemm_tc_experts_status).
#include "tcgen05.cuh"
#include <atomic>

namespace {

constexpr const char* WHO = "bl_gemm_tc_experts";

constexpr int BN = 128;                 // rows of W a tile
constexpr int BK = 64;
constexpr int RUN = 16;                 // rows of a run of gate (or up) rows
constexpr int X_BOX = 32;               // rows of x a copy
constexpr int W_BYTES = BN * BK * 2;
constexpr int THREADS = 224;            // warp 0: copies of W, warp 1: copies of x, warp 2: MMAs, warps 3..6: epilogue
constexpr uint32_t WAIT_LIMIT = 1u << 22;

template <int NT>
struct Ring {
    static constexpr int STAGE_BYTES = W_BYTES + NT * BK * 2;
    static constexpr int STAGES = (227 * 1024 - 1024 - 512) / STAGE_BYTES;
    static constexpr int OFF_BARS = STAGES * STAGE_BYTES;
    static constexpr int SMEM_BYTES = OFF_BARS + 512 + 1024;
    static constexpr int TMEM_COLS = 2 * NT;
    static_assert(NT % X_BOX == 0 && STAGES >= 4 && STAGES <= 14 && SMEM_BYTES <= 227 * 1024 && TMEM_COLS >= 32 && TMEM_COLS <= 512, "ring");
};

__device__ int g_status = 0;            // 0 = fine; else the code of the first wait that ran out

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* give_up, int code) {
    return mbar_wait_bounded(bar, parity, WAIT_LIMIT, give_up, &g_status, code);
}

// chunks[0].x: how many; chunks[1 + c]: {first row of x, rows (a multiple of 16, up to NT), expert, 0}.
template <bool GLU, typename TO, int NT>
__global__ void __launch_bounds__(THREADS, 1)
gemm_tc_experts_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const int4* __restrict__ chunks,
                       const float* __restrict__ act, TO* __restrict__ out, int N, int K) {
    using R = Ring<NT>;
    constexpr int STAGES = R::STAGES;
    constexpr int UNITS = GLU ? BN / 2 : BN;                                   // output columns a tile
    extern __shared__ unsigned char smem_raw[];
    if (threadIdx.x == 0) { tma_prefetch_map(&map_x); tma_prefetch_map(&map_w); }
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;               // the swizzled tiles need 1024-byte alignment
    unsigned char* smem = smem_raw + (base - smem_u32(smem_raw));
    const uint32_t full0 = base + R::OFF_BARS, empty0 = full0 + 8 * STAGES, acc_full0 = empty0 + 8 * STAGES, acc_empty0 = acc_full0 + 16;
    volatile int* give_up = reinterpret_cast<volatile int*>(smem + R::OFF_BARS + 384);
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem + R::OFF_BARS + 392);
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const int kblocks = (K + BK - 1) / BK, n_tiles = (N + UNITS - 1) / UNITS;

    if (threadIdx.x == 0) {
        *give_up = 0;
        for (int s = 0; s < STAGES; ++s) { mbar_init(full0 + 8 * s, 2); mbar_init(empty0 + 8 * s, 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(acc_full0 + 8 * b, 1); mbar_init(acc_empty0 + 8 * b, 4); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // Tensor memory is taken before the dependent-launch wait: whoever on this stream uses it triggers its successor only behind its
    // own allocation, so an allocation that has to wait here waits for a block that needs nothing from this one.
    if (warp == 2) {
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     :: "r"(smem_u32((const void*)tmem_slot)), "r"(R::TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = *tmem_slot;
    bl_pdl_wait();                                                             // chunks, x and out belong to the predecessor until here
    bl_pdl_trigger();
    const int items = chunks[0].x * n_tiles;

    if (warp < 2) {                                                            // stage it is stage it of the block, whatever its item
        if (elect_one()) {
            int it = 0;
            bool ok = true;
            for (int item = blockIdx.x; ok && item < items; item += gridDim.x) {
                const int4 c = chunks[1 + item / n_tiles];
                const int n0 = item % n_tiles * UNITS, row0 = c.z * (GLU ? 2 * N : N) + n0, boxes = (c.y + X_BOX - 1) / X_BOX;
                for (int kb = 0; kb < kblocks; ++kb, ++it) {
                    const int s = it % STAGES;
                    if (it >= STAGES && !mbar_wait(empty0 + 8 * s, (uint32_t)((it / STAGES - 1) & 1), give_up, 1)) { ok = false; break; }
                    const uint32_t dst = base + s * R::STAGE_BYTES, bar = full0 + 8 * s;
                    if (warp == 0) {
                        mbar_expect_tx(bar, W_BYTES);
                        if (GLU) {
#pragma unroll
                            for (int j = 0; j < BN / 2 / RUN; ++j) {
                                tma_load_2d(dst + 2 * j * RUN * BK * 2, &map_w, bar, kb * BK, row0 + j * RUN);
                                tma_load_2d(dst + (2 * j + 1) * RUN * BK * 2, &map_w, bar, kb * BK, row0 + N + j * RUN);
                            }
                        } else {
                            tma_load_2d(dst, &map_w, bar, kb * BK, row0);
                        }
                    } else {
                        mbar_expect_tx(bar, boxes * X_BOX * BK * 2);
                        for (int b = 0; b < boxes; ++b) tma_load_2d(dst + W_BYTES + b * X_BOX * BK * 2, &map_x, bar, kb * BK, c.x + b * X_BOX);
                    }
                }
            }
            if (*give_up)                                                      // let our own copies land before leaving
                for (int i = max(0, it - STAGES); i < it; ++i) mbar_wait_landed(full0 + 8 * (i % STAGES), (uint32_t)((i / STAGES) & 1), WAIT_LIMIT);
        }
        __syncwarp();
    } else if (warp == 2) {
        if (elect_one()) {
            int it = 0, local = 0;
            bool ok = true;
            for (int item = blockIdx.x; ok && item < items; item += gridDim.x, ++local) {
                // kind::f16: D 32-bit, A and B bfloat16 and K-major, N >> 3 at bit 17, M >> 4 at bit 24
                const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(chunks[1 + item / n_tiles].y >> 3) << 17) | ((uint32_t)(BN >> 4) << 24);
                const int buf = local & 1;
                if (local >= 2 && !mbar_wait(acc_empty0 + 8 * buf, (uint32_t)((local / 2 - 1) & 1), give_up, 3)) break;
                fence_after_sync();
                for (int kb = 0; kb < kblocks; ++kb, ++it) {
                    const int s = it % STAGES;
                    if (!mbar_wait(full0 + 8 * s, (uint32_t)((it / STAGES) & 1), give_up, 2)) { ok = false; break; }
                    fence_after_sync();
                    const uint64_t a = smem_desc(base + s * R::STAGE_BYTES), b = smem_desc(base + s * R::STAGE_BYTES + W_BYTES);
#pragma unroll
                    for (int k = 0; k < BK / 16; ++k) umma_bf16(tmem + buf * NT, a + 2 * k, b + 2 * k, idesc, (kb | k) != 0);
                    umma_commit(empty0 + 8 * s);
                }
                if (ok) umma_commit(acc_full0 + 8 * buf);
            }
        }
        __syncwarp();
    } else {
        // lane r of tensor memory is row r of the tile of W, its columns are the chunk's rows of x
        const int q = warp & 3;
        const BlGluArgs glu = bl_glu_args(GLU ? act : nullptr);
        int local = 0;
        for (int item = blockIdx.x; item < items; item += gridDim.x, ++local) {
            const int4 c = chunks[1 + item / n_tiles];
            const int buf = local & 1, n0 = item % n_tiles * UNITS;
            const bool ok = mbar_wait(acc_full0 + 8 * buf, (uint32_t)((local / 2) & 1), give_up, 4);
            if (!__all_sync(0xffffffffu, ok)) break;
            fence_after_sync();
            const uint32_t taddr = tmem + buf * NT + ((uint32_t)(q * 32) << 16);
            const int n = n0 + (GLU ? q * RUN + (lane & 15) : q * 32 + lane), odd = GLU ? lane >> 4 : 0;
            TO* dst = out + (size_t)(c.x + odd) * N + n;
#pragma unroll 1
            for (int t = 0; t < c.y; t += 16) {
                uint32_t r[16];
                tmem_ld16_wait(taddr + t, r);
                if (GLU) {
#pragma unroll
                    for (int j = 0; j < 16; j += 2) {                          // lanes 0..15 gate row t + j, lanes 16..31 row t + j + 1
                        const uint32_t other = __shfl_xor_sync(0xffffffffu, odd ? r[j] : r[j + 1], 16);
                        const float g = __uint_as_float(odd ? other : r[j]), u = __uint_as_float(odd ? r[j + 1] : other);
                        if (n < N) bl_store(dst + (size_t)(t + j) * N, bl_glu_fast(glu.kind, g, u, glu.limit));
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        if (n < N) bl_store(dst + (size_t)(t + j) * N, __uint_as_float(r[j]));
                }
            }
            fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(acc_empty0 + 8 * buf);
        }
    }
    __syncwarp();
    fence_before_sync();
    __syncthreads();
    if (warp == 2) {
        fence_after_sync();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(R::TMEM_COLS) : "memory");
    }
}

template <bool GLU, typename TO, int NT>
int launch(const CUtensorMap& mx, const CUtensorMap& mw, const int4* chunks, const float* act, void* out, int max_chunks, int N, int K, cudaStream_t s) {
    static std::atomic<bool> configured{false};
    if (!configured) {
        BL_CUDA(cudaFuncSetAttribute(gemm_tc_experts_kernel<GLU, TO, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, Ring<NT>::SMEM_BYTES));
        configured = true;
    }
    const long long items = (long long)max_chunks * ((N + (GLU ? BN / 2 : BN) - 1) / (GLU ? BN / 2 : BN));
    if (items > 0x7fffffffLL) BL_FAIL("bl_gemm_tc_experts: too many tiles");
    const int blocks = items < bl_device_sms() ? (int)items : bl_device_sms();
    BL_CUDA(bl_launch_dependent(gemm_tc_experts_kernel<GLU, TO, NT>, dim3((unsigned)blocks), dim3(THREADS), (size_t)Ring<NT>::SMEM_BYTES, s,
                                mx, mw, chunks, act, (TO*)out, N, K));
    BL_CHECK_LAUNCH("bl_gemm_tc_experts");
    return 0;
}

}  // namespace

extern "C" int bl_gemm_tc_experts(const void* x, const void* w, void* out, int out_dtype, int M, int N, int K, int epilogue, int n_experts,
                                  const int* chunks, int max_chunks, int chunk_rows, const float* act, void* stream) {
    if (M <= 0 || max_chunks <= 0) return 0;
    const bool glu = epilogue == BL_EPI_SWIGLU;
    if (N <= 0 || K <= 0 || n_experts <= 0 || chunks == nullptr || (chunk_rows != 64 && chunk_rows != 256))
        BL_FAIL("bl_gemm_tc_experts: bad sizes M=%d N=%d K=%d experts=%d chunks of %d", M, N, K, n_experts, chunk_rows);
    if (K % 8 != 0) BL_FAIL("bl_gemm_tc_experts: K=%d is not a multiple of 8 (TMA rows must be 16-byte multiples)", K);
    if (((uintptr_t)x | (uintptr_t)w | (uintptr_t)chunks) & 15) BL_FAIL("bl_gemm_tc_experts: x, W and the chunks must be 16-byte aligned");
    if (!(glu && out_dtype == BL_BF16) && !(epilogue == BL_EPI_NONE && out_dtype == BL_F32))
        BL_FAIL("bl_gemm_tc_experts: epilogue %d with results of type %d is not built", epilogue, out_dtype);
    const long long expert_rows = glu ? 2LL * N : N;
    if (n_experts * expert_rows > 0x7fffffffLL) BL_FAIL("bl_gemm_tc_experts: the stack of matrices has too many rows");
    CUtensorMap mx, mw;
    if (bl_make_map_bf16(WHO, &mx, x, M, K, X_BOX, BK)) return 1;
    if (bl_make_map_bf16(WHO, &mw, w, (int)(n_experts * expert_rows), K, glu ? RUN : BN, BK)) return 1;
    cudaStream_t s = (cudaStream_t)stream;
    const int4* c = (const int4*)chunks;
    if (glu) return chunk_rows == 64 ? launch<true, __nv_bfloat16, 64>(mx, mw, c, act, out, max_chunks, N, K, s)
                                     : launch<true, __nv_bfloat16, 256>(mx, mw, c, act, out, max_chunks, N, K, s);
    return chunk_rows == 64 ? launch<false, float, 64>(mx, mw, c, act, out, max_chunks, N, K, s)
                            : launch<false, float, 256>(mx, mw, c, act, out, max_chunks, N, K, s);
}

// Reads and clears the status word: 0 when no block has given up on a wait (1 copies, 2 issuer, 3 accumulator free, 4 epilogue).
extern "C" int bl_gemm_tc_experts_status(int* status) {
    int v = 0, zero = 0;
    BL_CUDA(cudaMemcpyFromSymbol(&v, g_status, sizeof(int)));
    if (v != 0) BL_CUDA(cudaMemcpyToSymbol(g_status, &zero, sizeof(int)));
    *status = v;
    return 0;
}
