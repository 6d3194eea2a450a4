// Matrix product for FEW rows (a decode step's) of large matrices on the fifth-generation tensor cores:
// out[M, N] = epilogue(x[M, K] . W[N, K]^T) with M up to 64, bfloat16 operands, 32-bit accumulation in tensor memory.
//
// Bound by the stream of W from HBM, so, as for an output head (gemm_tcgen05_cols.cu), W is the M side of the MMA and the rows of x,
// padded to NT, its N side: a stage of the ring is 128 rows of W by 64 of k (16 KB) and the NT x 64 of x that go with it (2 KB
// for 16 rows; x as the M side would pass 16 KB of padding through shared memory for each). What this kernel adds: the epilogues, and
// blocks for every shape. Where W has fewer tiles of 128 rows than the device SMs, a cluster of blocks shares a tile and cuts K;
// the partial sums meet through distributed shared memory, added in block order. Where it has more, one block an SM walks tiles,
// with two accumulators, so that a tile's epilogue runs under the next one's products. The ring's first round of W is asked for
// before the dependent-launch wait: W does not depend on the kernel before.
// SWIGLU: a tile is 64 gate rows of W and the 64 up rows that match.
// 16 rows, launches in a row on cold matrices: gate/up of 18,944 + 18,944 x 3,584 61.5 -> 42.3 us (6.4 TB/s), 3,584 x 3,584 12.0 -> 8.0,
// 8,208 x 2,048 14.5 -> 8.8, 11,008 + 11,008 x 2,048 46.7 -> 21.6; one row of 3,584 x 18,944 38.6 -> 27.1.
// One thread issues the copies, one the MMAs, four warps the epilogue. Every wait on an mbarrier is bounded; when a bound runs out
// the block records a code in a status word, lets its own copies land, still meets its cluster, frees its tensor memory and returns
// (bl_gemm_tc_few_status).
#include "tcgen05.cuh"
#include <atomic>
#include <mutex>

namespace {

constexpr const char* WHO = "bl_gemm_tc_few";

constexpr int BN = 128;                 // rows of W a tile
constexpr int BK = 64;
constexpr int W_BYTES = BN * BK * 2;
constexpr int THREADS = 192;            // warp 0: copies, warp 1: MMAs, warps 2..5: epilogue
constexpr int MAX_SPLIT = 8;            // the portable cluster size
constexpr int PITCH = BN + 4;           // floats from one token's sums to the next
constexpr uint32_t WAIT_LIMIT = 1u << 22;

template <int NT>
struct Ring {
    static constexpr int X_BYTES = NT * BK * 2, STAGE_BYTES = W_BYTES + X_BYTES;
    static constexpr int PART_BYTES = NT * PITCH * 4;
    static constexpr int STAGES_FIT = (227 * 1024 - 1024 - 512 - PART_BYTES) / STAGE_BYTES;
    static constexpr int STAGES = STAGES_FIT > 12 ? 12 : STAGES_FIT;
    static constexpr int OFF_PART = STAGES * STAGE_BYTES, OFF_BARS = OFF_PART + PART_BYTES;
    static constexpr int SMEM_BYTES = OFF_BARS + 512 + 1024;
    static constexpr int TMEM_COLS = 2 * NT < 32 ? 32 : 2 * NT;
    static_assert(NT % 16 == 0 && STAGES >= 4 && SMEM_BYTES <= 227 * 1024, "ring");
};

__device__ int g_status = 0;            // 0 = fine; else the code of the first wait that ran out

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* give_up, int code) {
    return mbar_wait_bounded(bar, parity, WAIT_LIMIT, give_up, &g_status, code);
}
__device__ __forceinline__ float4 ld_cluster4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}

template <int EPI, typename TO, int NT>
__global__ void __launch_bounds__(THREADS, 1)
gemm_tc_few_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const void* __restrict__ bias,
                   int bias_dtype, TO* __restrict__ out, int M, int N, int K, int split) {
    using R = Ring<NT>;
    constexpr bool GLU = EPI == BL_EPI_SWIGLU;
    constexpr int UNITS = GLU ? BN / 2 : BN;                                   // output columns a tile
    constexpr int STAGES = R::STAGES;
    // kind::f16: D 32-bit, A and B bfloat16 and K-major, N >> 3 at bit 17, M >> 4 at bit 24
    constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(NT >> 3) << 17) | ((uint32_t)(BN >> 4) << 24);
    extern __shared__ unsigned char smem_raw[];
    if (threadIdx.x == 0) { tma_prefetch_map(&map_x); tma_prefetch_map(&map_w); }
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;               // the swizzled tiles need 1024-byte alignment
    unsigned char* smem = smem_raw + (base - smem_u32(smem_raw));
    const uint32_t full0 = base + R::OFF_BARS, empty0 = full0 + 8 * STAGES, acc_full0 = empty0 + 8 * STAGES, acc_empty0 = acc_full0 + 16;
    volatile int* give_up = reinterpret_cast<volatile int*>(smem + R::OFF_BARS + 256);
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem + R::OFF_BARS + 264);
    float* part = reinterpret_cast<float*>(smem + R::OFF_PART);                // [NT][PITCH]: a tile's sums
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const int kblocks = (K + BK - 1) / BK, n_tiles = (N + UNITS - 1) / UNITS;
    // split > 1: the blocks of a cluster share tile blockIdx.x / split; split 1: block b walks tiles b, b + gridDim.x, ...
    const int rank = blockIdx.x % split, first = blockIdx.x / split, step = gridDim.x / split;
    const int kb0 = (int)((long long)rank * kblocks / split), nkb = (int)((long long)(rank + 1) * kblocks / split) - kb0;
    const int my_tiles = first < n_tiles ? (n_tiles - 1 - first) / step + 1 : 0;
    const int total = my_tiles * nkb;                                          // stages that this block fills

    if (threadIdx.x == 0) {
        *give_up = 0;
        for (int s = 0; s < STAGES; ++s) { mbar_init(full0 + 8 * s, 1); mbar_init(empty0 + 8 * s, 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(acc_full0 + 8 * b, 1); mbar_init(acc_empty0 + 8 * b, 4); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    auto load_w = [&](int it) {                                                // and announce the stage's bytes
        const int s = it % STAGES, n0 = (first + it / nkb * step) * UNITS, kb = kb0 + it % nkb;
        const uint32_t dst = base + s * R::STAGE_BYTES;
        mbar_expect_tx(full0 + 8 * s, R::STAGE_BYTES);
        if (GLU) {
            tma_load_2d(dst, &map_w, full0 + 8 * s, kb * BK, n0);
            tma_load_2d(dst + W_BYTES / 2, &map_w, full0 + 8 * s, kb * BK, N + n0);
        } else {
            tma_load_2d(dst, &map_w, full0 + 8 * s, kb * BK, n0);
        }
    };
    const int early = min(STAGES, total);
    if (warp == 0 && elect_one())
        for (int it = 0; it < early; ++it) load_w(it);
    __syncwarp();
    // Tensor memory, too, is taken before the wait: whoever on this stream uses it triggers its successor only behind its
    // own allocation, so an allocation that has to wait here waits for a block that needs nothing from this one.
    if (warp == 1) {
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     :: "r"(smem_u32((const void*)tmem_slot)), "r"(R::TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = *tmem_slot;
    bl_pdl_wait();                                                             // x and out belong to the predecessor until here
    bl_pdl_trigger();

    // What the epilogue does with the sums of four neighbouring output columns n .. n + 3 of row m.
    const BlGluArgs glu = bl_glu_args(GLU ? bias : nullptr);
    auto finish = [&](float (&v)[4], const float (&u)[4], int m, int n) {
        TO* dst = out + (size_t)m * N + n;
        const bool whole = (N & 3) == 0 && n + 3 < N;
        if (GLU) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float g = v[j], up = u[j];
                if (glu.bias && n + j < N) { g += glu.bias[n + j]; up += glu.bias[N + n + j]; }
                v[j] = bl_glu(glu.kind, g, up, glu.limit);                     // (the exponential and division of the kernel for few rows beside this one)
            }
        }
        if (EPI == BL_EPI_BIAS || (EPI == BL_EPI_RESIDUAL && bias != nullptr)) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (n + j < N) v[j] += bl_load_any(bias, bias_dtype, n + j);
        }
        if (whole) {
            if constexpr (sizeof(TO) == 4) {
                float4 r = make_float4(v[0], v[1], v[2], v[3]);
                if (EPI == BL_EPI_RESIDUAL) {
                    const float4 o = *reinterpret_cast<const float4*>(dst);
                    r.x += o.x; r.y += o.y; r.z += o.z; r.w += o.w;
                }
                *reinterpret_cast<float4*>(dst) = r;
            } else {
                const __nv_bfloat162 lo = __floats2bfloat162_rn(v[0], v[1]), hi = __floats2bfloat162_rn(v[2], v[3]);
                *reinterpret_cast<uint2*>(dst) = make_uint2(*reinterpret_cast<const unsigned*>(&lo), *reinterpret_cast<const unsigned*>(&hi));
            }
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (n + j >= N) break;
                if (EPI == BL_EPI_RESIDUAL) v[j] += bl_load(dst + j);
                bl_store(dst + j, v[j]);
            }
        }
    };
    constexpr int QUADS = UNITS / 4;

    if (warp == 0) {
        if (elect_one()) {
            int issued = 0;
            for (int it = 0; it < total; ++it) {
                const int s = it % STAGES;
                if (it >= early) {
                    if (!mbar_wait(empty0 + 8 * s, (uint32_t)((it / STAGES - 1) & 1), give_up, 1)) break;
                    load_w(it);
                }
                tma_load_2d(base + s * R::STAGE_BYTES + W_BYTES, &map_x, full0 + 8 * s, (kb0 + it % nkb) * BK, 0);
                issued = it + 1;
            }
            if (*give_up)                                                      // let our own copies land before leaving
                for (int it = max(0, issued - STAGES); it < issued; ++it) mbar_wait_landed(full0 + 8 * (it % STAGES), (uint32_t)((it / STAGES) & 1), WAIT_LIMIT);
        }
        __syncwarp();
    } else if (warp == 1) {
        if (elect_one()) {
            bool ok = true;
            int it = 0;
            for (int local = 0; ok && local < my_tiles; ++local) {
                const int buf = local & 1;
                if (local >= 2 && !mbar_wait(acc_empty0 + 8 * buf, (uint32_t)((local / 2 - 1) & 1), give_up, 4)) break;
                for (int kb = 0; kb < nkb; ++kb, ++it) {
                    const int s = it % STAGES;
                    if (!mbar_wait(full0 + 8 * s, (uint32_t)((it / STAGES) & 1), give_up, 2)) { ok = false; break; }
                    fence_after_sync();
                    const uint64_t a = smem_desc(base + s * R::STAGE_BYTES), b = smem_desc(base + s * R::STAGE_BYTES + W_BYTES);
#pragma unroll
                    for (int k = 0; k < BK / 16; ++k) umma_bf16(tmem + buf * NT, a + 2 * k, b + 2 * k, IDESC, (kb | k) != 0);
                    umma_commit(empty0 + 8 * s);
                }
                if (ok) umma_commit(acc_full0 + 8 * buf);
            }
        }
        __syncwarp();
    } else {
        // lane r of tensor memory is row r of the tile of W, its NT columns are the tokens
        const int q = warp & 3;
        bool ok = true;
        for (int local = 0; local < my_tiles; ++local) {
            const int buf = local & 1;
            // (a warp that has given up still comes to the barriers of the four: another may have found this tile complete)
            ok = ok && mbar_wait(acc_full0 + 8 * buf, (uint32_t)((local / 2) & 1), give_up, 5);
            ok = __all_sync(0xffffffffu, ok);
            if (ok) {
                fence_after_sync();
                const uint32_t taddr = tmem + buf * NT + ((uint32_t)(q * 32) << 16);
#pragma unroll
                for (int c = 0; c < NT; c += 16) {
                    uint32_t r[16];
                    tmem_ld16_wait(taddr + c, r);
#pragma unroll
                    for (int j = 0; j < 16; ++j) part[(c + j) * PITCH + q * 32 + lane] = __uint_as_float(r[j]);
                }
                fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(acc_empty0 + 8 * buf);
            }
            if (split > 1) break;                                              // one tile a cluster: the blocks meet below
            asm volatile("bar.sync 1, 128;" ::: "memory");                     // the four warps' sums
            const int n0 = (first + local * step) * UNITS;
            for (int e = threadIdx.x - 64; ok && e < M * QUADS; e += 128) {
                const int m = e / QUADS, c = e % QUADS * 4;
                if (n0 + c >= N) continue;
                const float4 a = *reinterpret_cast<const float4*>(part + m * PITCH + c);
                float v[4] = {a.x, a.y, a.z, a.w}, u[4] = {0.f, 0.f, 0.f, 0.f};
                if (GLU) {
                    const float4 b = *reinterpret_cast<const float4*>(part + m * PITCH + UNITS + c);
                    u[0] = b.x; u[1] = b.y; u[2] = b.z; u[3] = b.w;
                }
                finish(v, u, m, n0 + c);
            }
            asm volatile("bar.sync 1, 128;" ::: "memory");                     // the sums have been read
        }
    }
    if (split > 1) {
        __syncwarp();
        cluster_meet();                                                        // every block's sums are written and visible
        const uint32_t mine = base + R::OFF_PART;
        const int quads = M * QUADS, e1 = (int)((long long)(rank + 1) * quads / split), n0 = first * UNITS;
        for (int e = (int)((long long)rank * quads / split) + threadIdx.x; e < e1; e += THREADS) {
            const int m = e / QUADS, c = e % QUADS * 4;
            if (n0 + c >= N) continue;
            float v[4] = {0.f, 0.f, 0.f, 0.f}, u[4] = {0.f, 0.f, 0.f, 0.f};
            for (int r = 0; r < split; ++r) {
                uint32_t peer;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(mine + (uint32_t)(m * PITCH + c) * 4), "r"(r));
                const float4 a = ld_cluster4(peer);
                v[0] += a.x; v[1] += a.y; v[2] += a.z; v[3] += a.w;
                if (GLU) {
                    const float4 b = ld_cluster4(peer + UNITS * 4);
                    u[0] += b.x; u[1] += b.y; u[2] += b.z; u[3] += b.w;
                }
            }
            finish(v, u, m, n0 + c);
        }
    }
    __syncwarp();
    fence_before_sync();
    if (split > 1) cluster_meet(); else __syncthreads();                       // no block leaves while another may still read its sums
    if (warp == 1) {
        fence_after_sync();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(R::TMEM_COLS) : "memory");
    }
}

// Clusters of each size that the device holds at once with one block of this kernel an SM (clusters live inside one GPC, so fewer
// fit than SMs divided by their size), asked once.
const int* clusters_at_once() {
    static int active[MAX_SPLIT + 1] = {};
    static std::once_flag once;
    std::call_once(once, [] {
        auto kernel = gemm_tc_few_kernel<BL_EPI_NONE, float, 16>;
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Ring<16>::SMEM_BYTES) != cudaSuccess) { (void)cudaGetLastError(); return; }
        for (int sp = 2; sp <= MAX_SPLIT; ++sp) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(sp * bl_device_sms());
            cfg.blockDim = dim3(THREADS);
            cfg.dynamicSmemBytes = Ring<16>::SMEM_BYTES;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = sp; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
            cfg.attrs = attr; cfg.numAttrs = 1;
            int n = 0;
            if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) { (void)cudaGetLastError(); n = 0; }
            active[sp] = n;
        }
    });
    return active;
}

// How many blocks share a tile: the most of which the device holds as many clusters at once as there are tiles, two k blocks each at
// least; 1 where there are more tiles.
int split_for(int n_tiles, int kblocks) {
    const int* active = clusters_at_once();
    int best = 1;
    for (int sp = 2; sp <= MAX_SPLIT && 2 * sp <= kblocks; ++sp)
        if (active[sp] >= n_tiles) best = sp;
    return best;
}

template <int EPI, typename TO, int NT>
int launch(const void* x, const void* w, const void* bias, int bias_dtype, void* out, int M, int N, int K, cudaStream_t s) {
    static std::atomic<bool> configured{false};
    if (!configured) {
        BL_CUDA(cudaFuncSetAttribute(gemm_tc_few_kernel<EPI, TO, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, Ring<NT>::SMEM_BYTES));
        configured = true;
    }
    const bool glu = EPI == BL_EPI_SWIGLU;
    CUtensorMap mx, mw;
    if (bl_make_map_bf16(WHO, &mx, x, M, K, NT, BK)) return 1;
    if (bl_make_map_bf16(WHO, &mw, w, glu ? 2LL * N : N, K, glu ? BN / 2 : BN, BK)) return 1;
    const int units = glu ? BN / 2 : BN, n_tiles = (N + units - 1) / units, split = split_for(n_tiles, (K + BK - 1) / BK);
    if (split > 1) {
        BL_CUDA(bl_launch_dependent_clusters(gemm_tc_few_kernel<EPI, TO, NT>, dim3((unsigned)(n_tiles * split)), dim3(THREADS), (size_t)Ring<NT>::SMEM_BYTES, s,
                                             (unsigned)split, mx, mw, bias, bias_dtype, (TO*)out, M, N, K, split));
    } else {
        const int blocks = n_tiles < bl_device_sms() ? n_tiles : bl_device_sms();
        BL_CUDA(bl_launch_dependent(gemm_tc_few_kernel<EPI, TO, NT>, dim3((unsigned)blocks), dim3(THREADS), (size_t)Ring<NT>::SMEM_BYTES, s,
                                    mx, mw, bias, bias_dtype, (TO*)out, M, N, K, 1));
    }
    BL_CHECK_LAUNCH("bl_gemm_tc_few");
    return 0;
}

template <int EPI, typename TO>
int launch_rows(const void* x, const void* w, const void* bias, int bias_dtype, void* out, int M, int N, int K, cudaStream_t s) {
    return M <= 16 ? launch<EPI, TO, 16>(x, w, bias, bias_dtype, out, M, N, K, s)
         : M <= 32 ? launch<EPI, TO, 32>(x, w, bias, bias_dtype, out, M, N, K, s) : launch<EPI, TO, 64>(x, w, bias, bias_dtype, out, M, N, K, s);
}

}  // namespace

// The blocks of this kernel's launch (the blocks of clusters where tiles are shared, else one a tile, the SMs walk them in rounds).
extern "C" int bl_gemm_tc_few_blocks(int N, int K, int epilogue) {
    const int units = epilogue == BL_EPI_SWIGLU ? BN / 2 : BN, n_tiles = (N + units - 1) / units;
    return n_tiles * split_for(n_tiles, (K + BK - 1) / BK);
}

extern "C" int bl_gemm_tc_few_supported(int M, int N, int K) { return M >= 1 && M <= 64 && N >= 1 && K >= 8 && K % 8 == 0; }

extern "C" int bl_gemm_tc_few(const void* x, const void* w, const void* bias, int bias_dtype, void* out, int out_dtype, int M, int N, int K,
                              int epilogue, void* stream) {
    if (M <= 0) return 0;
    if (!bl_gemm_tc_few_supported(M, N, K)) BL_FAIL("bl_gemm_tc_few: M=%d N=%d K=%d is not built (up to 64 rows, K a multiple of 8)", M, N, K);
    if (((uintptr_t)x | (uintptr_t)w | (uintptr_t)out) & 15) BL_FAIL("bl_gemm_tc_few: x, W and out must be 16-byte aligned");
    if (epilogue == BL_EPI_BIAS && bias == nullptr) BL_FAIL("bl_gemm_tc_few: bias epilogue without a bias");
    cudaStream_t s = (cudaStream_t)stream;
    if (out_dtype == BL_F32) {
        switch (epilogue) {
            case BL_EPI_NONE: return launch_rows<BL_EPI_NONE, float>(x, w, bias, bias_dtype, out, M, N, K, s);
            case BL_EPI_BIAS: return launch_rows<BL_EPI_BIAS, float>(x, w, bias, bias_dtype, out, M, N, K, s);
            case BL_EPI_RESIDUAL: return launch_rows<BL_EPI_RESIDUAL, float>(x, w, bias, bias_dtype, out, M, N, K, s);
            default: break;
        }
    } else if (out_dtype == BL_BF16 && epilogue == BL_EPI_SWIGLU) {
        return launch_rows<BL_EPI_SWIGLU, __nv_bfloat16>(x, w, bias, bias_dtype, out, M, N, K, s);
    }
    BL_FAIL("bl_gemm_tc_few: epilogue %d with results of type %d is not built", epilogue, out_dtype);
}

// Reads and clears the status word: 0 when no block has given up on a wait (1 loader, 2 issuer, 4 accumulator free, 5 epilogue).
extern "C" int bl_gemm_tc_few_status(int* status) {
    int v = 0, zero = 0;
    BL_CUDA(cudaMemcpyFromSymbol(&v, g_status, sizeof(int)));
    if (v != 0) BL_CUDA(cudaMemcpyToSymbol(g_status, &zero, sizeof(int)));
    *status = v;
    return 0;
}
