// Plain matrix product on CUDA cores: out = epilogue(x . W^T), W stored (outputs x inputs) row-major
// as in the reference's `linear` (src/math.br:66-82) and its tiled GPU kernel LinearKernel
// (src/math_gpu.br:82-135). Every output element accumulates its products in ascending k in one
// 32-bit accumulator, whatever the number of rows, so results do not depend on how a batch is cut.
// This is the product of the 32-bit path where gemm_f32_tc.cu does not take it, and the twin that the
// tensor-core kernels are checked against.
#include "common.cuh"
#include "api.h"

namespace {

constexpr int TM = 64, TN = 64, TK = 16;

template <typename TX, typename TW, typename TO, int EPI>
__global__ void __launch_bounds__(256)
gemm_plain_kernel(const TX* __restrict__ x, const TW* __restrict__ w, const void* __restrict__ bias,
                  int bias_dtype, TO* __restrict__ out, int M, int N, int K, int ldx,
                  const float* __restrict__ coef, int group, float sign, int x_tanh = 0) {
    __shared__ float xs[TK][TM + 1];
    __shared__ float ws[TK][TN + 1];
    __shared__ float us[EPI == BL_EPI_SWIGLU ? TK : 1][TN + 1];
    const int m0 = blockIdx.y * TM, n0 = blockIdx.x * TN;
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;   // 16 x 16 threads, 4 x 4 outputs each
    float acc[4][4] = {};
    float acu[4][4] = {};
    for (int k0 = 0; k0 < K; k0 += TK) {
        for (int i = threadIdx.x; i < TM * TK; i += 256) {
            const int r = i / TK, c = i % TK;
            const int m = m0 + r, k = k0 + c;
            float xv = (m < M && k < K) ? bl_load(x + (size_t)m * ldx + k) : 0.f;
            if (EPI == BL_EPI_DECAY_EXP && x_tanh) xv = tanhf(xv);
            xs[c][r] = xv;
        }
        for (int i = threadIdx.x; i < TN * TK; i += 256) {
            const int r = i / TK, c = i % TK;
            const int n = n0 + r, k = k0 + c;
            const bool ok = n < N && k < K;
            ws[c][r] = ok ? bl_load(w + (size_t)n * K + k) : 0.f;
            if (EPI == BL_EPI_SWIGLU) us[c][r] = ok ? bl_load(w + (size_t)(N + n) * K + k) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < TK; ++k) {
            float a[4], b[4], u[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = xs[k][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = ws[k][tx * 4 + j];
            if (EPI == BL_EPI_SWIGLU) {
#pragma unroll
                for (int j = 0; j < 4; ++j) u[j] = us[k][tx * 4 + j];
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
                    if (EPI == BL_EPI_SWIGLU) acu[i][j] = fmaf(a[i], u[j], acu[i][j]);
                }
        }
        __syncthreads();
    }
    const BlGluArgs glu = bl_glu_args(EPI == BL_EPI_SWIGLU ? bias : nullptr);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = m0 + ty * 4 + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tx * 4 + j;
            if (n >= N) continue;
            TO* dst = out + (size_t)m * N + n;
            float v = acc[i][j];
            if (EPI == BL_EPI_BIAS) v += bl_load_any(bias, bias_dtype, n);
            if (EPI == BL_EPI_RESIDUAL) {
                if (bias) v += bl_load_any(bias, bias_dtype, n);
                v += bl_load(dst);
            }
            if (EPI == BL_EPI_SWIGLU) {
                float u = acu[i][j];
                if (glu.bias) { v += glu.bias[n]; u += glu.bias[N + n]; }
                v = bl_glu(glu.kind, v, u, glu.limit);
            }
            if (EPI == BL_EPI_DECAY) {                 // exp(-coef[head] * softplus(sign * (acc + bias))), head = n / group
                if (bias) v += bl_load_any(bias, bias_dtype, n);
                const float u = sign * v;
                v = expf(-coef[n / group] * (u > 20.f ? u : log1pf(expf(u))));
            }
            if (EPI == BL_EPI_DECAY_EXP) {             // exp(-exp(acc + bias))
                if (bias) v += bl_load_any(bias, bias_dtype, n);
                v = expf(-expf(v));
            }
            bl_store(dst, v);
        }
    }
}

template <typename TX, typename TW, typename TO>
int launch_epi(const void* x, const void* w, const void* bias, int bias_dtype, void* out,
               int M, int N, int K, int ldx, int epi, cudaStream_t s, const float* coef = nullptr, int group = 1, float sign = 1.f, int x_tanh = 0) {
    dim3 grid((N + TN - 1) / TN, (M + TM - 1) / TM);
#define BL_GO(E) gemm_plain_kernel<TX, TW, TO, E><<<grid, 256, 0, s>>>( \
        (const TX*)x, (const TW*)w, bias, bias_dtype, (TO*)out, M, N, K, ldx, coef, group, sign, x_tanh)
    switch (epi) {
        case BL_EPI_NONE: BL_GO(BL_EPI_NONE); break;
        case BL_EPI_BIAS: BL_GO(BL_EPI_BIAS); break;
        case BL_EPI_RESIDUAL: BL_GO(BL_EPI_RESIDUAL); break;
        case BL_EPI_SWIGLU: BL_GO(BL_EPI_SWIGLU); break;
        case BL_EPI_DECAY: BL_GO(BL_EPI_DECAY); break;
        case BL_EPI_DECAY_EXP: BL_GO(BL_EPI_DECAY_EXP); break;
        default: BL_FAIL("bl_gemm_plain: unknown epilogue %d", epi);
    }
#undef BL_GO
    BL_CHECK_LAUNCH("bl_gemm_plain");
    return 0;
}

template <typename TX, typename TW>
int launch_out(const void* x, const void* w, const void* bias, int bias_dtype, void* out, int out_dtype,
               int M, int N, int K, int ldx, int epi, cudaStream_t s) {
    if (out_dtype == BL_F32) return launch_epi<TX, TW, float>(x, w, bias, bias_dtype, out, M, N, K, ldx, epi, s);
    if (out_dtype == BL_BF16) {
        if (epi == BL_EPI_RESIDUAL) BL_FAIL("bl_gemm_plain: the residual stream is 32-bit; output dtype must be float32");
        return launch_epi<TX, TW, __nv_bfloat16>(x, w, bias, bias_dtype, out, M, N, K, ldx, epi, s);
    }
    BL_FAIL("bl_gemm_plain: unknown output dtype %d", out_dtype);
}

// ---- products with a short K (the second factor of a low-rank pair) --------------------------------------------------------
// The same sums (one accumulator an output, ascending k) for 32-bit x and 32-bit results with K up to RANK_MAX: a thread holds a
// row of W in registers and goes down the rows of x, which the block has brought to shared memory (a broadcast each). W is on its
// way before the kernel before has finished (so it must not be that kernel's result: W, bias and coefficients are weights). Tiles of 64 x 64 gave a decode step 16 blocks and no early start (8 rows of 1,024 x
// 16 in a decode step's chain 9.6 us, and 1,840 rows 15 us).
constexpr int RANK_MAX = 64, RANK_THREADS = 128;

template <typename TW, int EPI, int KM>
__global__ void __launch_bounds__(RANK_THREADS)
gemm_rank_kernel(const float* __restrict__ x, const TW* __restrict__ w, const void* __restrict__ bias, int bias_dtype, float* __restrict__ out,
                 int M, int N, int K, int ldx, const float* __restrict__ coef, int group, float sign, int x_tanh, int rows) {
    extern __shared__ __align__(16) float xrow[];                 // [rows][K]
    bl_pdl_trigger();
    const int n = blockIdx.x * RANK_THREADS + threadIdx.x, m0 = blockIdx.y * rows;
    float wr[KM];
#pragma unroll
    for (int k = 0; k < KM; k += 4) {
        if (n < N && k < K) {                                     // K is a multiple of four
            if constexpr (sizeof(TW) == 4) {
                const float4 f = *reinterpret_cast<const float4*>(w + (size_t)n * K + k);
                wr[k] = f.x; wr[k + 1] = f.y; wr[k + 2] = f.z; wr[k + 3] = f.w;
            } else {
                const uint2 u = *reinterpret_cast<const uint2*>(w + (size_t)n * K + k);
                const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x)), b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
                wr[k] = a.x; wr[k + 1] = a.y; wr[k + 2] = b.x; wr[k + 3] = b.y;
            }
        } else {
            wr[k] = wr[k + 1] = wr[k + 2] = wr[k + 3] = 0.f;
        }
    }
    const float bn = bias != nullptr && n < N ? bl_load_any(bias, bias_dtype, n) : 0.f;
    const float cn = EPI == BL_EPI_DECAY && n < N ? coef[n / group] : 0.f;
    bl_pdl_wait();
    const int here = min(rows, M - m0), k4 = K >> 2;
    for (int c = threadIdx.x; c < here * k4; c += RANK_THREADS) {
        float4 f = *reinterpret_cast<const float4*>(x + (size_t)(m0 + c / k4) * ldx + (c % k4) * 4);
        if (EPI == BL_EPI_DECAY_EXP && x_tanh) f = make_float4(tanhf(f.x), tanhf(f.y), tanhf(f.z), tanhf(f.w));
        *reinterpret_cast<float4*>(xrow + 4 * c) = f;
    }
    __syncthreads();
    if (n >= N) return;
#pragma unroll 2
    for (int i = 0; i < here; ++i) {
        float acc = 0.f;
#pragma unroll
        for (int k = 0; k < KM; k += 4) {
            if (k < K) {
                const float4 f = *reinterpret_cast<const float4*>(xrow + i * K + k);
                acc = fmaf(f.x, wr[k], acc); acc = fmaf(f.y, wr[k + 1], acc); acc = fmaf(f.z, wr[k + 2], acc); acc = fmaf(f.w, wr[k + 3], acc);
            }
        }
        float v = acc;
        if (EPI != BL_EPI_NONE && bias) v += bn;
        if (EPI == BL_EPI_DECAY) {
            const float u = sign * v;
            v = expf(-cn * (u > 20.f ? u : log1pf(expf(u))));
        }
        if (EPI == BL_EPI_DECAY_EXP) v = expf(-expf(v));
        out[(size_t)(m0 + i) * N + n] = v;
    }
}

template <typename TW, int EPI>
int launch_rank(const float* x, const TW* w, const void* bias, int bias_dtype, float* out, int M, int N, int K, int ldx, cudaStream_t s,
                const float* coef, int group, float sign, int x_tanh) {
    // rows a block: up to 16, fewer where the launch would not give every SM four blocks
    const int across = (N + RANK_THREADS - 1) / RANK_THREADS;
    int rows = 16;
    while (rows > 1 && (long long)across * ((M + rows - 1) / rows) < 4 * bl_device_sms()) rows >>= 1;
    const dim3 grid(across, (M + rows - 1) / rows);
    const size_t bytes = (size_t)rows * K * sizeof(float);
#define BL_GO(KM) BL_CUDA(bl_launch_dependent(gemm_rank_kernel<TW, EPI, KM>, grid, dim3(RANK_THREADS), bytes, s, x, w, bias, bias_dtype, out, \
        M, N, K, ldx, coef, group, sign, x_tanh, rows))
    if (K <= 16) BL_GO(16); else if (K <= 32) BL_GO(32); else BL_GO(64);
#undef BL_GO
    BL_CHECK_LAUNCH("bl_gemm_plain (short K)");
    return 0;
}

// Short K, whole 16-byte pieces of x and four values of W (the sums are the same either way).
template <typename TW>
bool rank_fits(const float* x, const TW* w, int M, int K, int ldx) {
    return K <= RANK_MAX && K % 4 == 0 && ldx % 4 == 0 && ((uintptr_t)x & 15) == 0 && ((uintptr_t)w & (4 * sizeof(TW) - 1)) == 0 && M <= 65535;
}

// ---- the 32-bit product with tiles in flight ---------------------------------------------------------------------------
// The same sums (one accumulator an output, ascending k, so the same bits as the kernel above and independent of the tile)
// for 32-bit x and W whose rows are whole 16-byte pieces: BK values of k of a tile's rows come by cp.async into a ring of
// three stages as they lie in memory, rows padded by 16 bytes so that the eight rows that lanes of a quarter warp read
// fall on different banks; a thread's TR x TC outputs lie (rows, columns of threads) apart, so its operands are 16-byte
// loads of four k each. With SWIGLU the tile's upper half of W rows are the up rows, and a thread holds both sums of a unit.
// Bound by the FMA pipes for many rows (41 TFLOP/s at 2,048 rows; FMAs with three register operands reach 59 of the pipes'
// 74), by W's bytes for few.
template <int BM, int BN, int TR, int TC, int EPI>
__global__ void __launch_bounds__((BM / TR) * (BN / TC))
gemm_f32_kernel(const float* __restrict__ x, const float* __restrict__ w, const void* __restrict__ bias, int bias_dtype,
                float* __restrict__ out, int M, int N, int K, int ldx) {
    constexpr int THREADS = (BM / TR) * (BN / TC), BK = 32, LD = BK + 4, STAGES = 3, GR = BM / TR, GC = BN / TC;
    constexpr bool GLU = EPI == BL_EPI_SWIGLU;
    constexpr int COLS = GLU ? BN / 2 : BN;               // outputs a row of the tile
    static_assert(GC % 8 == 0 && GR % 4 == 0, "a warp is 4 rows of 8 threads");
    extern __shared__ __align__(16) float ring[];         // [STAGES][BM + BN][LD]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tx = (warp % (GC / 8)) * 8 + (lane & 7), ty = (warp / (GC / 8)) * 4 + (lane >> 3);
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * COLS;
    bl_pdl_wait();
    auto fetch = [&](int k0, float* stage) {
#pragma unroll 4
        for (int c = tid; c < (BM + BN) * (BK / 4); c += THREADS) {
            const int row = c / (BK / 4), k = k0 + (c % (BK / 4)) * 4;
            const float* src;
            bool ok = k < K;
            if (row < BM) {
                ok = ok && m0 + row < M;
                src = x + (size_t)(ok ? m0 + row : 0) * ldx + (ok ? k : 0);
            } else {
                const int j = row - BM, n = n0 + (GLU && j >= COLS ? j - COLS : j);
                ok = ok && n < N;
                src = w + (size_t)(ok ? (GLU && j >= COLS ? N + n : n) : 0) * K + (ok ? k : 0);
            }
            const unsigned dst = (unsigned)__cvta_generic_to_shared(stage + row * LD + (c % (BK / 4)) * 4);
            const int bytes = ok ? 16 : 0;                // 0: the piece is filled with zeros
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" :: "r"(dst), "l"(src), "r"(bytes));
        }
        asm volatile("cp.async.commit_group;\n" ::);
    };
    float acc[TR][TC];
#pragma unroll
    for (int i = 0; i < TR; ++i)
#pragma unroll
        for (int j = 0; j < TC; ++j) acc[i][j] = 0.f;
    const int steps = (K + BK - 1) / BK;
    fetch(0, ring);
    if (steps > 1) fetch(BK, ring + (BM + BN) * LD);
    else asm volatile("cp.async.commit_group;\n" ::);
    for (int s = 0; s < steps; ++s) {
        asm volatile("cp.async.wait_group 1;\n" ::);
        __syncthreads();                                  // stage s has landed; everybody is through with stage s - 1
        if (s + 2 < steps) fetch((s + 2) * BK, ring + (s + 2) % STAGES * (BM + BN) * LD);
        else asm volatile("cp.async.commit_group;\n" ::);
        const float* xs = ring + s % STAGES * (BM + BN) * LD + ty * LD;
        const float* ws = ring + s % STAGES * (BM + BN) * LD + (BM + tx) * LD;
#pragma unroll
        for (int k = 0; k < BK; k += 4) {
            float4 a[TR];
#pragma unroll
            for (int i = 0; i < TR; ++i) a[i] = *reinterpret_cast<const float4*>(xs + i * GR * LD + k);
#pragma unroll
            for (int j = 0; j < TC; ++j) {
                const float4 b = *reinterpret_cast<const float4*>(ws + j * GC * LD + k);
#pragma unroll
                for (int i = 0; i < TR; ++i) {
                    acc[i][j] = fmaf(a[i].x, b.x, acc[i][j]);
                    acc[i][j] = fmaf(a[i].y, b.y, acc[i][j]);
                    acc[i][j] = fmaf(a[i].z, b.z, acc[i][j]);
                    acc[i][j] = fmaf(a[i].w, b.w, acc[i][j]);
                }
            }
        }
    }
    bl_pdl_trigger();
    const BlGluArgs glu = bl_glu_args(GLU ? bias : nullptr);
#pragma unroll
    for (int i = 0; i < TR; ++i) {
        const int m = m0 + ty + i * GR;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < (GLU ? TC / 2 : TC); ++j) {
            const int n = n0 + tx + j * GC;
            if (n >= N) continue;
            float* dst = out + (size_t)m * N + n;
            float v = acc[i][j];
            if (EPI == BL_EPI_BIAS) v += bl_load_any(bias, bias_dtype, n);
            if (EPI == BL_EPI_RESIDUAL) {
                if (bias) v += bl_load_any(bias, bias_dtype, n);
                v += *dst;
            }
            if (GLU) {
                float u = acc[i][GLU ? j + TC / 2 : j];
                if (glu.bias) { v += glu.bias[n]; u += glu.bias[N + n]; }
                v = bl_glu(glu.kind, v, u, glu.limit);
            }
            *dst = v;
        }
    }
}

template <int BM, int BN, int TR, int TC>
int launch_f32(const float* x, const float* w, const void* bias, int bias_dtype, float* out, int M, int N, int K, int ldx, int epi,
               cudaStream_t s) {
    const int cols = epi == BL_EPI_SWIGLU ? BN / 2 : BN;
    const dim3 grid((N + cols - 1) / cols, (M + BM - 1) / BM), block((BM / TR) * (BN / TC));
    constexpr size_t bytes = (size_t)3 * (BM + BN) * 36 * sizeof(float);
#define BL_GO(E) do { \
        static thread_local bool allowed = false; \
        if (!allowed) { BL_CUDA(cudaFuncSetAttribute(gemm_f32_kernel<BM, BN, TR, TC, E>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes)); allowed = true; } \
        BL_CUDA(bl_launch_dependent(gemm_f32_kernel<BM, BN, TR, TC, E>, grid, block, bytes, s, x, w, bias, bias_dtype, out, M, N, K, ldx)); } while (0)
    switch (epi) {
        case BL_EPI_NONE: BL_GO(BL_EPI_NONE); break;
        case BL_EPI_BIAS: BL_GO(BL_EPI_BIAS); break;
        case BL_EPI_RESIDUAL: BL_GO(BL_EPI_RESIDUAL); break;
        default: BL_GO(BL_EPI_SWIGLU); break;
    }
#undef BL_GO
    BL_CHECK_LAUNCH("bl_gemm_plain (32-bit tiles)");
    return 0;
}

// Which tile: the least of ceil(blocks / SMs) blocks in a row at a tile's pace, but no less than one block alone takes
// (microseconds for 896 values of k, measured at 1 to 2,048 rows of six products; the ratio of K scales both). Few rows
// are bound by a block's chain of stages, many by the FMA pipes: 366 rows of 896 x 4,864 take 145 us in 32 x 32 tiles,
// 188 in 64 x 32 (the kernel above: 914); 2,048 rows of 11,008 + 11,008 x 2,048 4.5 ms in 64 x 32, 5.8 in 32 x 32
// (8.0; 41 TFLOP/s of the 59 that dependent FMAs with three operands reach here); one row of 151,936 x 896 101 us in
// 4 x 64 (860; 5.4 TB/s). Tiles of 64 x 64, 128 x 64 and 128 x 128 were no faster at any of these sizes.
// A successor is let in when the sums are done: let in at the start, its waiting blocks pile up on the SMs that this launch
// leaves empty and it runs at the pace of those (366 rows of 896 x 4,864: 193 us).
struct F32Tile { int bm, bn; float alone, pace; };
constexpr F32Tile F32_TILES[] = {{64, 32, 18.5f, 13.2f}, {32, 32, 11.8f, 8.3f}, {16, 64, 12.8f, 9.4f},
                                 {16, 32, 9.3f, 6.4f}, {4, 64, 11.8f, 5.9f}, {4, 16, 6.8f, 1.95f}};

int launch_f32_tiles(const float* x, const float* w, const void* bias, int bias_dtype, float* out, int M, int N, int K, int ldx, int epi,
                     cudaStream_t s) {
    int best = 0;
    float best_us = 0.f;
    const int sms = bl_device_sms();
    for (int v = 0; v < (int)(sizeof(F32_TILES) / sizeof(F32_TILES[0])); ++v) {
        const F32Tile& t = F32_TILES[v];
        const int cols = epi == BL_EPI_SWIGLU ? t.bn / 2 : t.bn;
        const long long down = (M + t.bm - 1) / t.bm, blocks = (long long)((N + cols - 1) / cols) * down;
        if (down > 65535) continue;
        const float us = fmaxf(t.alone, (float)((blocks + sms - 1) / sms) * t.pace);
        if (best_us == 0.f || us < best_us) { best = v; best_us = us; }
    }
    switch (best) {
        case 0: return launch_f32<64, 32, 4, 4>(x, w, bias, bias_dtype, out, M, N, K, ldx, epi, s);
        case 1: return launch_f32<32, 32, 4, 2>(x, w, bias, bias_dtype, out, M, N, K, ldx, epi, s);
        case 2: return launch_f32<16, 64, 4, 2>(x, w, bias, bias_dtype, out, M, N, K, ldx, epi, s);
        case 3: return launch_f32<16, 32, 2, 2>(x, w, bias, bias_dtype, out, M, N, K, ldx, epi, s);
        case 4: return launch_f32<4, 64, 1, 2>(x, w, bias, bias_dtype, out, M, N, K, ldx, epi, s);
        default: return launch_f32<4, 16, 1, 2>(x, w, bias, bias_dtype, out, M, N, K, ldx, epi, s);
    }
}

// 32-bit rows of whole 16-byte pieces; everything else, bfloat16 and the decays' epilogues take the kernel above.
bool f32_tiles_fit(const void* x, const void* w, int K, int ldx, int epi, int out_dtype) {
    return out_dtype == BL_F32 && K % 4 == 0 && ldx % 4 == 0 && (((uintptr_t)x | (uintptr_t)w) & 15) == 0 &&
           (epi == BL_EPI_NONE || epi == BL_EPI_BIAS || epi == BL_EPI_RESIDUAL || epi == BL_EPI_SWIGLU);
}

}  // namespace

extern "C" int bl_gemm_plain(const void* x, int x_dtype, const void* w, int w_dtype, const void* bias,
                             int bias_dtype, void* out, int out_dtype, int M, int N, int K, int epilogue,
                             void* stream) {
    return bl_gemm_plain_ld(x, x_dtype, K, w, w_dtype, bias, bias_dtype, out, out_dtype, M, N, K, epilogue, stream);
}

extern "C" int bl_gemm_plain_ld(const void* x, int x_dtype, int ldx, const void* w, int w_dtype, const void* bias,
                                int bias_dtype, void* out, int out_dtype, int M, int N, int K, int epilogue,
                                void* stream) {
    if (M <= 0) return 0;
    if (ldx < K) BL_FAIL("bl_gemm_plain: rows of x are %d apart but hold %d values", ldx, K);
    if (N <= 0 || K <= 0) BL_FAIL("bl_gemm_plain: bad sizes N=%d K=%d", N, K);
    if (epilogue == BL_EPI_BIAS && bias == nullptr) BL_FAIL("bl_gemm_plain: bias epilogue without a bias");
    if (epilogue == BL_EPI_BIAS && bias_dtype != BL_F32 && bias_dtype != BL_BF16)
        BL_FAIL("bl_gemm_plain: unknown bias dtype %d", bias_dtype);
    cudaStream_t s = (cudaStream_t)stream;
    if (x_dtype == BL_F32 && w_dtype == BL_F32 && f32_tiles_fit(x, w, K, ldx, epilogue, out_dtype))
        return launch_f32_tiles((const float*)x, (const float*)w, bias, bias_dtype, (float*)out, M, N, K, ldx, epilogue, s);
    if (x_dtype == BL_F32 && w_dtype == BL_F32)
        return launch_out<float, float>(x, w, bias, bias_dtype, out, out_dtype, M, N, K, ldx, epilogue, s);
    if (x_dtype == BL_BF16 && w_dtype == BL_BF16)
        return launch_out<__nv_bfloat16, __nv_bfloat16>(x, w, bias, bias_dtype, out, out_dtype, M, N, K, ldx, epilogue, s);
    if (x_dtype == BL_F32 && w_dtype == BL_BF16 && out_dtype == BL_F32 && (epilogue == BL_EPI_NONE || epilogue == BL_EPI_BIAS) &&
        rank_fits((const float*)x, (const __nv_bfloat16*)w, M, K, ldx)) {
        const float* xf = (const float*)x;
        const __nv_bfloat16* wb = (const __nv_bfloat16*)w;
        if (epilogue == BL_EPI_NONE) return launch_rank<__nv_bfloat16, BL_EPI_NONE>(xf, wb, nullptr, 0, (float*)out, M, N, K, ldx, s, nullptr, 1, 1.f, 0);
        return launch_rank<__nv_bfloat16, BL_EPI_BIAS>(xf, wb, bias, bias_dtype, (float*)out, M, N, K, ldx, s, nullptr, 1, 1.f, 0);
    }
    if (x_dtype == BL_F32 && w_dtype == BL_BF16)
        return launch_out<float, __nv_bfloat16>(x, w, bias, bias_dtype, out, out_dtype, M, N, K, ldx, epilogue, s);
    BL_FAIL("bl_gemm_plain: unsupported input dtypes x=%d w=%d", x_dtype, w_dtype);
}

// out[m, n] = exp(-coef[n / group] * softplus(sign * (x[m, :] . W[n, :] + bias[n]))), 32-bit: the decays of a linear
// recurrence from their pre-activation, as the epilogue of the product that makes it (x 32-bit rows ldx apart).
extern "C" int bl_gemm_plain_decay(const float* x, int ldx, const void* w, int w_dtype, const void* bias, int bias_dtype,
                                   float* out, int M, int N, int K, const float* coef, int group, float sign, void* stream) {
    if (M <= 0) return 0;
    if (N <= 0 || K <= 0 || ldx < K || group <= 0 || N % group != 0 || coef == nullptr)
        BL_FAIL("bl_gemm_plain_decay: bad sizes N=%d K=%d ldx=%d group=%d", N, K, ldx, group);
    cudaStream_t s = (cudaStream_t)stream;
    if (w_dtype == BL_F32 && rank_fits(x, (const float*)w, M, K, ldx))
        return launch_rank<float, BL_EPI_DECAY>(x, (const float*)w, bias, bias_dtype, out, M, N, K, ldx, s, coef, group, sign, 0);
    if (w_dtype == BL_F32) return launch_epi<float, float, float>(x, w, bias, bias_dtype, out, M, N, K, ldx, BL_EPI_DECAY, s, coef, group, sign);
    if (w_dtype == BL_BF16 && rank_fits(x, (const __nv_bfloat16*)w, M, K, ldx))
        return launch_rank<__nv_bfloat16, BL_EPI_DECAY>(x, (const __nv_bfloat16*)w, bias, bias_dtype, out, M, N, K, ldx, s, coef, group, sign, 0);
    if (w_dtype == BL_BF16) return launch_epi<float, __nv_bfloat16, float>(x, w, bias, bias_dtype, out, M, N, K, ldx, BL_EPI_DECAY, s, coef, group, sign);
    BL_FAIL("bl_gemm_plain_decay: unknown matrix dtype %d", w_dtype);
}

// out[m, n] = exp(-exp(u[m, :] . W[n, :] + bias[n])), u = tanh(x) where x_tanh != 0, else x (32-bit rows ldx apart): decays
// whose pre-activation is a product in two factors with a tanh between them, as the epilogue of the second factor.
extern "C" int bl_gemm_plain_decay_exp(const float* x, int ldx, int x_tanh, const void* w, int w_dtype, const void* bias, int bias_dtype,
                                       float* out, int M, int N, int K, void* stream) {
    if (M <= 0) return 0;
    if (N <= 0 || K <= 0 || ldx < K) BL_FAIL("bl_gemm_plain_decay_exp: bad sizes N=%d K=%d ldx=%d", N, K, ldx);
    cudaStream_t s = (cudaStream_t)stream;
    if (w_dtype == BL_F32 && rank_fits(x, (const float*)w, M, K, ldx))
        return launch_rank<float, BL_EPI_DECAY_EXP>(x, (const float*)w, bias, bias_dtype, out, M, N, K, ldx, s, nullptr, 1, 1.f, x_tanh);
    if (w_dtype == BL_F32) return launch_epi<float, float, float>(x, w, bias, bias_dtype, out, M, N, K, ldx, BL_EPI_DECAY_EXP, s, nullptr, 1, 1.f, x_tanh);
    if (w_dtype == BL_BF16 && rank_fits(x, (const __nv_bfloat16*)w, M, K, ldx))
        return launch_rank<__nv_bfloat16, BL_EPI_DECAY_EXP>(x, (const __nv_bfloat16*)w, bias, bias_dtype, out, M, N, K, ldx, s, nullptr, 1, 1.f, x_tanh);
    if (w_dtype == BL_BF16) return launch_epi<float, __nv_bfloat16, float>(x, w, bias, bias_dtype, out, M, N, K, ldx, BL_EPI_DECAY_EXP, s, nullptr, 1, 1.f, x_tanh);
    BL_FAIL("bl_gemm_plain_decay_exp: unknown matrix dtype %d", w_dtype);
}
