// The 32-bit product on the fifth-generation tensor cores: out[M, N] = epilogue(x[M, K] . W[N, K]^T), 32-bit operands and results.
//
// A 32-bit number has 24 significant bits. It is split into three bfloat16 numbers of 8 (each the rest so far rounded to nearest;
// Henry, Tang and Heinecke, "Leveraging the bfloat16 artificial intelligence datatype for higher-precision computations", 2019), whose
// sum IS the number. Of the nine products of two such triples all but the last (2^-32 of the whole at most) are made, each exact.
// The tensor cores add into a 32-bit accumulator, but they cut bits off where a register's addition rounds, an error that has a sign
// and grows with the number of additions. So the first parts' products have an accumulator of their own, which holds one of them exactly,
// for 32 values of k at a time: threads add such segments up in registers, rounded to nearest, in ascending k. The other products,
// 2^-8 of those, stay in a second accumulator, which is added at the end. A product alone is then rounded as an FMA rounds it, and
// K = 896 makes 29 rounded additions where a chain of FMAs makes 896. Errors against 64 bits are no larger than such a chain's, of
// rows with a few numbers as of full ones (the tests of this kernel have both).
//
// W is the M side of the MMA (128 rows of W a tile; with SWIGLU 64 gate rows and the 64 up rows that match) and NT rows of x its
// N side. A block: TMA brings 32 values of k of the tile's rows into a ring; 8 warps split them and store the parts where the MMAs
// read them (64-byte swizzle); a warp of its own issues the segment's MMAs into one of two accumulators (and the one of the small
// products) and refills the ring; 4 or 8 warps add the other accumulator to their registers. (Rows fetched ahead into the splitters' own
// registers cannot be: the fence that shows their stores to the tensor cores waits for every load under way, 1,600 cycles a
// segment.) At the end the tile passes through shared memory to the epilogue. Products of few tiles cut K over the blocks of a
// cluster (f32_tc_spans), whose totals are added in ascending k through distributed shared memory. What a result is computed from, and
// in which order, depends on N and K only: it is the same whatever rows stand beside a row and however wide a tile is (the same promise
// that the kernels in gemm_plain.cu make, which keep the small products, rows that are no whole 16-byte pieces, and steps that are
// asked to do without tensor cores).
// A sum that is not finite (an infinity or NaN among the inputs, or an overflow) is worked out again as a chain of FMAs over the
// inputs themselves. So is a small one, |sum| < 2^-48, of a row of x or of W with an operand other than 0 below 2^-50: the parts of such
// operands may lie below bfloat16's smallest numbers (an operand from 2^-110 on loses nothing, a smaller one 2^-134 at most), and
// products of them below 32-bit ones. With the other operand under 2^40 (else the row's every sum is worked out again) that is
// less than 2^-24 of any larger sum.
//
// Bound by the splitting: 8.5 instructions a number in chains, at 54 % of the issue slots (366 rows below), beside shared memory, which
// takes a segment as it comes once, its parts (6 bytes a number) once, and gives them to the eight MMAs of each 16 values of k. Issued by a warp that splits as well, the MMAs held up the next segment's splitting (4,864 +
// 4,864 x 896: 1 row 27.3 us, 366 rows 89). Microseconds, FMAs (gemm_plain.cu) -> this:
//   rows                          1             16            128           366           2,048
//   1,152 x 896, bias             7.8 -> 7.7    8.7 -> 8.1    19.7 -> 18.8   31 -> 26     118 -> 75
//   896 x 896, residual           7.7 -> 7.8    8.8 -> 8.1    17.8 -> 10.5   33 -> 15     110 -> 64
//   4,864 + 4,864 x 896, gated   13.6 -> 23.7    25 -> 24.2     71 -> 36    178 -> 69     876 -> 308
//   896 x 4,864, residual          55 -> 31      48 -> 31.3     84 -> 34    158 -> 42     557 -> 179
// Up to some ten rows, which FMAs take as fast as W streams, the widest products (from 73 tiles on, whose K is not cut) are slower than
// before: one row of 11,008 + 11,008 x 2,048 57 -> 104, of 18,944 + 18,944 x 3,584 120 -> 181. The other products of a layer make up for
// it (a layer's four, one row: 0.5B sizes 83 -> 70, 3B 230 -> 201, 7B 421 -> 366), and one kernel for all numbers of rows is what
// keeps a row's bits.
// Every wait on an mbarrier is bounded; when a bound runs out the block records a code in a status word and stops computing, but
// still meets its cluster, frees its tensor memory and returns (bl_gemm_f32_tc_status).
#include "tcgen05.cuh"
#include <atomic>

namespace {

constexpr int BM = 128;                    // rows of W a tile
constexpr int MAX_COLUMNS = 1 << 15;       // more: an output head
constexpr int BK = 32;                     // values of k a segment: rows of 128 bytes as they come, 64 bytes a part
constexpr int SPLITTERS = 256, ADDERS = 256, THREADS = SPLITTERS + ADDERS + 32;    // the last warp issues
constexpr float SMALL_SUM = 3.5527136788005009e-15f;          // 2^-48
constexpr uint32_t SMALL_OPERAND = (127u - 50u) << 24;         // 2^-50, its bits without the sign, doubled
constexpr float HUGE_OPERAND = 1099511627776.f;                // 2^40
constexpr uint32_t WAIT_LIMIT = 1u << 22;

template <int NT>
struct Tile {
    static constexpr int RAW_W = BM * 128, RAW_BYTES = RAW_W + NT * 128;  // a segment as it comes
    static constexpr int W_BYTES = BM * 64, X_BYTES = NT * 64, PART_BYTES = 3 * (W_BYTES + X_BYTES);     // and in parts: W's three, x's three
    static constexpr int PARTS = NT >= 64 ? 2 : 3;                        // stages of parts
    static constexpr int RAWS = NT == 128 ? 3 : NT >= 64 ? 4 : 5;         // stages of the ring
    static constexpr int TMEM_COLS = NT >= 96 ? 512 : 4 * NT;             // three accumulators of NT columns
    static constexpr int HALVES = NT >= 64 ? 2 : 1;                       // the columns are dealt to one or two groups of four adder warps
    static constexpr int COLS = NT / HALVES;
    static constexpr int CHUNKS = 4 + (NT + 31) / 32;                     // 16-byte pieces of a segment a splitter
    static constexpr int OFF_RAW = PARTS * PART_BYTES, OFF_BARS = OFF_RAW + RAWS * RAW_BYTES, OFF_MARKS = OFF_BARS + 256;
    static constexpr int SMEM_BYTES = OFF_MARKS + BM + NT + 1024;
    static_assert(NT % 16 == 0 && COLS % 16 == 0 && 2 * BM * NT * 4 <= OFF_BARS && SMEM_BYTES <= 227 * 1024, "tile");
};

__device__ int g_status = 0;               // 0 = fine; else the code of the first wait that ran out

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* give_up, int code) {
    return mbar_wait_bounded(bar, parity, WAIT_LIMIT, give_up, &g_status, code);
}
// Operand tile of rows of 64 bytes (32 bfloat16 values of k) with 64-byte swizzle: groups of 8 rows 512 bytes apart.
__device__ __forceinline__ uint64_t smem_desc64(uint32_t addr) {
    const uint32_t lo = ((addr >> 4) & 0x3FFFu) | (1u << 16);
    const uint32_t hi = (512u >> 4) | (1u << 14) | (4u << 29);
    return ((uint64_t)hi << 32) | lo;
}
// The next parts of two numbers as a pair, and what is left of them.
__device__ __forceinline__ uint32_t next_parts(float& a, float& b) {
    const __nv_bfloat162 p = __floats2bfloat162_rn(a, b);
    const uint32_t u = *reinterpret_cast<const uint32_t*>(&p);
    a -= __uint_as_float(u << 16);
    b -= __uint_as_float(u & 0xffff0000u);
    return u;
}
__device__ __forceinline__ float ld_cluster(uint32_t addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}
// The sum as a chain of FMAs in ascending k.
__device__ __noinline__ float plain_dot(const float* x, const float* w, int K) {
    float acc = 0.f;
    for (int k = 0; k < K; ++k) acc = fmaf(x[k], w[k], acc);
    return acc;
}

template <int EPI, int NT>
__global__ void __launch_bounds__(THREADS, 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const float* __restrict__ x,
                   const float* __restrict__ w, const void* __restrict__ bias, int bias_dtype, float* __restrict__ out, int M, int N, int K,
                   int ldx, int spans, int m_tiles) {
    using T = Tile<NT>;
    constexpr bool GLU = EPI == BL_EPI_SWIGLU;
    constexpr int UNITS = GLU ? BM / 2 : BM;                              // outputs of a row of x a tile
    constexpr int PARTS = T::PARTS, RAWS = T::RAWS;
    // D 32-bit, A and B bfloat16 and K-major, N >> 3 at bit 17, M >> 4 at bit 24
    constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(NT >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
    extern __shared__ unsigned char smem_raw[];
    if (threadIdx.x == 0) { tma_prefetch_map(&map_x); tma_prefetch_map(&map_w); }
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    unsigned char* smem = smem_raw + (base - smem_u32(smem_raw));
    const uint32_t raw_full0 = base + T::OFF_BARS, raw_read0 = raw_full0 + 8 * RAWS, full0 = raw_read0 + 8 * RAWS, empty0 = full0 + 8 * PARTS,
                   sum0 = empty0 + 8 * PARTS, taken0 = sum0 + 16;
    volatile int* give_up = reinterpret_cast<volatile int*>(smem + T::OFF_BARS + 192);
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem + T::OFF_BARS + 200);
    int* any_small = reinterpret_cast<int*>(smem + T::OFF_BARS + 208);    // whether a row of the tile has a small operand
    unsigned char* marks = smem + T::OFF_MARKS;                           // of the tile's rows of W and then of x: 1 a small operand, 2 a huge one
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    // a cluster is the spans of one tile; the tiles of rows are neighbours, so that a tile of W is fetched from memory once
    const int span = blockIdx.x % spans, tile = blockIdx.x / spans;
    const int m0 = tile % m_tiles * NT, n0 = tile / m_tiles * UNITS;
    const int all = (K + BK - 1) / BK, each = (all + spans - 1) / spans;
    const int first = min(span * each, all), steps = min(each, all - first);
    if (threadIdx.x == 0) {
        *give_up = 0;
        *any_small = 0;
        for (int s = 0; s < RAWS; ++s) { mbar_init(raw_full0 + 8 * s, 1); mbar_init(raw_read0 + 8 * s, SPLITTERS / 32); }
        for (int s = 0; s < PARTS; ++s) { mbar_init(full0 + 8 * s, SPLITTERS / 32); mbar_init(empty0 + 8 * s, 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(sum0 + 8 * b, 1); mbar_init(taken0 + 8 * b, 4 * T::HALVES); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    auto load_w = [&](int s) {                                             // and announce the segment's bytes
        const uint32_t bar = raw_full0 + 8 * (s % RAWS), dst = base + T::OFF_RAW + s % RAWS * T::RAW_BYTES;
        mbar_expect_tx(bar, T::RAW_BYTES);
        tma_load_2d(dst, &map_w, bar, (first + s) * BK, n0);
        if (GLU) tma_load_2d(dst + T::RAW_W / 2, &map_w, bar, (first + s) * BK, N + n0);
    };
    auto load_x = [&](int s) {
        tma_load_2d(base + T::OFF_RAW + s % RAWS * T::RAW_BYTES + T::RAW_W, &map_x, raw_full0 + 8 * (s % RAWS), (first + s) * BK, m0);
    };
    const int early = min(RAWS, steps);
    if (warp == 16 && elect_one())                                         // W does not depend on the kernel before this one
        for (int s = 0; s < early; ++s) load_w(s);
    __syncwarp();
    if (warp == 8) {
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     :: "r"(smem_u32((const void*)tmem_slot)), "r"(T::TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = *tmem_slot;
    bool ok = true;
    float* sums = reinterpret_cast<float*>(smem);                          // in the end: [first products, small ones][column][row of the tile]
    bl_pdl_wait();
    bl_pdl_trigger();

    if (warp == 16) {
        // ================= the segments' MMAs and copies
        int issued = early;
        if (elect_one())
            for (int s = 0; s < early; ++s) load_x(s);
        __syncwarp();
        for (int s = 0; s < steps; ++s) {
            const int rs = s % RAWS, st = s % PARTS, b = s & 1;
            ok = mbar_wait(full0 + 8 * st, (uint32_t)((s / PARTS) & 1), give_up, 2);
            if (ok && s >= 2) ok = mbar_wait(taken0 + 8 * b, (uint32_t)((s / 2 - 1) & 1), give_up, 2);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            if (elect_one()) {
                fence_after_sync();
                const uint32_t stage = base + st * T::PART_BYTES, sum = tmem + b * NT, rest = tmem + 2 * NT;
                const uint64_t w1 = smem_desc64(stage), w2 = smem_desc64(stage + T::W_BYTES), w3 = smem_desc64(stage + 2 * T::W_BYTES);
                const uint64_t x1 = smem_desc64(stage + 3 * T::W_BYTES), x2 = smem_desc64(stage + 3 * T::W_BYTES + T::X_BYTES),
                               x3 = smem_desc64(stage + 3 * T::W_BYTES + 2 * T::X_BYTES);
#pragma unroll
                for (int k = 0; k < BK / 8; k += 2) {                  // 16 values of k, two 16-byte units of a descriptor
                    umma_bf16(sum, w1 + k, x1 + k, IDESC, k != 0);
                    umma_bf16(rest, w1 + k, x2 + k, IDESC, (s | k) != 0);
                    umma_bf16(rest, w1 + k, x3 + k, IDESC, 1);
                    umma_bf16(rest, w2 + k, x1 + k, IDESC, 1);
                    umma_bf16(rest, w2 + k, x2 + k, IDESC, 1);
                    umma_bf16(rest, w2 + k, x3 + k, IDESC, 1);
                    umma_bf16(rest, w3 + k, x1 + k, IDESC, 1);
                    umma_bf16(rest, w3 + k, x2 + k, IDESC, 1);
                }
                umma_commit(empty0 + 8 * st);
                umma_commit(sum0 + 8 * b);
            }
            __syncwarp();
            if (s + RAWS < steps) {                                        // the ring's stage takes the segment RAWS on
                ok = mbar_wait(raw_read0 + 8 * rs, (uint32_t)((s / RAWS) & 1), give_up, 2);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                if (elect_one()) { load_w(s + RAWS); load_x(s + RAWS); }
                __syncwarp();
                issued = s + RAWS + 1;
            }
        }
        if (*give_up)                                                      // let our own copies land before leaving
            for (int s = max(0, issued - RAWS); s < issued; ++s) mbar_wait_landed(raw_full0 + 8 * (s % RAWS), (uint32_t)((s / RAWS) & 1), WAIT_LIMIT);
    } else if (warp >= 8) {
        // ================= splitters: thread (row t / 8 + 32 i, piece t % 8) of W (i < 4) and of x (i >= 4)
        const int t = threadIdx.x - ADDERS, row = t >> 3, piece = t & 7;
        const uint32_t from = base + T::OFF_RAW + (uint32_t)row * 128 + (uint32_t)piece * 16;
        const uint32_t to = base + (uint32_t)row * 64 + (uint32_t)(((piece >> 1) ^ ((row >> 1) & 3)) << 4) + (piece & 1) * 8;       // (rows 32 apart swizzle alike)
        uint32_t held = 0;                                                 // two bits of each of the thread's rows: a small operand, a huge one
        for (int s = 0; s < steps; ++s) {
            const int rs = s % RAWS, st = s % PARTS;
            ok = mbar_wait(raw_full0 + 8 * rs, (uint32_t)((s / RAWS) & 1), give_up, 1);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            float4 v[T::CHUNKS];
#pragma unroll
            for (int i = 0; i < T::CHUNKS; ++i) {
                if (i >= 4 && row + 32 * (i - 4) >= NT) continue;
                asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[i].x), "=f"(v[i].y), "=f"(v[i].z), "=f"(v[i].w)
                             : "r"(from + rs * T::RAW_BYTES + i * 4096) : "memory");
            }
            if (s >= PARTS) {
                ok = mbar_wait(empty0 + 8 * st, (uint32_t)((s / PARTS - 1) & 1), give_up, 1);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
            }
#pragma unroll
            for (int i = 0; i < T::CHUNKS; ++i) {
                if (i >= 4 && row + 32 * (i - 4) >= NT) continue;
                float4 a = v[i];
                const uint32_t least = min(min(2 * __float_as_uint(a.x) - 1, 2 * __float_as_uint(a.y) - 1), min(2 * __float_as_uint(a.z) - 1, 2 * __float_as_uint(a.w) - 1));   // 0 is the largest
                const float most = fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fmaxf(fabsf(a.z), fabsf(a.w)));
                if (least < SMALL_OPERAND - 1) held |= 1u << (2 * i);
                if (most >= HUGE_OPERAND) held |= 2u << (2 * i);
                const uint32_t at = to + st * T::PART_BYTES + (i < 4 ? i * 2048 : 3 * T::W_BYTES + (i - 4) * 2048);
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    const uint32_t lo = next_parts(a.x, a.y), hi = next_parts(a.z, a.w);
                    asm volatile("st.shared.v2.b32 [%0], {%1, %2};" :: "r"(at + j * (i < 4 ? T::W_BYTES : T::X_BYTES)), "r"(lo), "r"(hi) : "memory");
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) { mbar_arrive(full0 + 8 * st); mbar_arrive(raw_read0 + 8 * rs); }
        }
#pragma unroll
        for (int d = 1; d < 8; d *= 2) held |= __shfl_xor_sync(0xffffffffu, held, d);          // the row's eight threads
        if (piece == 0) {
#pragma unroll
            for (int i = 0; i < T::CHUNKS; ++i)
                if (i < 4 || row + 32 * (i - 4) < NT) marks[row + 32 * i] = (unsigned char)(held >> (2 * i) & 3);
            if (held & 0x55555555u) *any_small = 1;
        }
    } else if (warp < 4 * T::HALVES) {
        // ================= adders: row 32 (warp & 3) + lane of the tile, COLS of its columns
        const uint32_t t_at = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (warp >> 2) * T::COLS;
        float acc[T::COLS];
#pragma unroll
        for (int j = 0; j < T::COLS; ++j) acc[j] = 0.f;
        for (int s = 0; s < steps; ++s) {
            const int b = s & 1;
            ok = mbar_wait(sum0 + 8 * b, (uint32_t)((s >> 1) & 1), give_up, 3);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            fence_after_sync();
#pragma unroll
            for (int c = 0; c < T::COLS; c += 16) {
                uint32_t r[16];
                tmem_ld16_wait(t_at + b * NT + c, r);
#pragma unroll
                for (int j = 0; j < 16; ++j) acc[c + j] += __uint_as_float(r[j]);
            }
            fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(taken0 + 8 * b);
        }
        // the last segment's MMAs have read the parts, which make room for the sums, and for those of the small products
        const int at = (warp >> 2) * T::COLS * BM + (warp & 3) * 32 + lane;
#pragma unroll
        for (int j = 0; j < T::COLS; ++j) sums[at + j * BM] = acc[j];
#pragma unroll
        for (int c = 0; c < T::COLS; c += 16) {
            uint32_t r[16] = {};
            if (ok && steps > 0) tmem_ld16_wait(t_at + 2 * NT + c, r);          // (the warps agree on ok, and the last segment's barrier has been waited for)
#pragma unroll
            for (int j = 0; j < 16; ++j) sums[BM * NT + at + (c + j) * BM] = __uint_as_float(r[j]);
        }
    }
    if (spans > 1) cluster_meet(); else __syncthreads();
    const BlGluArgs glu = bl_glu_args(GLU ? bias : nullptr);
    auto peer_byte = [&](const void* at, int r) {                          // a byte of the shared memory of block r of the cluster
        if (spans == 1) return (int)*reinterpret_cast<const unsigned char*>(at);
        uint32_t peer, v;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(smem_u32(at)), "r"(r));
        asm volatile("ld.shared::cluster.u8 %0, [%1];" : "=r"(v) : "r"(peer) : "memory");
        return (int)v;
    };
    int small_tile = 0;
    for (int r = 0; r < spans; ++r) small_tile |= peer_byte(any_small, r);
    // Whether the sum of row `col` of the tile's x and row `u` of its W is worked out again: by what these two rows hold, nothing else.
    auto again = [&](float sum, int u, int col) {
        if (!isfinite(sum)) return true;
        if (!small_tile) return false;
        int mark = 0;
        for (int r = 0; r < spans; ++r) mark |= peer_byte(marks + u, r) | peer_byte(marks + BM + col, r);
        return (mark & 1) != 0 && ((mark & 2) != 0 || fabsf(sum) < SMALL_SUM);
    };
    // the outputs of the tile, neighbours along n in neighbouring threads; a cluster's blocks take a share each
    for (int e = span * THREADS + threadIdx.x; e < NT * UNITS; e += spans * THREADS) {
        const int u = e % UNITS, col = e / UNITS;
        const int m = m0 + col, n = n0 + u;
        if (m >= M || n >= N) continue;
        const uint32_t mine = base + (uint32_t)(col * BM + u) * 4, small = BM * NT * 4;      // (the up sums of a gated tile are its rows 64 on)
        float s = 0.f, up = 0.f;
        if (spans == 1) {
            const float* at = reinterpret_cast<const float*>(smem + (mine - base));
            s = at[0] + at[BM * NT];
            if (GLU) up = at[UNITS] + at[BM * NT + UNITS];
        } else {
            float rest = 0.f, up_rest = 0.f;
            for (int r = 0; r < spans; ++r) {                              // ascending k
                uint32_t peer;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(mine), "r"(r));
                s += ld_cluster(peer);
                rest += ld_cluster(peer + small);
                if (GLU) { up += ld_cluster(peer + 4 * UNITS); up_rest += ld_cluster(peer + small + 4 * UNITS); }
            }
            s += rest;
            up += up_rest;
        }
        if (again(s, u, col)) s = plain_dot(x + (size_t)m * ldx, w + (size_t)n * K, K);
        if (GLU && again(up, UNITS + u, col)) up = plain_dot(x + (size_t)m * ldx, w + (size_t)(N + n) * K, K);
        float* dst = out + (size_t)m * N + n;
        if (EPI == BL_EPI_BIAS) s += bl_load_any(bias, bias_dtype, n);
        if (EPI == BL_EPI_RESIDUAL) {
            if (bias) s += bl_load_any(bias, bias_dtype, n);
            s += *dst;
        }
        if (GLU) {
            if (glu.bias) { s += glu.bias[n]; up += glu.bias[N + n]; }
            s = bl_glu(glu.kind, s, up, glu.limit);
        }
        *dst = s;
    }
    fence_before_sync();
    if (spans > 1) cluster_meet(); else __syncthreads();                   // no block leaves while another may still read its sums
    if (warp == 8) {
        fence_after_sync();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(T::TMEM_COLS) : "memory");
    }
}

// A row-major matrix of 32-bit numbers, rows `ld` apart, as a tensor map with boxes of box_rows rows of BK values as they lie.
int make_map(CUtensorMap* map, const float* p, long long rows, long long cols, long long ld, int box_rows) {
    BlEncodeTiled enc = bl_tensor_map_encoder();
    if (enc == nullptr) BL_FAIL("bl_gemm_f32_tc: cuTensorMapEncodeTiled is not available from the driver");
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * 4};
    cuuint32_t box[2] = {BK, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(p), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) BL_FAIL("bl_gemm_f32_tc: cuTensorMapEncodeTiled failed with code %d (rows %lld, columns %lld)", (int)r, rows, cols);
    return 0;
}

template <int EPI, int NT>
int launch(const float* x, const float* w, const void* bias, int bias_dtype, float* out, int M, int N, int K, int ldx, int spans, cudaStream_t s) {
    static std::atomic<bool> allowed{false};
    if (!allowed) {
        BL_CUDA(cudaFuncSetAttribute(gemm_f32_tc_kernel<EPI, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, Tile<NT>::SMEM_BYTES));
        allowed = true;
    }
    const int units = EPI == BL_EPI_SWIGLU ? BM / 2 : BM;
    const int m_tiles = (M + NT - 1) / NT;
    CUtensorMap mx, mw;
    if (make_map(&mx, x, M, K, ldx, NT)) return 1;
    if (make_map(&mw, w, EPI == BL_EPI_SWIGLU ? 2LL * N : N, K, K, units)) return 1;
    const dim3 grid((unsigned)((long long)((N + units - 1) / units) * m_tiles * spans));
    if (spans > 1) {
        BL_CUDA(bl_launch_dependent_clusters(gemm_f32_tc_kernel<EPI, NT>, grid, dim3(THREADS), (size_t)Tile<NT>::SMEM_BYTES, s, (unsigned)spans,
                                             mx, mw, x, w, bias, bias_dtype, out, M, N, K, ldx, spans, m_tiles));
    } else {
        BL_CUDA(bl_launch_dependent(gemm_f32_tc_kernel<EPI, NT>, grid, dim3(THREADS), (size_t)Tile<NT>::SMEM_BYTES, s,
                                    mx, mw, x, w, bias, bias_dtype, out, M, N, K, ldx, spans, m_tiles));
    }
    BL_CHECK_LAUNCH("bl_gemm_f32_tc");
    return 0;
}

template <int EPI>
int launch_width(const float* x, const float* w, const void* bias, int bias_dtype, float* out, int M, int N, int K, int ldx, int spans, cudaStream_t s) {
    // The width of a tile: the least of rounds of blocks times a segment's cycles (linear in the rows of W and x that pass through
    // shared memory).
    const int units = EPI == BL_EPI_SWIGLU ? BM / 2 : BM;
    const long long n_tiles = (N + units - 1) / units;
    const int slots = spans > 1 ? bl_device_sms() / spans - (spans > 2 ? 1 : 0) : bl_device_sms();       // tiles under way at once
    const int widths[] = {128, 96, 64, 32, 16};
    int best = 0;
    double least = 0.0;
    for (int i = 0; i < 5; ++i) {
        const int nt = widths[i];
        const long long tiles = n_tiles * ((M + nt - 1) / nt);
        const double cost = (double)((tiles + slots - 1) / slots) * (640 + 5 * nt);
        if (i == 0 || cost < least) { least = cost; best = nt; }
    }
    switch (best) {
        case 128: return launch<EPI, 128>(x, w, bias, bias_dtype, out, M, N, K, ldx, spans, s);
        case 96: return launch<EPI, 96>(x, w, bias, bias_dtype, out, M, N, K, ldx, spans, s);
        case 64: return launch<EPI, 64>(x, w, bias, bias_dtype, out, M, N, K, ldx, spans, s);
        case 32: return launch<EPI, 32>(x, w, bias, bias_dtype, out, M, N, K, ldx, spans, s);
        default: return launch<EPI, 16>(x, w, bias, bias_dtype, out, M, N, K, ldx, spans, s);
    }
}

// Into how many spans K is cut, over the blocks of a cluster: four where the clusters of a row of tiles fit the device at once (up to 33
// tiles), two up to 72, if the spans keep four segments each. By N and K alone: which spans a sum is made of must not depend on the rows.
// Few rows, whose launch is one row of tiles, gain more than many lose in blocks of their own beginning and end. Uncut -> cut, microseconds,
// 1, 128 and 2,048 rows: 4,224 x 2,048 (33 tiles) 58 -> 18, 55 -> 29, 318 -> 425; 4,608 x 3,584 (36) 86 -> 45, 88 -> 53, 460 -> 495 (FMAs 42,
// 150, 1,150); 6,144 x 2,048 (48) 55 -> 31, 62 -> 43, 407 -> 443; gated 4,608 + 4,608 x 1,536 (72) 43 -> 23, 48 -> 34, 425 -> 511.
int f32_tc_spans(int N, int K, int epi) {
    const int units = epi == BL_EPI_SWIGLU ? BM / 2 : BM, n_tiles = (N + units - 1) / units;
    return n_tiles <= 33 && K >= 4 * 4 * BK ? 4 : n_tiles <= 72 && K >= 2 * 4 * BK ? 2 : 1;
}

}  // namespace

// Whether the tensor cores take a product of these sizes (rows of whole 16-byte pieces): by N and K alone, see above. Products of
// more columns are output heads: mostly a row or a few of them, which FMAs stream faster than W can be split (151,936 x 896: one
// row 104 us against 208, 16 rows 150 and 210, 33 rows 448 and 265).
extern "C" int bl_gemm_f32_tc_supported(int N, int K, int ldx) {
    return N >= 128 && N <= MAX_COLUMNS && K >= 256 && K % 4 == 0 && ldx % 4 == 0;
}

extern "C" int bl_gemm_f32_tc(const float* x, int ldx, const float* w, const void* bias, int bias_dtype, float* out, int M, int N, int K,
                              int epilogue, void* stream) {
    if (M <= 0) return 0;
    if (N <= 0 || K <= 0 || ldx < K || !bl_gemm_f32_tc_supported(N, K, ldx) || (((uintptr_t)x | (uintptr_t)w) & 15))
        BL_FAIL("bl_gemm_f32_tc: N=%d K=%d ldx=%d is not what this kernel takes", N, K, ldx);
    if (epilogue == BL_EPI_BIAS && bias == nullptr) BL_FAIL("bl_gemm_f32_tc: bias epilogue without a bias");
    if (epilogue == BL_EPI_BIAS && bias_dtype != BL_F32 && bias_dtype != BL_BF16) BL_FAIL("bl_gemm_f32_tc: unknown bias dtype %d", bias_dtype);
    const int spans = f32_tc_spans(N, K, epilogue);
    if ((long long)((N + 63) / 64) * ((M + 15) / 16) * spans > 0x7fffffffLL) BL_FAIL("bl_gemm_f32_tc: too many blocks");
    cudaStream_t s = (cudaStream_t)stream;
    switch (epilogue) {
        case BL_EPI_NONE: return launch_width<BL_EPI_NONE>(x, w, bias, bias_dtype, out, M, N, K, ldx, spans, s);
        case BL_EPI_BIAS: return launch_width<BL_EPI_BIAS>(x, w, bias, bias_dtype, out, M, N, K, ldx, spans, s);
        case BL_EPI_RESIDUAL: return launch_width<BL_EPI_RESIDUAL>(x, w, bias, bias_dtype, out, M, N, K, ldx, spans, s);
        case BL_EPI_SWIGLU: return launch_width<BL_EPI_SWIGLU>(x, w, bias, bias_dtype, out, M, N, K, ldx, spans, s);
        default: BL_FAIL("bl_gemm_f32_tc: unknown epilogue %d", epilogue);
    }
}

// Reads and clears the status word: 0 when no block has given up on a wait (1 a splitter, 2 the issuing warp, 3 an adder). Synchronises.
extern "C" int bl_gemm_f32_tc_status(int* status) {
    int v = 0, zero = 0;
    BL_CUDA(cudaMemcpyFromSymbol(&v, g_status, sizeof(int)));
    if (v != 0) BL_CUDA(cudaMemcpyToSymbol(g_status, &zero, sizeof(int)));
    *status = v;
    return 0;
}
