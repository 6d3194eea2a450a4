// Plain paged causal grouped-query attention: one warp per (token, head), keys in ascending position,
// softmax in its online form with 32-bit statistics. Formulas: gqa_attention_ext (src/math.br:304-359):
// kv head = head / (H / KV), score = dot * scale (scale after the dot), causal with the reference's
// `causal_offset` (src/math_gpu.br:3044-3047), window: key j is seen while j + window > position
// (src/math.br:327-328); online form as FlashAttnKernel (src/math_gpu.br:3224-3287).
// A (token, head) is computed the same way whatever else is in the batch: its chunks of 32 keys start
// at its first visible key. This is the 32-bit path's attention and the twin of the fast kernels.
// Options (bl_attention_plain_ext): values of another head size than the keys; a sink per head, a learned score that
// joins the softmax's denominator once, unscaled, without a value; a gate per (token, head) whose sigmoid multiplies
// the head's output, or one per (token, head, channel); a cap c on the scores, s <- c tanh(s / c), applied to the scaled score before the softmax.
#include "common.cuh"
#include <atomic>
#include "api.h"

namespace {

constexpr int MAX_DH = 256;
constexpr int WARPS = 4;

// VEC: 32-bit keys whose rows are whole 16-byte pieces are read a piece at a time (the dot product stays one chain in
// ascending d). NV: 32-column groups of the values, so that a lane does not walk groups the head does not have.
template <typename TT, bool VEC, int NV>
__global__ void __launch_bounds__(WARPS * 32)
attention_plain_kernel(const TT* __restrict__ q, const TT* __restrict__ kc, const TT* __restrict__ vc,
                       const int* __restrict__ tok_req, const int* __restrict__ cu_q,
                       const int* __restrict__ ctx_len, const int* __restrict__ block_table, int max_pages,
                       TT* __restrict__ out, int T, int H, int KV, int dh, int dv, int page_size, int window,
                       float scale, const void* __restrict__ sinks, int sink_dtype, const float* gate, int ld_gate, int gate_dim, float softcap) {
    __shared__ __align__(16) float qs[WARPS][MAX_DH];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int item = blockIdx.x * WARPS + warp;
    if (item >= T * H) return;                 // whole warps leave together; no block-wide barrier below
    const int t = item / H, h = item % H;
    const int r = tok_req[t];
    const int q_len = cu_q[r + 1] - cu_q[r];
    const int pos = ctx_len[r] - q_len + (t - cu_q[r]);
    const int kvh = h / (H / KV);
    const int lo = window > 0 ? max(0, pos - window + 1) : 0;
    const TT* qrow = q + ((size_t)t * H + h) * dh;
    for (int d = lane; d < dh; d += 32) qs[warp][d] = bl_load(qrow + d);
    __syncwarp();
    const int* bt = block_table + (size_t)r * max_pages;
    const size_t head_off = (size_t)kvh * page_size * dh, v_head_off = (size_t)kvh * page_size * dv;
    const size_t page_stride = (size_t)KV * page_size * dh, v_page_stride = (size_t)KV * page_size * dv;
    float m = -INFINITY, l = 0.f;
    float acc[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) acc[i] = 0.f;
    for (int base = lo; base <= pos; base += 32) {
        const int j = base + lane;
        const bool valid = j <= pos;
        float s = -INFINITY;
        unsigned long long vrow = 0;                   // where the values of this lane's key lie
        if (valid) {
            const int page = bt[j / page_size], at = j % page_size;
            vrow = (size_t)page * v_page_stride + v_head_off + (size_t)at * dv;
            const TT* krow = kc + (size_t)page * page_stride + head_off + (size_t)at * dh;
            float dot = 0.f;
            if constexpr (VEC) {
#pragma unroll 8
                for (int d = 0; d < dh; d += 4) {
                    const float4 a = *reinterpret_cast<const float4*>(&qs[warp][d]), b = *reinterpret_cast<const float4*>(krow + d);
                    dot = fmaf(a.x, b.x, dot); dot = fmaf(a.y, b.y, dot); dot = fmaf(a.z, b.z, dot); dot = fmaf(a.w, b.w, dot);
                }
            } else {
                for (int d = 0; d < dh; ++d) dot = fmaf(qs[warp][d], bl_load(krow + d), dot);
            }
            s = dot * scale;
            if (softcap > 0.f) s = softcap * tanhf(s / softcap);
        }
        const float m_new = fmaxf(m, bl_warp_max(s));
        const float p = valid ? expf(s - m_new) : 0.f;
        const float alpha = expf(m - m_new);           // first chunk: exp(-inf) = 0
        l = l * alpha + bl_warp_sum(p);
#pragma unroll
        for (int i = 0; i < NV; ++i) acc[i] *= alpha;
        const int n = min(32, pos - base + 1);
        for (int j0 = 0; j0 < n; j0 += 8) {            // eight keys' values in flight, added in ascending position
            float v[8][NV];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const unsigned long long row = __shfl_sync(0xffffffffu, vrow, j0 + u);
#pragma unroll
                for (int i = 0; i < NV; ++i)
                    if (j0 + u < n && lane + 32 * i < dv) v[u][i] = bl_load(vc + row + lane + 32 * i);
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const float pj = __shfl_sync(0xffffffffu, p, j0 + u);
#pragma unroll
                for (int i = 0; i < NV; ++i)
                    if (j0 + u < n && lane + 32 * i < dv) acc[i] = fmaf(pj, v[u][i], acc[i]);
            }
        }
        m = m_new;
    }
    if (sinks) {                                       // one more term of the denominator, after the last key
        const float sk = bl_load_any(sinks, sink_dtype, h);
        const float m_new = fmaxf(m, sk);
        const float alpha = expf(m - m_new);
        l = l * alpha + expf(sk - m_new);
#pragma unroll
        for (int i = 0; i < NV; ++i) acc[i] *= alpha;
    }
    TT* orow = out + ((size_t)t * H + h) * dv;
    float inv = l > 0.f ? 1.0f / l : 0.f;
    if (gate && gate_dim == 0) inv *= bl_sigmoid(gate[(size_t)t * ld_gate + h]);
    const float* crow = gate && gate_dim ? gate + (size_t)t * ld_gate + (size_t)h * gate_dim : nullptr;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int d = lane + 32 * i;
        if (d < dv) bl_store(orow + d, crow ? acc[i] * inv * bl_sigmoid(crow[d]) : acc[i] * inv);
    }
}

// The same for many 32-bit rows: a warp takes up to HPW heads of a token that share a key/value head, and the same sums in the same
// order. The kernel above reads a key's row by the lane that owns the key, 32 lines a load, which is what it waits for; here a
// chunk's keys and values pass through the warp's shared memory in whole lines (cp.async: the values arrive under the scores, the next
// keys under the products with the values) and serve all its heads.
template <int HPW, int NV>
__global__ void __launch_bounds__(WARPS * 32)
attention_plain_heads_kernel(const float* __restrict__ q, const float* __restrict__ kc, const float* __restrict__ vc,
                             const int* __restrict__ tok_req, const int* __restrict__ cu_q, const int* __restrict__ ctx_len,
                             const int* __restrict__ block_table, int max_pages, float* __restrict__ out, int T, int H, int KV, int dh, int dv,
                             int page_size, int window, float scale, const void* __restrict__ sinks, int sink_dtype, const float* gate,
                             int ld_gate, int gate_dim, float softcap) {
    extern __shared__ __align__(16) float sm[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ldk = dh + 4;                            // padded: eight rows' pieces of 16 bytes fall on different banks
    float* qs = sm + (size_t)warp * (HPW * dh + 32 * (ldk + dv + HPW));     // [HPW][dh]
    float* ks = qs + HPW * dh;                         // [32][ldk]
    float* vs = ks + 32 * ldk;                         // [32][dv]
    float* ps = vs + 32 * dv;                          // [32][HPW]
    const int G = H / KV, per = (G + HPW - 1) / HPW;
    const int item = blockIdx.x * WARPS + warp;
    bl_pdl_trigger();
    bl_pdl_wait();
    if (item >= T * KV * per) return;                  // whole warps leave together; no block-wide barrier below
    const int t = item / (KV * per), kvh = item / per % KV, h0 = kvh * G + item % per * HPW;
    const int nh = min(HPW, (kvh + 1) * G - h0);
    const int r = tok_req[t];
    const int q_len = cu_q[r + 1] - cu_q[r];
    const int pos = ctx_len[r] - q_len + (t - cu_q[r]);
    const int lo = window > 0 ? max(0, pos - window + 1) : 0;
    for (int d = lane; d < HPW * dh; d += 32) qs[d] = d < nh * dh ? q[((size_t)t * H + h0) * dh + d] : 0.f;
    const int* bt = block_table + (size_t)r * max_pages;
    // Rows [base, base + 32) of a cache, those past `pos` left out, 2^n4 pieces of 16 bytes a row: a lane knows where one row lies.
    auto copy = [&](float* dst, int ld, const float* cache, int n4, int base) {
        const int j = min(base + lane, pos), width = 4 << n4;
        const long long mine = ((long long)bt[j / page_size] * KV + kvh) * page_size + j % page_size;
        const int rows = min(32, pos - base + 1), col = lane & ((1 << n4) - 1);
#pragma unroll 4
        for (int row0 = 0; row0 < rows; row0 += 32 >> n4) {
            const int row = row0 + (lane >> n4);
            const long long at = __shfl_sync(0xffffffffu, mine, row & 31);
            if (row < rows)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n"
                             :: "r"((unsigned)__cvta_generic_to_shared(dst + row * ld + col * 4)), "l"(cache + at * width + col * 4));
        }
        asm volatile("cp.async.commit_group;\n" ::);
    };
    const int k_log = 31 - __clz(dh >> 2), v_log = 31 - __clz(dv >> 2);
    float m[HPW], l[HPW], acc[HPW][NV];
#pragma unroll
    for (int h = 0; h < HPW; ++h) {
        m[h] = -INFINITY; l[h] = 0.f;
#pragma unroll
        for (int i = 0; i < NV; ++i) acc[h][i] = 0.f;
    }
    copy(ks, ldk, kc, k_log, lo);
    for (int base = lo; base <= pos; base += 32) {
        copy(vs, dv, vc, v_log, base);
        asm volatile("cp.async.wait_group 1;\n" ::);   // the keys
        __syncwarp();
        const bool valid = base + lane <= pos;
        float s[HPW];
#pragma unroll
        for (int h = 0; h < HPW; ++h) s[h] = 0.f;
#pragma unroll 4
        for (int d = 0; d < dh; d += 4) {
            const float4 b = *reinterpret_cast<const float4*>(ks + lane * ldk + d);
#pragma unroll
            for (int h = 0; h < HPW; ++h) {
                const float4 a = *reinterpret_cast<const float4*>(qs + h * dh + d);
                s[h] = fmaf(a.x, b.x, s[h]); s[h] = fmaf(a.y, b.y, s[h]); s[h] = fmaf(a.z, b.z, s[h]); s[h] = fmaf(a.w, b.w, s[h]);
            }
        }
        __syncwarp();                                  // the keys have been read
        if (base + 32 <= pos) copy(ks, ldk, kc, k_log, base + 32);
        else asm volatile("cp.async.commit_group;\n" ::);
#pragma unroll
        for (int h = 0; h < HPW; ++h) {
            float sc = s[h] * scale;
            if (softcap > 0.f) sc = softcap * tanhf(sc / softcap);
            if (!valid) sc = -INFINITY;                // (whatever the lane's row of the buffer holds)
            const float m_new = fmaxf(m[h], bl_warp_max(sc));
            const float p = valid ? expf(sc - m_new) : 0.f;
            const float alpha = expf(m[h] - m_new);    // first chunk: exp(-inf) = 0
            l[h] = l[h] * alpha + bl_warp_sum(p);
#pragma unroll
            for (int i = 0; i < NV; ++i) acc[h][i] *= alpha;
            ps[lane * HPW + h] = p;
            m[h] = m_new;
        }
        asm volatile("cp.async.wait_group 1;\n" ::);   // the values
        __syncwarp();
        const int n = min(32, pos - base + 1);
#pragma unroll 4
        for (int j = 0; j < n; ++j) {                  // ascending position
            float v[NV], p[HPW];
#pragma unroll
            for (int i = 0; i < NV; ++i) v[i] = lane + 32 * i < dv ? vs[j * dv + lane + 32 * i] : 0.f;
#pragma unroll
            for (int h = 0; h < HPW; ++h) p[h] = ps[j * HPW + h];
#pragma unroll
            for (int h = 0; h < HPW; ++h)
#pragma unroll
                for (int i = 0; i < NV; ++i) acc[h][i] = fmaf(p[h], v[i], acc[h][i]);
        }
        __syncwarp();                                  // values and weights have been read
    }
#pragma unroll
    for (int h = 0; h < HPW; ++h) {
        if (h >= nh) continue;
        const int head = h0 + h;
        if (sinks) {                                   // one more term of the denominator, after the last key
            const float sk = bl_load_any(sinks, sink_dtype, head);
            const float m_new = fmaxf(m[h], sk);
            const float alpha = expf(m[h] - m_new);
            l[h] = l[h] * alpha + expf(sk - m_new);
#pragma unroll
            for (int i = 0; i < NV; ++i) acc[h][i] *= alpha;
        }
        float inv = l[h] > 0.f ? 1.0f / l[h] : 0.f;
        if (gate && gate_dim == 0) inv *= bl_sigmoid(gate[(size_t)t * ld_gate + head]);
        const float* crow = gate && gate_dim ? gate + (size_t)t * ld_gate + (size_t)head * gate_dim : nullptr;
        float* orow = out + ((size_t)t * H + head) * dv;
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const int d = lane + 32 * i;
            if (d < dv) orow[d] = crow ? acc[h][i] * inv * bl_sigmoid(crow[d]) : acc[h][i] * inv;
        }
    }
}

// Rows times heads from which warps with several heads each fill the device, heads a warp takes.
constexpr int HEADS_MIN_ITEMS = 2048, HEADS_A_WARP = 4, HEADS_MAX_DH = 128;

}  // namespace

extern "C" int bl_attention_plain(const void* q, const void* k_cache, const void* v_cache, int dtype,
                                  const int* tok_req, const int* cu_q, const int* ctx_len,
                                  const int* block_table, int max_pages, void* out, int T, int H, int KV,
                                  int dh, int page_size, int window, float scale, void* stream) {
    return bl_attention_plain_ext(q, k_cache, v_cache, dtype, tok_req, cu_q, ctx_len, block_table, max_pages, out, T, H, KV,
                                  dh, dh, page_size, window, scale, nullptr, 0, nullptr, 0, stream);
}

extern "C" int bl_attention_plain_ext(const void* q, const void* k_cache, const void* v_cache, int dtype,
                                      const int* tok_req, const int* cu_q, const int* ctx_len,
                                      const int* block_table, int max_pages, void* out, int T, int H, int KV,
                                      int dh, int dv, int page_size, int window, float scale, const void* sinks,
                                      int sink_dtype, const float* gate, int ld_gate, void* stream) {
    return bl_attention_plain_cap(q, k_cache, v_cache, dtype, tok_req, cu_q, ctx_len, block_table, max_pages, out, T, H, KV,
                                  dh, dv, page_size, window, scale, sinks, sink_dtype, gate, ld_gate, 0, 0.f, stream);
}

extern "C" int bl_attention_plain_cap(const void* q, const void* k_cache, const void* v_cache, int dtype,
                                      const int* tok_req, const int* cu_q, const int* ctx_len,
                                      const int* block_table, int max_pages, void* out, int T, int H, int KV,
                                      int dh, int dv, int page_size, int window, float scale, const void* sinks,
                                      int sink_dtype, const float* gate, int ld_gate, int gate_dim, float softcap, void* stream) {
    if (T <= 0) return 0;
    if (!(softcap >= 0.f)) BL_FAIL("bl_attention_plain: a cap on the scores must not be negative, got %g", (double)softcap);
    if (dv <= 0 || dv > MAX_DH) BL_FAIL("bl_attention_plain: value head size %d is outside 1..%d", dv, MAX_DH);
    if (gate_dim && (!gate || gate_dim != dv || ld_gate < H * dv)) BL_FAIL("bl_attention_plain: a gate of %d channels a head in rows of %d for %d heads of %d", gate_dim, ld_gate, H, dv);
    if (gate && ld_gate < H) BL_FAIL("bl_attention_plain: gate rows of %d hold fewer than %d heads", ld_gate, H);
    if (H <= 0 || KV <= 0 || H % KV != 0) BL_FAIL("bl_attention_plain: %d heads cannot share %d key/value heads", H, KV);
    if (dh <= 0 || dh > MAX_DH) BL_FAIL("bl_attention_plain: head size %d is outside 1..%d", dh, MAX_DH);
    if (page_size <= 0 || max_pages <= 0 || window < 0) BL_FAIL("bl_attention_plain: bad page size, table width or window");
    cudaStream_t s = (cudaStream_t)stream;
    const int blocks = (T * H + WARPS - 1) / WARPS;
    const bool vec = dtype == BL_F32 && dh % 4 == 0 && ((uintptr_t)k_cache & 15) == 0;
    // Several heads a warp: rows and values of 4, 8, .. 128 values, heads that share keys, and enough of them.
    const auto power = [](int n) { return n >= 4 && n <= HEADS_MAX_DH && (n & (n - 1)) == 0; };
    if (vec && H > KV && power(dh) && power(dv) && ((uintptr_t)v_cache & 15) == 0 && (long long)T * H >= HEADS_MIN_ITEMS) {
        const int per = (H / KV + HEADS_A_WARP - 1) / HEADS_A_WARP;
        const int grid = (T * KV * per + WARPS - 1) / WARPS;
        const size_t smem = (size_t)WARPS * (HEADS_A_WARP * dh + 32 * (dh + 4 + dv + HEADS_A_WARP)) * sizeof(float);
#define BL_HEADS(NV) do { \
            static std::atomic<bool> allowed{false}; \
            if (!allowed) { BL_CUDA(cudaFuncSetAttribute(attention_plain_heads_kernel<HEADS_A_WARP, NV>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                (int)(WARPS * (HEADS_A_WARP * HEADS_MAX_DH + 32 * (2 * HEADS_MAX_DH + 4 + HEADS_A_WARP)) * sizeof(float)))); allowed = true; } \
            BL_CUDA(bl_launch_dependent(attention_plain_heads_kernel<HEADS_A_WARP, NV>, dim3(grid), dim3(WARPS * 32), smem, s, (const float*)q, (const float*)k_cache, \
                (const float*)v_cache, tok_req, cu_q, ctx_len, block_table, max_pages, (float*)out, T, H, KV, dh, dv, page_size, window, scale, sinks, \
                sink_dtype, gate, ld_gate, gate_dim, softcap)); } while (0)
        if (dv <= 64) BL_HEADS(2); else BL_HEADS(4);
#undef BL_HEADS
        BL_CHECK_LAUNCH("bl_attention_plain");
        return 0;
    }
#define BL_GO(TT, VEC, NV) attention_plain_kernel<TT, VEC, NV><<<blocks, WARPS * 32, 0, s>>>((const TT*)q, (const TT*)k_cache, \
            (const TT*)v_cache, tok_req, cu_q, ctx_len, block_table, max_pages, (TT*)out, T, H, KV, dh, dv, \
            page_size, window, scale, sinks, sink_dtype, gate, ld_gate, gate_dim, softcap)
#define BL_GO_NV(TT, VEC) do { if (dv <= 64) BL_GO(TT, VEC, 2); else if (dv <= 128) BL_GO(TT, VEC, 4); else BL_GO(TT, VEC, 8); } while (0)
    if (dtype == BL_F32 && vec) BL_GO_NV(float, true);
    else if (dtype == BL_F32) BL_GO_NV(float, false);
    else if (dtype == BL_BF16) BL_GO_NV(__nv_bfloat16, false);
    else
        BL_FAIL("bl_attention_plain: unknown dtype %d", dtype);
#undef BL_GO_NV
#undef BL_GO
    BL_CHECK_LAUNCH("bl_attention_plain");
    return 0;
}
