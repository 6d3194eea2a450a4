// Linear recurrences with a matrix state per head, S [key channels, value channels], carried per request in a state
// slot, for prompts' portions and single decoded tokens alike (a request's tokens are cu_q[r] .. cu_q[r + 1] - 1 of
// the batch; a request without tokens is left alone). Three rules share one kernel:
//   gated linear attention   S <- diag(a) S + k v^T;                                   o = S^T q
//   gated delta rule         S <- diag(a) S;  u = beta (v - S^T k);  S <- S + k u^T;   o = S^T q
//   read-out before the write, with a bonus for the current token
//                            o = S^T q + b v;  S <- diag(a) S + k v^T                  (b per token and head, given)
// with a decay per key channel a, given per token, head and channel (the product that makes its pre-activation z turns it
// into exp(-coef[head] * softplus(sign * z)); sign -1, coef 1 / tau gives sigmoid(z)^(1 / tau)). State, decays, gates and
// all sums are 32-bit. The columns of S are
// independent of one another, so a block owns a few columns of one (request, head) and walks the request's tokens in
// order; a column's rows are spread over KS lanes of a warp that add up with a fixed butterfly. What a token's result is
// does not depend on the batch or on how the tokens were cut into steps.
// Also here: the short causal convolution + SiLU + unit norm in front of the delta rule, the hand-over of the
// convolution's last inputs to the state slot, and the per-head RMS norm with an output gate behind both rules.
#include "common.cuh"
#include "api.h"

namespace {

constexpr int WARPS = 4;
constexpr int RKMAX = 16;          // rows of a column that one lane holds
constexpr int MAX_TAPS = 16;
constexpr int SCAN_SMEM_BYTES = 40 * 1024;
constexpr int SCAN_VEC_ROWS = 16;    // rows a lane holds in the kernel with 16-byte fetches, where the key size allows
constexpr int SCAN_SPLIT_MIN = 256;  // tokens of a request in one step from which its portion is cut into parts that run side by side

__device__ __forceinline__ float sigmoidf_(float x) { return 1.0f / (1.0f + expf(-x)); }

__device__ __forceinline__ void store4(float* p, float a, float b, float c, float d) { *reinterpret_cast<float4*>(p) = make_float4(a, b, c, d); }
__device__ __forceinline__ void store4(__nv_bfloat16* p, float a, float b, float c, float d) {
    const __nv_bfloat162 lo = __floats2bfloat162_rn(a, b), hi = __floats2bfloat162_rn(c, d);
    uint2 pk;
    pk.x = *reinterpret_cast<const unsigned*>(&lo); pk.y = *reinterpret_cast<const unsigned*>(&hi);
    *reinterpret_cast<uint2*>(p) = pk;
}

__device__ __forceinline__ void cp_async4(float* smem, const float* gmem) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" :: "r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem));
}
__device__ __forceinline__ void cp_async16(float* smem, const float* gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" :: "r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
// Two 32-bit numbers in one register pair, for the instructions that work on both at once.
__device__ __forceinline__ uint64_t f2_pack(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void f2_unpack(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t f2_mul(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" :: "n"(N)); }

// The tokens of a request pass through shared memory in chunks of `chunk` tokens, two buffers taking turns: while the
// warps walk one chunk, the next one's q, k, z, v and beta are on their way (cp.async); when it has arrived the block
// squashes beta in place, once for all its columns.
template <int RULE>
__global__ void __launch_bounds__(WARPS * 32)
recurrent_scan_kernel(const float* q, int ldq, const float* k, int ldk, const float* v, int ldv, const float* z, int ldz,
                      const float* beta, int ldb, float q_scale,
                      float* state, size_t slot_stride, const int* __restrict__ slots, const int* __restrict__ cu_q,
                      float* out, int H, int G, int dk, int dv, int KS, int chunk, int vec) {
    bl_pdl_trigger();
    bl_pdl_wait();
    extern __shared__ __align__(16) float sm[];
    constexpr bool DELTA = RULE == BL_RULE_DELTA, BONUS = RULE == BL_RULE_BONUS;
    const int r = blockIdx.z, h = blockIdx.y;
    const int t0 = cu_q[r], n = cu_q[r + 1] - t0;
    if (n <= 0) return;
    const int gh = h / (H / G);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int CW = 32 / KS, cols_blk = WARPS * CW;
    const int s = lane / CW, cc = lane % CW;
    const int c = (blockIdx.x * WARPS + warp) * CW + cc;
    const bool col_ok = c < dv;
    const int per_tok = 3 * dk + cols_blk + 4;              // q | k | decay | v | beta (+ padding to 16 bytes)
    const int buf_floats = chunk * per_tok;
    float* S = state + (size_t)slots[r] * slot_stride + (size_t)h * dk * dv;
    const int col0 = blockIdx.x * cols_blk;

    auto issue = [&](int base, float* buf) {
        const int m = min(chunk, n - base);
        for (int tt = warp; tt < m; tt += WARPS) {
            const size_t tok = (size_t)(t0 + base + tt);
            float* dst = buf + (size_t)tt * per_tok;
            const float* gq = q + tok * ldq + gh * dk;
            const float* gk = k + tok * ldk + gh * dk;
            const float* gz = z + tok * ldz + h * dk;
            if (vec) {
                for (int d = lane * 4; d < dk; d += 128) {
                    cp_async16(dst + d, gq + d); cp_async16(dst + dk + d, gk + d); cp_async16(dst + 2 * dk + d, gz + d);
                }
            } else {
                for (int d = lane; d < dk; d += 32) {
                    cp_async4(dst + d, gq + d); cp_async4(dst + dk + d, gk + d); cp_async4(dst + 2 * dk + d, gz + d);
                }
            }
            const float* gv = v + tok * ldv + h * dv + col0;
            for (int j = lane; j < cols_blk; j += 32) {
                if (col0 + j < dv) cp_async4(dst + 3 * dk + j, gv + j);
                else dst[3 * dk + j] = 0.f;
            }
            if ((DELTA || BONUS) && lane == 0) cp_async4(dst + 3 * dk + cols_blk, beta + tok * ldb + h);
        }
        cp_async_commit();
    };

    issue(0, sm);
    float st[RKMAX];
#pragma unroll
    for (int i = 0; i < RKMAX; ++i) {
        const int row = i * KS + s;
        st[i] = (row < dk && col_ok) ? S[(size_t)row * dv + c] : 0.f;
    }
    int which = 0;
    for (int base = 0; base < n; base += chunk, which ^= 1) {
        const int m = min(chunk, n - base);
        float* buf = sm + (size_t)which * buf_floats;
        if (base + chunk < n) { issue(base + chunk, sm + (size_t)(which ^ 1) * buf_floats); cp_async_wait<1>(); }
        else cp_async_wait<0>();
        __syncthreads();
        if (DELTA) {
            for (int tt = threadIdx.x; tt < m; tt += WARPS * 32) {
                float* b = buf + (size_t)tt * per_tok + 3 * dk + cols_blk;
                *b = sigmoidf_(*b);
            }
            __syncthreads();
        }
        // A token's q, k and decays are fetched into registers while the token before is worked on: the fetches do not
        // depend on the state, the arithmetic does, and a warp has no other warp to hide its latencies behind.
        float cq[RKMAX], ck[RKMAX], cd[RKMAX], nq[RKMAX], nk[RKMAX], nd[RKMAX];
        float cv, cb = 0.f, nv = 0.f, nb = 0.f;
        auto fetch = [&](int tt, float (&fq)[RKMAX], float (&fk)[RKMAX], float (&fd)[RKMAX], float& fv, float& fb) {
            const float* pq = buf + (size_t)tt * per_tok;
#pragma unroll
            for (int i = 0; i < RKMAX; ++i) {
                const int row = i * KS + s;
                const int rr = min(row, dk - 1);
                const bool ok = row < dk;
                fq[i] = ok ? pq[rr] : 0.f;
                fk[i] = ok ? pq[dk + rr] : 0.f;
                fd[i] = pq[2 * dk + rr];
            }
            fv = pq[3 * dk + warp * CW + cc];
            if (DELTA || BONUS) fb = pq[3 * dk + cols_blk];
        };
        fetch(0, cq, ck, cd, cv, cb);
        for (int tt = 0; tt < m; ++tt) {
            if (tt + 1 < m) fetch(tt + 1, nq, nk, nd, nv, nb);
            float o;
            if (!DELTA) {
                float o0 = 0.f, o1 = 0.f;
#pragma unroll
                for (int i = 0; i < RKMAX; i += 2) {
                    if (BONUS) { o0 = fmaf(st[i], cq[i], o0); o1 = fmaf(st[i + 1], cq[i + 1], o1); }   // the state before the write
                    st[i] = fmaf(cd[i], st[i], ck[i] * cv);
                    st[i + 1] = fmaf(cd[i + 1], st[i + 1], ck[i + 1] * cv);
                    if (!BONUS) { o0 = fmaf(st[i], cq[i], o0); o1 = fmaf(st[i + 1], cq[i + 1], o1); }
                }
                o = o0 + o1;
                for (int x = 16; x >= CW; x >>= 1) o += __shfl_xor_sync(0xffffffffu, o, x);
                if (BONUS) o = fmaf(cb, cv, o);
            } else {
                float sk0 = 0.f, sk1 = 0.f, sq0 = 0.f, sq1 = 0.f, kq0 = 0.f, kq1 = 0.f;
#pragma unroll
                for (int i = 0; i < RKMAX; i += 2) {
                    st[i] *= cd[i];
                    st[i + 1] *= cd[i + 1];
                    sk0 = fmaf(st[i], ck[i], sk0); sk1 = fmaf(st[i + 1], ck[i + 1], sk1);
                    sq0 = fmaf(st[i], cq[i], sq0); sq1 = fmaf(st[i + 1], cq[i + 1], sq1);
                    kq0 = fmaf(ck[i], cq[i], kq0); kq1 = fmaf(ck[i + 1], cq[i + 1], kq1);
                }
                float sk_ = sk0 + sk1, sq_ = sq0 + sq1, kq = kq0 + kq1;
                for (int x = 16; x >= CW; x >>= 1) {
                    sk_ += __shfl_xor_sync(0xffffffffu, sk_, x);
                    sq_ += __shfl_xor_sync(0xffffffffu, sq_, x);
                    kq += __shfl_xor_sync(0xffffffffu, kq, x);
                }
                const float u = cb * (cv - sk_);
#pragma unroll
                for (int i = 0; i < RKMAX; ++i) st[i] = fmaf(ck[i], u, st[i]);
                o = fmaf(kq, u, sq_);                  // S^T q after the write: (a S)^T q + (k . q) u
            }
            if (s == 0 && col_ok) out[(size_t)(t0 + base + tt) * H * dv + h * dv + c] = o * q_scale;
#pragma unroll
            for (int i = 0; i < RKMAX; ++i) { cq[i] = nq[i]; ck[i] = nk[i]; cd[i] = nd[i]; }
            cv = nv; cb = nb;
        }
        __syncthreads();                               // the buffer is free for the chunk after next
    }
#pragma unroll
    for (int i = 0; i < RKMAX; ++i) {
        const int row = i * KS + s;
        if (row < dk && col_ok) S[(size_t)row * dv + c] = st[i];
    }
}

// Of the requests whose portions are long enough to be cut, how many stand before r: its place in the scratch, which holds the
// cut requests only (not the running ones beside them). All threads of the block come here.
__device__ __forceinline__ int scan_cut_place(const int* __restrict__ cu_q, int r) {
    int n = 0;
    for (int i0 = 0; i0 < r; i0 += blockDim.x) {
        const int i = i0 + threadIdx.x;
        n += __syncthreads_count(i < r && cu_q[i + 1] - cu_q[i] >= SCAN_SPLIT_MIN);
    }
    return n;
}

// The same walk for key sizes that split evenly: a lane holds RK4 * 4 CONSECUTIVE rows of its column (dk = KS * RK4 * 4),
// so a token's q, k and decays reach its registers as 16-byte loads at fixed offsets, two tokens' registers take turns
// (no copies), and the dot products run in two chains. Where a launch has few blocks a warp has no other warp on its
// scheduler to hide latencies behind (a request gives H * dv / (WARPS * CW) blocks): what counts is the number of
// instructions per token. DENSE: for launches of more blocks than two an SM: one token's registers instead of two, so that
// four blocks fit an SM and hide each other's latencies. The order of every sum is the same in both.
// CUT: portions may be cut. A launch of few blocks that cuts nothing (decode steps of a few requests) goes without the code for it:
// its set-up counts there (8 requests, 7 heads of 64 x 128: 3.9 -> 3.5 us, delta rule 4.2 -> 3.5).
// NC: columns a lane holds, 1 or 4 neighbours. A token's q, k and decays come from shared memory once for all of them: with one column
// a warp's 12 loads of 16 bytes feed 48 multiplications a lane, and where many warps walk side by side the SM's shared-memory port is
// what they wait for (48 cycles a token and warp); with four a warp takes longer over a token, which a launch of few warps would feel.
// QUIET: the first pass over a portion that was cut: no read-out. With four blocks an SM, up to 32 parts instead of 16 and
// the folds' loads in flight, a Fezopel prefill of 2,048 tokens (0.5B sizes, six recurrent layers) 2,629 -> 2,090 us.
// KSC: the number of lanes that share a column where the build is for one (0: any, an argument).
// Two neighbouring rows go through the instructions that work on a pair of 32-bit numbers (each rounded as the scalar instruction
// rounds it): a token's time is its instructions and their latencies.
template <int RULE, int RK4, int NC, int KSC, bool DENSE, bool QUIET, bool CUT>
__global__ void __launch_bounds__(WARPS * 32, NC > 1 ? 3 : DENSE ? 4 : 1)
recurrent_scan_vec_kernel(const float* q, int ldq, const float* k, int ldk, const float* v, int ldv, const float* z, int ldz,
                          const float* beta, int ldb, float q_scale,
                          float* state, size_t slot_stride, const int* __restrict__ slots, const int* __restrict__ cu_q,
                          float* out, int H, int G, int dk, int dv, int lanes, int chunk, int vec,
                          int nc, int n_cut, int* places, float* part_s, float* part_p, const float* part_start) {
    bl_pdl_trigger();
    bl_pdl_wait();
    extern __shared__ __align__(16) float sm[];
    constexpr bool DELTA = RULE == BL_RULE_DELTA, BONUS = RULE == BL_RULE_BONUS;
    constexpr int RK = RK4 * 4, RP = RK / 2;                     // rows a lane holds, pairs of them
    const int KS = KSC ? KSC : lanes;
    // A long portion of a request may be cut into nc parts that run side by side (the recurrence is linear in S). First pass
    // (QUIET): every part from a ZERO state, leaving its own contribution S_part and its transition P (a product of decays a
    // row; of the delta rule a matrix). Between the passes a fold (S <- P S + S_part) leaves every part's start state in
    // scratch and the final state in the slot. Second pass: a part runs from its start state and writes the outputs. Short
    // portions (and nc 1, and long ones past the n_cut that scratch is there for) take one block per (request, head, columns)
    // through the second pass alone.
    const int r = CUT ? blockIdx.z / nc : blockIdx.z, part = CUT ? blockIdx.z % nc : 0, h = blockIdx.y;
    const int n_all = cu_q[r + 1] - cu_q[r];
    if (n_all <= 0) return;
    // The first pass counts out a request's place in the scratch (-1: not cut) and leaves it for the launches behind it;
    // where scratch is there for all requests, it is r. (Counted
    // in the second pass too, it cost the walk in one piece its registers: 188 -> 204, 8 heads of 128 x 256 385 -> 436 us.)
    int place = 0;
    if (QUIET) {
        place = n_all < SCAN_SPLIT_MIN ? -1 : places ? scan_cut_place(cu_q, r) : r;
        if (place >= n_cut) place = -1;
        if (places && blockIdx.x == 0 && h == 0 && part == 0 && threadIdx.x == 0) places[r] = place;
    } else if (CUT && nc > 1) {
        place = places ? places[r] : n_all >= SCAN_SPLIT_MIN ? r : -1;
    }
    const bool split = CUT && nc > 1 && place >= 0;
    if (!split && (part != 0 || QUIET)) return;
    // (of more parts than tokens some are empty: they leave a zero state and the identity)
    const int t_first = split ? (int)((long long)part * n_all / nc) : 0;
    const int t0 = cu_q[r] + t_first, n = (split ? (int)((long long)(part + 1) * n_all / nc) : n_all) - t_first;
    const int gh = h / (H / G);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int CW = 32 / KS, cols_blk = WARPS * CW * NC;          // CW: lanes side by side along the columns
    const int s = lane / CW, cc = lane % CW;
    const int c = ((blockIdx.x * WARPS + warp) * CW + cc) * NC;  // the lane's first column (NC 4: dv and dk are multiples of 4)
    // The delta rule's transition over a part is a key x key matrix: pass 1 makes it in dk further columns that start as
    // the identity and see values of zero (column dv + j ends as the part's transition applied to unit vector j).
    const int n_cols = dv + (DELTA && QUIET ? dk : 0);
    const bool col_ok = c < n_cols;
    const int per_tok = 3 * dk + cols_blk + 4;
    const int buf_floats = chunk * per_tok;
    float* S = state + (size_t)slots[r] * slot_stride + (size_t)h * dk * dv;
    const int col0 = blockIdx.x * cols_blk;
    if (col0 >= n_cols) return;
    const int row0 = s * RK;

    auto issue = [&](int base, float* buf) {
        const int m = min(chunk, n - base);
        for (int tt = warp; tt < m; tt += WARPS) {
            const size_t tok = (size_t)(t0 + base + tt);
            float* dst = buf + (size_t)tt * per_tok;
            const float* gq = q + tok * ldq + gh * dk;
            const float* gk = k + tok * ldk + gh * dk;
            const float* gz = z + tok * ldz + h * dk;
            if (vec) {
                for (int d = lane * 4; d < dk; d += 128) {
                    if (!QUIET) cp_async16(dst + d, gq + d);
                    cp_async16(dst + dk + d, gk + d); cp_async16(dst + 2 * dk + d, gz + d);
                }
            } else {
                for (int d = lane; d < dk; d += 32) {
                    if (!QUIET) cp_async4(dst + d, gq + d);
                    cp_async4(dst + dk + d, gk + d); cp_async4(dst + 2 * dk + d, gz + d);
                }
            }
            const float* gv = v + tok * ldv + h * dv + col0;
            if (NC > 1) {
                for (int j = lane * 4; j < cols_blk; j += 128) {
                    if (col0 + j < dv) cp_async16(dst + 3 * dk + j, gv + j);
                    else *reinterpret_cast<float4*>(dst + 3 * dk + j) = make_float4(0.f, 0.f, 0.f, 0.f);
                }
            } else
            for (int j = lane; j < cols_blk; j += 32) {
                if (col0 + j < dv) cp_async4(dst + 3 * dk + j, gv + j);
                else dst[3 * dk + j] = 0.f;
            }
            if ((DELTA || BONUS) && lane == 0) cp_async4(dst + 3 * dk + cols_blk, beta + tok * ldb + h);
        }
        cp_async_commit();
    };

    issue(0, sm);
    uint64_t st[NC][RP], pr[QUIET && !DELTA ? RP : 1];           // a column's rows in pairs
    const size_t part_base = ((size_t)place * nc) * H + h;       // + p * H for part p
    auto read_row = [&](const float* p, float (&x)[NC]) {        // the lane's columns of a row
        if constexpr (NC == 4) {
            const float4 f = *reinterpret_cast<const float4*>(p);
            x[0] = f.x; x[1] = f.y; x[2] = f.z; x[3] = f.w;
        } else {
            x[0] = *p;
        }
    };
    auto write_row = [&](float* p, const float (&x)[NC]) {
        if constexpr (NC == 4) *reinterpret_cast<float4*>(p) = make_float4(x[0], x[1], x[2], x[3]);
        else *p = x[0];
    };
    const float* start = split ? part_start + ((part_base + (size_t)part * H) * dk + row0) * dv + c : S + (size_t)row0 * dv + c;
#pragma unroll
    for (int i = 0; i < RP; ++i) {
        float a[NC], b[NC];
#pragma unroll
        for (int j = 0; j < NC; ++j) {
            a[j] = QUIET && DELTA && c + j >= dv && row0 + 2 * i == c + j - dv ? 1.f : 0.f;
            b[j] = QUIET && DELTA && c + j >= dv && row0 + 2 * i + 1 == c + j - dv ? 1.f : 0.f;
        }
        if (!QUIET && col_ok) { read_row(start + (size_t)(2 * i) * dv, a); read_row(start + (size_t)(2 * i + 1) * dv, b); }
#pragma unroll
        for (int j = 0; j < NC; ++j) st[j][i] = f2_pack(a[j], b[j]);
        if (QUIET && !DELTA) pr[QUIET && !DELTA ? i : 0] = f2_pack(1.f, 1.f);
    }
    // the lane's columns of its rows, to `p` with rows dv (or dk) apart
    auto write_state = [&](float* p, int ld) {
#pragma unroll
        for (int i = 0; i < RP; ++i) {
            float a[NC], b[NC];
#pragma unroll
            for (int j = 0; j < NC; ++j) f2_unpack(st[j][i], a[j], b[j]);
            write_row(p + (size_t)(2 * i) * ld, a);
            write_row(p + (size_t)(2 * i + 1) * ld, b);
        }
    };
    const int v_off = 3 * dk + (warp * CW + cc) * NC, b_off = 3 * dk + cols_blk;
    const int dk4 = dk >> 2;

    struct Tok { ulonglong2 q[QUIET ? 1 : RK4], k[RK4], d[RK4]; float v[NC], b; };
    auto fetch = [&](const float* tokp, Tok& t) {
        const ulonglong2* p4 = reinterpret_cast<const ulonglong2*>(tokp + row0);
#pragma unroll
        for (int j = 0; j < RK4; ++j) {
            if (!QUIET) t.q[QUIET ? 0 : j] = p4[j];
            t.k[j] = p4[dk4 + j]; t.d[j] = p4[2 * dk4 + j];
        }
        if constexpr (NC == 4) {
            const float4 x = *reinterpret_cast<const float4*>(tokp + v_off);
            t.v[0] = x.x; t.v[1] = x.y; t.v[2] = x.z; t.v[3] = x.w;
        } else {
            t.v[0] = tokp[v_off];
        }
        t.b = (DELTA || BONUS) ? tokp[b_off] : 0.f;
    };
    // The sums of a column's rows over the KS lanes that hold them, always in the order of the butterfly. With four columns a
    // lane gives the sums away that it does not go on with: two after the first exchange, one after the second; it ends with `kept`
    // of them, from column `mine` on.
    const int kept = NC == 1 || KS == 1 ? NC : KS == 2 ? 2 : 1;
    const int mine = NC == 1 || KS == 1 ? 0 : KS == 2 ? (lane >> 4) * 2 : (lane >> 4) * 2 + ((lane >> 3) & 1);
    const bool speaks = NC == 1 ? s == 0 : KS <= 4 || (s & (KS / 4 - 1)) == 0;       // of the lanes that end with equal sums, one writes them
    auto column_sums = [&](float (&o)[NC]) {
        if constexpr (NC == 1) {
            for (int x = 16; x >= CW; x >>= 1) o[0] += __shfl_xor_sync(0xffffffffu, o[0], x);
        } else if (KS > 1) {
            const bool up = (lane & 16) != 0;
            const float g0 = __shfl_xor_sync(0xffffffffu, up ? o[0] : o[2], 16), g1 = __shfl_xor_sync(0xffffffffu, up ? o[1] : o[3], 16);
            o[0] = (up ? o[2] : o[0]) + g0;
            o[1] = (up ? o[3] : o[1]) + g1;
            if (KS > 2) {
                const bool up2 = (lane & 8) != 0;
                const float g = __shfl_xor_sync(0xffffffffu, up2 ? o[0] : o[1], 8);
                o[0] = (up2 ? o[1] : o[0]) + g;
                for (int x = 4; x >= CW; x >>= 1) o[0] += __shfl_xor_sync(0xffffffffu, o[0], x);
            }
        }
    };
    auto kept_of = [&](const float (&a)[NC], int j) {            // a[mine + j], without an index that is not known
        if constexpr (NC == 1) return a[0];
        else if (KS == 1) return a[j];
        else if (KS == 2) return mine ? a[2 + (j & 1)] : a[j & 1];
        else return mine & 2 ? (mine & 1 ? a[3] : a[2]) : (mine & 1 ? a[1] : a[0]);
    };
    auto step = [&](const Tok& t, size_t tok) {
        auto q2 = [&](int i) { return i & 1 ? t.q[QUIET ? 0 : i >> 1].y : t.q[QUIET ? 0 : i >> 1].x; };
        auto k2 = [&](int i) { return i & 1 ? t.k[i >> 1].y : t.k[i >> 1].x; };
        auto d2 = [&](int i) { return i & 1 ? t.d[i >> 1].y : t.d[i >> 1].x; };
        const uint64_t zero = f2_pack(0.f, 0.f);
        auto both = [](uint64_t x) { float a, b; f2_unpack(x, a, b); return a + b; };
        float o[NC], u[NC];
        if (!DELTA) {
#pragma unroll
            for (int j = 0; j < NC; ++j) {
                const uint64_t v2 = f2_pack(t.v[j], t.v[j]);
                uint64_t o2 = zero;
#pragma unroll
                for (int i = 0; i < RP; ++i) {
                    if (BONUS && !QUIET) o2 = f2_fma(st[j][i], q2(i), o2);                       // the state before the write
                    st[j][i] = f2_fma(d2(i), st[j][i], f2_mul(k2(i), v2));
                    if (!BONUS && !QUIET) o2 = f2_fma(st[j][i], q2(i), o2);
                }
                o[j] = both(o2);
            }
            if (QUIET) {
#pragma unroll
                for (int i = 0; i < (QUIET && !DELTA ? RP : 1); ++i) pr[i] = f2_mul(pr[i], d2(i));
                return;
            }
            column_sums(o);
        } else {
            float sk[NC], sq[NC];
            uint64_t kq2 = zero;
#pragma unroll
            for (int j = 0; j < NC; ++j) {
                uint64_t sk2 = zero, sq2 = zero;
#pragma unroll
                for (int i = 0; i < RP; ++i) {
                    st[j][i] = f2_mul(st[j][i], d2(i));
                    sk2 = f2_fma(st[j][i], k2(i), sk2);
                    if (!QUIET) {
                        sq2 = f2_fma(st[j][i], q2(i), sq2);
                        if (j == 0) kq2 = f2_fma(k2(i), q2(i), kq2);
                    }
                }
                sk[j] = both(sk2); sq[j] = both(sq2);
            }
            float kq = both(kq2);
            for (int x = 16; x >= CW; x >>= 1) {                 // every lane needs the columns' S^T k
#pragma unroll
                for (int j = 0; j < NC; ++j) sk[j] += __shfl_xor_sync(0xffffffffu, sk[j], x);
                if (!QUIET) kq += __shfl_xor_sync(0xffffffffu, kq, x);
            }
            if (!QUIET) column_sums(sq);
#pragma unroll
            for (int j = 0; j < NC; ++j) u[j] = t.b * (t.v[j] - sk[j]);
#pragma unroll
            for (int j = 0; j < NC; ++j) {
                const uint64_t u2 = f2_pack(u[j], u[j]);
#pragma unroll
                for (int i = 0; i < RP; ++i) st[j][i] = f2_fma(k2(i), u2, st[j][i]);
            }
            if (!QUIET) {
#pragma unroll
                for (int j = 0; j < NC; ++j) o[j] = j < kept ? fmaf(kq, kept_of(u, j), sq[j]) : 0.f;
            }
        }
        if (!QUIET && speaks && col_ok) {
            float* dst = out + tok * H * dv + h * dv + c + mine;
#pragma unroll
            for (int j = 0; j < NC; ++j)
                if (j < kept) dst[j] = (BONUS ? fmaf(t.b, kept_of(t.v, j), o[j]) : o[j]) * q_scale;
        }
    };

    int which = 0;
    for (int base = 0; base < n; base += chunk, which ^= 1) {
        const int m = min(chunk, n - base);
        float* buf = sm + (size_t)which * buf_floats;
        if (base + chunk < n) { issue(base + chunk, sm + (size_t)(which ^ 1) * buf_floats); cp_async_wait<1>(); }
        else cp_async_wait<0>();
        __syncthreads();
        if (DELTA) {
            for (int tt = threadIdx.x; tt < m; tt += WARPS * 32) {
                float* b = buf + (size_t)tt * per_tok + b_off;
                *b = sigmoidf_(*b);
            }
            __syncthreads();
        }
        const size_t tok0 = (size_t)(t0 + base);
        int tt = 0;
        if (DENSE) {
            for (; tt < m; ++tt) {
                Tok t;
                fetch(buf + (size_t)tt * per_tok, t);
                step(t, tok0 + tt);
            }
            __syncthreads();
            continue;
        }
        Tok ta, tb;
        fetch(buf, ta);
        for (; tt + 1 < m; tt += 2) {
            fetch(buf + (size_t)(tt + 1) * per_tok, tb);
            step(ta, tok0 + tt);
            if (tt + 2 < m) fetch(buf + (size_t)(tt + 2) * per_tok, ta);
            step(tb, tok0 + tt + 1);
        }
        if (tt < m) step(ta, tok0 + tt);
        __syncthreads();                               // the buffer is free for the chunk after next
    }
    if (split) {
        if (QUIET && DELTA) {
            float* ps = part_s + (part_base + (size_t)part * H) * dk * dv;
            float* pm = part_p + (part_base + (size_t)part * H) * dk * dk;      // [row][unit vector]
            if (c < dv) write_state(ps + (size_t)row0 * dv + c, dv);
            else if (col_ok) write_state(pm + (size_t)row0 * dk + (c - dv), dk);
        } else if (QUIET) {
            float* ps = part_s + (part_base + (size_t)part * H) * dk * dv;
            float* pp = part_p + (part_base + (size_t)part * H) * dk;
            if (col_ok) write_state(ps + (size_t)row0 * dv + c, dv);
            if (blockIdx.x == 0 && warp == 0 && cc == 0) {
#pragma unroll
                for (int i = 0; i < (QUIET && !DELTA ? RP : 1); ++i) {
                    float a, b;
                    f2_unpack(pr[i], a, b);
                    pp[row0 + 2 * i] = a; pp[row0 + 2 * i + 1] = b;
                }
            }
        }
        return;                                        // the slot is written by the fold
    }
    if (col_ok) write_state(S + (size_t)row0 * dv + c, dv);
}

// Between the two passes of a cut portion of the delta rule: start[0] = the slot's state, start[p + 1] = P_p start[p] +
// S_part_p (P_p a key x key matrix), the last one into the slot. A block owns FOLD_COLS columns of one (request, head) and
// keeps the current state's columns in shared memory, two buffers taking turns. The parts follow one another, so a part's
// time is a chain of trips to L2: few columns a block (more blocks), P in 16-byte pieces, a row's pieces in flight together.
constexpr int FOLD_COLS = 8, FOLD_MAX_DK = 128;
__global__ void __launch_bounds__(256)
scan_fold_matrix_kernel(float* state, size_t slot_stride, const int* __restrict__ slots, const int* __restrict__ cu_q,
                        const int* places, const float* part_s, const float* part_pm, float* part_start, int H, int dk, int dv, int nc) {
    bl_pdl_trigger();
    bl_pdl_wait();
    __shared__ float cur[2][FOLD_MAX_DK][FOLD_COLS];
    const int r = blockIdx.z, h = blockIdx.y, c0 = blockIdx.x * FOLD_COLS;
    if (cu_q[r + 1] - cu_q[r] < SCAN_SPLIT_MIN) return;
    const int place = places ? places[r] : r;
    if (place < 0) return;
    float* S = state + (size_t)slots[r] * slot_stride + (size_t)h * dk * dv;
    const size_t base = ((size_t)place * nc) * H + h;
    const int col = threadIdx.x % FOLD_COLS, rg = threadIdx.x / FOLD_COLS;
    constexpr int GROUPS = 256 / FOLD_COLS;                                     // row groups
    const bool ok = c0 + col < dv;
    for (int row = rg; row < dk; row += GROUPS) {
        const float x = ok ? S[(size_t)row * dv + c0 + col] : 0.f;
        cur[0][row][col] = x;
        if (ok) part_start[((base + 0) * dk + row) * dv + c0 + col] = x;
    }
    __syncthreads();
    int w = 0;
    for (int p = 0; p < nc; ++p, w ^= 1) {
        const float* pm = part_pm + (base + (size_t)p * H) * dk * dk;
        const float* ps = part_s + (base + (size_t)p * H) * dk * dv;
        for (int row = rg; row < dk; row += GROUPS) {
            float acc = ok ? ps[(size_t)row * dv + c0 + col] : 0.f;
            const float4* prow = reinterpret_cast<const float4*>(pm + (size_t)row * dk);    // dk is a multiple of 4
#pragma unroll 8
            for (int j = 0; j < dk >> 2; ++j) {
                const float4 a = prow[j];
                acc = fmaf(a.x, cur[w][4 * j][col], acc); acc = fmaf(a.y, cur[w][4 * j + 1][col], acc);
                acc = fmaf(a.z, cur[w][4 * j + 2][col], acc); acc = fmaf(a.w, cur[w][4 * j + 3][col], acc);
            }
            cur[w ^ 1][row][col] = acc;
            if (ok) {
                if (p + 1 < nc) part_start[((base + (size_t)(p + 1) * H) * dk + row) * dv + c0 + col] = acc;
                else S[(size_t)row * dv + c0 + col] = acc;
            }
        }
        __syncthreads();
    }
}

// The same for values in groups of four: a thread holds the TPR-th part of a row of P (up to 64 values) in registers, the next part's
// on its way while it multiplies this one's, and 4 GROUPS columns of the state, which all rows read from shared memory as broadcasts. The
// kernel above asks for a part's P when the part before it is done, a trip to L2 (or two) a part, and reads the state a value
// at a time. Sums in its order (two halves of a row, where there are two, added at the end).
template <int TPR, int GROUPS>
__global__ void __launch_bounds__(TPR == 1 ? 64 : 256)
scan_fold_matrix4_kernel(float* state, size_t slot_stride, const int* __restrict__ slots, const int* __restrict__ cu_q,
                         const int* places, const float* part_s, const float* part_pm, float* part_start, int H, int dk, int dv, int nc) {
    bl_pdl_trigger();
    bl_pdl_wait();
    constexpr int PIECES = 16;                          // of four values of P a thread
    __shared__ float4 cur[2][FOLD_MAX_DK][GROUPS];
    const int r = blockIdx.z, h = blockIdx.y, c0 = blockIdx.x * 4 * GROUPS;
    if (cu_q[r + 1] - cu_q[r] < SCAN_SPLIT_MIN) return;
    const int place = places ? places[r] : r;
    if (place < 0) return;
    float* S = state + (size_t)slots[r] * slot_stride + (size_t)h * dk * dv;
    const size_t base = ((size_t)place * nc) * H + h;
    const int row = threadIdx.x / TPR, half = threadIdx.x % TPR, k0 = half * 4 * PIECES;
    const int pieces = min(PIECES, (dk - k0) >> 2);     // dk is a multiple of 4
    float4 pa[PIECES], pb[PIECES], sa[GROUPS], sb[GROUPS];
    auto fetch = [&](int p, float4 (&m)[PIECES], float4 (&a)[GROUPS]) {
        if (p >= nc) return;
        const float4* pm = reinterpret_cast<const float4*>(part_pm + ((base + (size_t)p * H) * dk + row) * dk + k0);
#pragma unroll
        for (int j = 0; j < PIECES; ++j)
            if (j < pieces) m[j] = pm[j];
        const float4* ps = reinterpret_cast<const float4*>(part_s + ((base + (size_t)p * H) * dk + row) * dv + c0);
#pragma unroll
        for (int g = 0; g < GROUPS; ++g)
            a[g] = half == 0 && c0 + 4 * g < dv ? ps[g] : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    auto part = [&](int p, const float4 (&m)[PIECES], const float4 (&a)[GROUPS]) {
        const int w = p & 1;
        float4 acc[GROUPS];
#pragma unroll
        for (int g = 0; g < GROUPS; ++g) acc[g] = a[g];
#pragma unroll
        for (int j = 0; j < PIECES; ++j) {
            if (j >= pieces) continue;
            const float e[4] = {m[j].x, m[j].y, m[j].z, m[j].w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int g = 0; g < GROUPS; ++g) {
                    const float4 c = cur[w][k0 + 4 * j + i][g];
                    acc[g].x = fmaf(e[i], c.x, acc[g].x); acc[g].y = fmaf(e[i], c.y, acc[g].y);
                    acc[g].z = fmaf(e[i], c.z, acc[g].z); acc[g].w = fmaf(e[i], c.w, acc[g].w);
                }
        }
#pragma unroll
        for (int g = 0; g < GROUPS; ++g) {
            if (TPR == 2) {
                acc[g].x += __shfl_xor_sync(0xffffffffu, acc[g].x, 1); acc[g].y += __shfl_xor_sync(0xffffffffu, acc[g].y, 1);
                acc[g].z += __shfl_xor_sync(0xffffffffu, acc[g].z, 1); acc[g].w += __shfl_xor_sync(0xffffffffu, acc[g].w, 1);
            }
            if (half == 0) {
                cur[w ^ 1][row][g] = acc[g];
                if (c0 + 4 * g < dv) {
                    float* to = p + 1 < nc ? part_start + ((base + (size_t)(p + 1) * H) * dk + row) * dv : S + (size_t)row * dv;
                    *reinterpret_cast<float4*>(to + c0 + 4 * g) = acc[g];
                }
            }
        }
        __syncthreads();
    };
    fetch(0, pa, sa);
#pragma unroll
    for (int g = 0; g < GROUPS; ++g) {
        if (half != 0) continue;
        const bool ok = c0 + 4 * g < dv;
        const float4 x = ok ? *reinterpret_cast<const float4*>(S + (size_t)row * dv + c0 + 4 * g) : make_float4(0.f, 0.f, 0.f, 0.f);
        cur[0][row][g] = x;
        if (ok) *reinterpret_cast<float4*>(part_start + (base * dk + row) * dv + c0 + 4 * g) = x;
    }
    __syncthreads();
    for (int p = 0; p < nc; p += 2) {
        fetch(p + 1, pb, sb);
        part(p, pa, sa);
        if (p + 1 >= nc) break;
        fetch(p + 2, pa, sa);
        part(p + 1, pb, sb);
    }
}

// The same where the transition is a decay per row: start[p + 1] = P_p o start[p] + S_part_p. Every part's start takes the
// place of its contribution in part_s.
__global__ void scan_fold_kernel(float* state, size_t slot_stride, const int* __restrict__ slots, const int* __restrict__ cu_q,
                                 const int* places, float* part_s, const float* part_p, int H, int dk, int dv, int nc) {
    bl_pdl_trigger();
    bl_pdl_wait();
    const int r = blockIdx.z, h = blockIdx.y;
    if (cu_q[r + 1] - cu_q[r] < SCAN_SPLIT_MIN) return;
    const int place = places ? places[r] : r;
    if (place < 0) return;
    float* S = state + (size_t)slots[r] * slot_stride + (size_t)h * dk * dv;
    const size_t base = ((size_t)place * nc) * H + h;
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= dk * dv) return;
    const int row = e / dv;
    float sv = S[e];
    for (int p0 = 0; p0 < nc; p0 += 8) {               // eight parts' values in flight
        float add[8], mul[8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (p0 + i < nc) {
                mul[i] = part_p[(base + (size_t)(p0 + i) * H) * dk + row];
                add[i] = part_s[(base + (size_t)(p0 + i) * H) * dk * dv + e];
            }
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (p0 + i < nc) {
                part_s[(base + (size_t)(p0 + i) * H) * dk * dv + e] = sv;
                sv = fmaf(mul[i], sv, add[i]);
            }
    }
    S[e] = sv;
}

// y[t, h, :] = u / sqrt(mean(u^2) + eps) * w * gate(g[t, h, :]); w is one vector of dv values shared by the heads, or
// (w_per_head) H * dv values. The heads of a row of o lie o_head_stride values apart. floor null: u = o[t, h, :dv]; else
// u = o[t, h, :dv] / (max(|o[t, h, dv]|, floor[t, h]) + 1e-6): the read-out of a matrix memory whose normaliser was walked
// as one more value column. One warp per (token, head).
template <typename TY>
__global__ void __launch_bounds__(WARPS * 32)
head_norm_gate_kernel(const float* o, int o_head_stride, const void* __restrict__ w, int w_dtype, int w_per_head, const float* floor,
                      const float* gate, int ld_gate, int gate_kind, TY* __restrict__ y, int items, int H, int dv, float eps) {
    bl_pdl_trigger();
    bl_pdl_wait();
    const int lane = threadIdx.x & 31;
    const int item = blockIdx.x * WARPS + (threadIdx.x >> 5);
    if (item >= items) return;
    const int t = item / H, h = item % H;
    const float* src = o + (size_t)item * o_head_stride;
    const float pre = floor ? 1.0f / (fmaxf(fabsf(src[dv]), floor[item]) + 1e-6f) : 1.0f;
    float ss = 0.f;
    for (int i = lane; i < dv; i += 32) { const float u = src[i] * pre; ss += u * u; }
    const float inv = pre / sqrtf(bl_warp_sum(ss) / (float)dv + eps);
    const float* g = gate ? gate + (size_t)t * ld_gate + h * dv : nullptr;
    const size_t w0 = w_per_head ? (size_t)h * dv : 0;
    for (int i = lane; i < dv; i += 32) {
        float val = src[i] * inv * (w ? bl_load_any(w, w_dtype, w0 + i) : 1.f);
        if (g) val *= gate_kind == BL_GATE_SILU ? bl_silu(g[i]) : sigmoidf_(g[i]);
        bl_store(y + (size_t)item * dv + i, val);
    }
}

// The same for heads of whole groups of four (and no read-out to divide): a lane holds its values from the first read, with
// gate and weight on their way beside them. The kernel above reads value by value, and a gate behind the sum (1,840 rows of 8 heads of
// 256 14.5 us, 8 rows in a decode step's chain 5).
template <typename TY, int NV>
__global__ void __launch_bounds__(WARPS * 32)
head_norm_gate4_kernel(const float* o, int o_head_stride, const void* __restrict__ w, int w_dtype, int w_per_head,
                       const float* gate, int ld_gate, int gate_kind, TY* __restrict__ y, int items, int H, int dv, float eps) {
    bl_pdl_trigger();
    const int lane = threadIdx.x & 31;
    const int item = blockIdx.x * WARPS + (threadIdx.x >> 5);
    const int t = item / H, h = item % H;
    const size_t w0 = w_per_head ? (size_t)h * dv : 0;
    float wv[NV][4];
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        const int i = (lane + 32 * j) * 4;
#pragma unroll
        for (int e = 0; e < 4; ++e) wv[j][e] = w && i < dv ? bl_load_any(w, w_dtype, w0 + i + e) : 1.f;
    }
    bl_pdl_wait();
    if (item >= items) return;
    const float* src = o + (size_t)item * o_head_stride;
    const float* g = gate ? gate + (size_t)t * ld_gate + h * dv : nullptr;
    float4 v[NV], gv[NV];
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        const int i = (lane + 32 * j) * 4;
        v[j] = i < dv ? *reinterpret_cast<const float4*>(src + i) : make_float4(0.f, 0.f, 0.f, 0.f);
        if (g && i < dv) gv[j] = *reinterpret_cast<const float4*>(g + i);
    }
#pragma unroll
    for (int j = 0; j < NV; ++j) ss += (v[j].x * v[j].x + v[j].y * v[j].y) + (v[j].z * v[j].z + v[j].w * v[j].w);
    const float inv = 1.0f / sqrtf(bl_warp_sum(ss) / (float)dv + eps);
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        const int i = (lane + 32 * j) * 4;
        if (i >= dv) continue;
        const float* u = reinterpret_cast<const float*>(&v[j]);
        const float* gg = reinterpret_cast<const float*>(&gv[j]);
        float out[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            out[e] = u[e] * inv * wv[j][e];
            if (g) out[e] *= gate_kind == BL_GATE_SILU ? bl_silu(gg[e]) : sigmoidf_(gg[e]);
        }
        store4(y + (size_t)item * dv + i, out[0], out[1], out[2], out[3]);
    }
}

// The gates of a matrix memory with exponential gating: one warp per (request, head) walks the request's tokens in order.
// Per token: log input gate i = cap tanh((zi + bi) / cap), log forget gate f = log sigmoid(cap tanh((zf + bf) / cap)), the
// running maximum m' = max(f + m, i) (m starts at 0 in a fresh slot and is kept in the slot at off_m), and from them the
// decay a = e^(f + m - m'), the input weight e = e^(i - m') and the floor e^(-m') of the read-out's denominator, into
// gates [3, T, H]. 32 tokens at a time: their gates in parallel (a lane each; the next 32 tokens' pre-activations are
// fetched before), the maxima as a chain of 32 steps of two dependent instructions.
__global__ void __launch_bounds__(32)
memory_gate_chain_kernel(const float* proj, int ld, int off_i, int off_f, const void* __restrict__ bi, int bi_dtype,
                         const void* __restrict__ bf, int bf_dtype, float cap, float* state, size_t slot_stride, size_t off_m,
                         const int* __restrict__ slots, const int* __restrict__ cu_q, float* gates, int T, int H) {
    bl_pdl_trigger();
    bl_pdl_wait();
    const int r = blockIdx.y, h = blockIdx.x, lane = threadIdx.x;
    const int t0 = cu_q[r], n_tok = cu_q[r + 1] - t0;
    if (n_tok <= 0) return;
    float* mp = state + (size_t)slots[r] * slot_stride + off_m + h;
    float m = *mp;
    const float b_i = bl_load_any(bi, bi_dtype, h), b_f = bl_load_any(bf, bf_dtype, h);
    const float inv_cap = 1.0f / cap;
    float zi = 0.f, zf = 0.f;
    if (lane < n_tok) { const float* row = proj + (size_t)(t0 + lane) * ld; zi = row[off_i + h]; zf = row[off_f + h]; }
    for (int base = 0; base < n_tok; base += 32) {
        const int cnt = min(32, n_tok - base);
        float nzi = 0.f, nzf = 0.f;
        if (base + 32 + lane < n_tok) { const float* row = proj + (size_t)(t0 + base + 32 + lane) * ld; nzi = row[off_i + h]; nzf = row[off_f + h]; }
        const float gi = cap * tanhf((zi + b_i) * inv_cap);
        const float z = cap * tanhf((zf + b_f) * inv_cap);
        const float gf = fminf(z, 0.f) - log1pf(expf(-fabsf(z)));
        float m_before = 0.f, m_mine = 0.f;
        for (int tt = 0; tt < cnt; ++tt) {
            const float f_t = __shfl_sync(0xffffffffu, gf, tt), i_t = __shfl_sync(0xffffffffu, gi, tt);
            const float m_new = fmaxf(f_t + m, i_t);
            if (lane == tt) { m_before = m; m_mine = m_new; }
            m = m_new;
        }
        if (lane < cnt) {
            const size_t at = (size_t)(t0 + base + lane) * H + h;
            gates[at] = expf(gf + m_before - m_mine);
            gates[(size_t)T * H + at] = expf(gi - m_mine);
            gates[2 * (size_t)T * H + at] = expf(-m_mine);
        }
        zi = nzi; zf = nzf;
    }
    if (lane == 0) *mp = m;
}

// What the scan of a matrix memory reads, from the projections and the gates: decay[t, h, :] = a[t, h] for every key
// channel, k_out[t, h, :] = e[t, h] * k[t, h, :], v_out[t, h, :] = (v[t, h, :], 1): the one in the last column makes the
// normaliser n the state's last value column, and n . q the last column of the read-out. One block per token.
__global__ void __launch_bounds__(WARPS * 32)
memory_expand_kernel(const float* proj, int ld, int off_k, int off_v, const float* __restrict__ gates, float* decay, float* k_out,
                     float* v_out, int T, int H, int dk, int dv) {
    bl_pdl_trigger();
    bl_pdl_wait();
    const int t = blockIdx.x;
    const float* row = proj + (size_t)t * ld;
    for (int e = threadIdx.x; e < H * dk; e += WARPS * 32) {
        const size_t g = (size_t)t * H + e / dk;
        decay[(size_t)t * H * dk + e] = gates[g];
        k_out[(size_t)t * H * dk + e] = gates[(size_t)T * H + g] * row[off_k + e];
    }
    for (int e = threadIdx.x; e < H * (dv + 1); e += WARPS * 32) {
        const int h = e / (dv + 1), c = e % (dv + 1);
        v_out[(size_t)t * H * (dv + 1) + e] = c < dv ? row[off_v + h * dv + c] : 1.0f;
    }
}

// Token shift: out[s, t, c] = x[t, c] + (x'[t, c] - x[t, c]) * mu[s, c] for s < n_mix, x' the row of the request's token
// before (from the slot's `prev` [d] for a step's first token: zeros in a fresh slot). One block per token; four channels
// a thread (16-byte loads, 8- or 16-byte stores) where the rows allow it.
template <typename TY>
__global__ void __launch_bounds__(WARPS * 32)
shift_mix_kernel(const float* x, int ld, const float* __restrict__ mu, int n_mix, const float* prev, size_t slot_stride,
                 const int* __restrict__ slots, const int* __restrict__ tok_req, const int* __restrict__ cu_q, TY* __restrict__ out,
                 int T, int d, int vec) {
    bl_pdl_trigger();
    bl_pdl_wait();
    const int t = blockIdx.x;
    const int r = tok_req[t];
    const float* before = t > cu_q[r] ? x + (size_t)(t - 1) * ld : prev + (size_t)slots[r] * slot_stride;
    const float* cur = x + (size_t)t * ld;
    if (vec) {
        for (int c = threadIdx.x * 4; c < d; c += WARPS * 32 * 4) {
            const float4 xc = *reinterpret_cast<const float4*>(cur + c), xb = *reinterpret_cast<const float4*>(before + c);
            const float4 dx = make_float4(xb.x - xc.x, xb.y - xc.y, xb.z - xc.z, xb.w - xc.w);
            for (int s = 0; s < n_mix; ++s) {
                const float4 m = *reinterpret_cast<const float4*>(mu + (size_t)s * d + c);
                store4(out + ((size_t)s * T + t) * d + c, fmaf(dx.x, m.x, xc.x), fmaf(dx.y, m.y, xc.y), fmaf(dx.z, m.z, xc.z), fmaf(dx.w, m.w, xc.w));
            }
        }
        return;
    }
    for (int c = threadIdx.x; c < d; c += WARPS * 32) {
        const float xc = cur[c], dx = before[c] - xc;
        for (int s = 0; s < n_mix; ++s)
            bl_store(out + ((size_t)s * T + t) * d + c, fmaf(dx, mu[(size_t)s * d + c], xc));
    }
}

// b[t, h] = sum_c u[h, c] * k[t, h, c] * q[t, h, c]: what the current token adds to its own read-out; one warp per (t, h).
__global__ void __launch_bounds__(WARPS * 32)
bonus_dot_kernel(const float* q, int ldq, const float* k, int ldk, const void* __restrict__ u, int u_dtype, float* out,
                 int items, int H, int dk) {
    bl_pdl_trigger();
    bl_pdl_wait();
    const int lane = threadIdx.x & 31;
    const int item = blockIdx.x * WARPS + (threadIdx.x >> 5);
    if (item >= items) return;
    const int t = item / H, h = item % H;
    const float* qr = q + (size_t)t * ldq + (size_t)h * dk;
    const float* kr = k + (size_t)t * ldk + (size_t)h * dk;
    float acc = 0.f;
    for (int c = lane; c < dk; c += 32) acc = fmaf(bl_load_any(u, u_dtype, (size_t)h * dk + c) * kr[c], qr[c], acc);
    acc = bl_warp_sum(acc);
    if (lane == 0) out[item] = acc;
}

// One block per token: y[t, ch] = silu(sum_i taps[ch, i] * x[t - (n_taps - 1) + i, ch]), the inputs before the step's
// first token of the request coming from the slot's tail (its last n_taps - 1 inputs, oldest first; zeros at the
// start of a sequence). Then the first `unit_heads` heads of `dk` columns are made unit vectors, x / sqrt(sum x^2 +
// unit_eps), the first `scaled_heads` of them also times q_scale.
__global__ void __launch_bounds__(WARPS * 32)
conv_silu_unit_kernel(const float* x, int ld, const float* __restrict__ taps, int n_taps, const float* tail, size_t slot_stride,
                      const int* __restrict__ slots, const int* __restrict__ tok_req, const int* __restrict__ cu_q, float* y,
                      int C, int unit_heads, int scaled_heads, int dk, float q_scale, float unit_eps, const void* __restrict__ bias,
                      int bias_dtype) {
    bl_pdl_trigger();
    bl_pdl_wait();
    const int t = blockIdx.x;
    const int r = tok_req[t];
    const int j = t - cu_q[r];
    const float* tl = tail + (size_t)slots[r] * slot_stride;
    for (int ch = threadIdx.x; ch < C; ch += WARPS * 32) {
        float acc = bias ? bl_load_any(bias, bias_dtype, ch) : 0.f;
        for (int i = 0; i < n_taps; ++i) {
            const int off = j - (n_taps - 1) + i;
            const float xv = off >= 0 ? x[(size_t)(t - j + off) * ld + ch] : tl[(size_t)(n_taps - 1 + off) * C + ch];
            acc = fmaf(taps[(size_t)ch * n_taps + i], xv, acc);
        }
        y[(size_t)t * C + ch] = bl_silu(acc);
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    for (int hh = threadIdx.x >> 5; hh < unit_heads; hh += WARPS) {
        float* p = y + (size_t)t * C + (size_t)hh * dk;
        float ss = 0.f;
        for (int d = lane; d < dk; d += 32) ss += p[d] * p[d];
        const float inv = (hh < scaled_heads ? q_scale : 1.f) / sqrtf(bl_warp_sum(ss) + unit_eps);
        for (int d = lane; d < dk; d += 32) p[d] *= inv;
    }
}

// The same for four taps, channels in groups of four with 16-byte accesses: the unit heads' values stay in shared memory
// between the convolution and the norm (the kernel above writes, reads and writes them again, and reads each tap of a
// channel by itself). Sums in the order of the kernel above. Bound by trips to L2 for few tokens (8 of 4,096 channels
// 21 -> 5.2 us) and by the rows' bytes for many (2,048 of 1,792 channels 30 -> 19 us; for that many
// tokens see the kernel behind this one).
constexpr int CONV4_THREADS = 256;
__global__ void __launch_bounds__(CONV4_THREADS)
conv4_silu_unit_kernel(const float* x, int ld, const float4* __restrict__ taps, const float* tail, size_t slot_stride,
                       const int* __restrict__ slots, const int* __restrict__ tok_req, const int* __restrict__ cu_q, float* y,
                       int C, int unit_heads, int scaled_heads, int dk, float q_scale, float unit_eps, const void* __restrict__ bias,
                       int bias_dtype) {
    bl_pdl_trigger();
    bl_pdl_wait();
    extern __shared__ __align__(16) float units[];               // [unit_heads * dk]
    const int lane = threadIdx.x & 31, unit_cols = unit_heads * dk;
    const int t = blockIdx.x;
    const int r = tok_req[t];
    const int j = t - cu_q[r];
    const float* tl = tail + (size_t)slots[r] * slot_stride;
    for (int ch = threadIdx.x * 4; ch < C; ch += CONV4_THREADS * 4) {
        float4 in[4], tp[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int off = j - 3 + i;
            in[i] = *reinterpret_cast<const float4*>(off >= 0 ? x + (size_t)(t - j + off) * ld + ch : tl + (size_t)(3 + off) * C + ch);
            tp[i] = taps[ch + i];                            // the four taps of channel ch + i
        }
        float acc[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            float a = bias ? bl_load_any(bias, bias_dtype, ch + e) : 0.f;
            a = fmaf(tp[e].x, reinterpret_cast<const float*>(&in[0])[e], a);
            a = fmaf(tp[e].y, reinterpret_cast<const float*>(&in[1])[e], a);
            a = fmaf(tp[e].z, reinterpret_cast<const float*>(&in[2])[e], a);
            a = fmaf(tp[e].w, reinterpret_cast<const float*>(&in[3])[e], a);
            acc[e] = bl_silu(a);
        }
        *reinterpret_cast<float4*>(ch < unit_cols ? units + ch : y + (size_t)t * C + ch) = make_float4(acc[0], acc[1], acc[2], acc[3]);
    }
    __syncthreads();
    for (int hh = threadIdx.x >> 5; hh < unit_heads; hh += CONV4_THREADS / 32) {
        const float* p = units + (size_t)hh * dk;
        float ss = 0.f;
        for (int d = lane; d < dk; d += 32) ss += p[d] * p[d];
        const float inv = (hh < scaled_heads ? q_scale : 1.f) / sqrtf(bl_warp_sum(ss) + unit_eps);
        for (int d = lane; d < dk; d += 32) y[(size_t)t * C + (size_t)hh * dk + d] = p[d] * inv;
    }
}

// The same for many tokens: a block takes CONV_RUN neighbouring tokens, and a thread goes down them with its channels' taps and
// last inputs in registers. One token a block reads every input four times and the taps (16 bytes a channel, as much as four inputs)
// once a token, all through L2, which is what it waits for (1,840 tokens of 4,096 channels 39 us, of which 9 are bytes; 2,048 of
// 1,792 24 us). A request's first tokens fetch the inputs before them from its tail.
constexpr int CONV_RUN = 4;
__global__ void __launch_bounds__(CONV4_THREADS)
conv4_silu_unit_run_kernel(const float* x, int ld, const float4* __restrict__ taps, const float* tail, size_t slot_stride,
                           const int* __restrict__ slots, const int* __restrict__ tok_req, const int* __restrict__ cu_q, float* y,
                           int T, int C, int unit_heads, int scaled_heads, int dk, float q_scale, float unit_eps, const void* __restrict__ bias,
                           int bias_dtype) {
    bl_pdl_trigger();
    extern __shared__ __align__(16) float units[];               // [CONV_RUN][unit_heads * dk]
    const int lane = threadIdx.x & 31, unit_cols = unit_heads * dk;
    const int t0 = blockIdx.x * CONV_RUN, n = min(CONV_RUN, T - t0);
    int place[CONV_RUN];                                         // a token's place in its request
    const float* tl[CONV_RUN];
#pragma unroll
    for (int u = 0; u < CONV_RUN; ++u) {
        const int r = tok_req[t0 + min(u, n - 1)];
        place[u] = t0 + u - cu_q[r];
        tl[u] = tail + (size_t)slots[r] * slot_stride;
    }
    bl_pdl_wait();
    for (int ch = threadIdx.x * 4; ch < C; ch += CONV4_THREADS * 4) {
        float4 tp[4], in[CONV_RUN + 3];                          // in[u + i]: input i of the four that token u sums
        float b[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) tp[i] = taps[ch + i];        // the four taps of channel ch + i
#pragma unroll
        for (int i = 0; i < 3; ++i) {                            // before the first token
            const int off = place[0] - 3 + i;
            in[i] = *reinterpret_cast<const float4*>(off >= 0 ? x + ((ptrdiff_t)t0 - 3 + i) * ld + ch : tl[0] + (size_t)(3 + off) * C + ch);
        }
#pragma unroll
        for (int u = 0; u < CONV_RUN; ++u)
            if (u < n) in[u + 3] = *reinterpret_cast<const float4*>(x + (size_t)(t0 + u) * ld + ch);
#pragma unroll
        for (int e = 0; e < 4; ++e) b[e] = bias ? bl_load_any(bias, bias_dtype, ch + e) : 0.f;
#pragma unroll
        for (int u = 0; u < CONV_RUN; ++u) {
            if (u >= n) continue;
            float4 q[3] = {in[u], in[u + 1], in[u + 2]};
            if (u > 0 && place[u] < 3 && place[u] <= u) {        // its request begins in this block: what precedes its first token is in the tail
#pragma unroll
                for (int i = 0; i < 3; ++i)
                    if (place[u] - 3 + i < 0) q[i] = *reinterpret_cast<const float4*>(tl[u] + (size_t)(place[u] + i) * C + ch);
            }
            float acc[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                float a = b[e];
                a = fmaf(tp[e].x, reinterpret_cast<const float*>(&q[0])[e], a);
                a = fmaf(tp[e].y, reinterpret_cast<const float*>(&q[1])[e], a);
                a = fmaf(tp[e].z, reinterpret_cast<const float*>(&q[2])[e], a);
                a = fmaf(tp[e].w, reinterpret_cast<const float*>(&in[u + 3])[e], a);
                acc[e] = bl_silu(a);
            }
            *reinterpret_cast<float4*>(ch < unit_cols ? units + (size_t)u * unit_cols + ch : y + (size_t)(t0 + u) * C + ch) = make_float4(acc[0], acc[1], acc[2], acc[3]);
        }
    }
    __syncthreads();
    for (int item = threadIdx.x >> 5; item < n * unit_heads; item += CONV4_THREADS / 32) {
        const int u = item / unit_heads, hh = item % unit_heads;
        const float* p = units + (size_t)u * unit_cols + (size_t)hh * dk;
        float ss = 0.f;
        for (int d = lane; d < dk; d += 32) ss += p[d] * p[d];
        const float inv = (hh < scaled_heads ? q_scale : 1.f) / sqrtf(bl_warp_sum(ss) + unit_eps);
        for (int d = lane; d < dk; d += 32) y[(size_t)(t0 + u) * C + (size_t)hh * dk + d] = p[d] * inv;
    }
}

// After the step's convolutions have read the tail: the last n_taps - 1 inputs of each request with tokens.
__global__ void conv_tail_update_kernel(const float* x, int ld, int n_taps, float* tail, size_t slot_stride,
                                        const int* __restrict__ slots, const int* __restrict__ cu_q, int C) {
    bl_pdl_trigger();
    bl_pdl_wait();
    const int r = blockIdx.y;
    const int ch = blockIdx.x * blockDim.x + threadIdx.x;
    const int t0 = cu_q[r], n = cu_q[r + 1] - t0;
    if (n <= 0 || ch >= C) return;
    float* tl = tail + (size_t)slots[r] * slot_stride;
    float keep[MAX_TAPS];
#pragma unroll
    for (int i = 0; i < MAX_TAPS; ++i) {
        if (i < n_taps - 1) {
            const int off = n - (n_taps - 1) + i;
            keep[i] = off >= 0 ? x[(size_t)(t0 + off) * ld + ch] : tl[(size_t)(n_taps - 1 + off) * C + ch];
        }
    }
#pragma unroll
    for (int i = 0; i < MAX_TAPS; ++i)
        if (i < n_taps - 1) tl[(size_t)i * C + ch] = keep[i];
}


// In front of a recurrence with a FIXED decay per head (retention): q and k of every head rotated by the token's position
// (the first 2 * rot_half values of a head in pairs (i, i + rot_half), angle = float(position) * inv_freq[i], all 32-bit),
// k times k_scale after the rotation, and the head's decay written for each of its key channels (what the scan reads).
// One block per token.
__global__ void __launch_bounds__(WARPS * 32)
rope_decay_prep_kernel(const float* proj, int ld, int off_k, const int* __restrict__ positions, const float* __restrict__ inv_freq,
                       int rot_half, const float* __restrict__ head_decay, float k_scale, float* q_out, float* k_out,
                       float* decay_out, int H, int dk) {
    bl_pdl_trigger();
    bl_pdl_wait();
    const int t = blockIdx.x;
    const float pos = (float)positions[t];
    const float* src = proj + (size_t)t * ld;
    const size_t row = (size_t)t * H * dk;
    for (int e = threadIdx.x; e < H * dk; e += WARPS * 32) {
        const int h = e / dk, d = e % dk;
        float qv = src[e], kv = src[off_k + e];
        if (d < 2 * rot_half) {
            const int i = d < rot_half ? d : d - rot_half;
            float sn, cs;
            sincosf(pos * inv_freq[i], &sn, &cs);
            const int other = d < rot_half ? e + rot_half : e - rot_half;
            const float qo = src[other], ko = src[off_k + other];
            if (d < rot_half) { qv = qv * cs - qo * sn; kv = kv * cs - ko * sn; }
            else { qv = qv * cs + qo * sn; kv = kv * cs + ko * sn; }
        }
        q_out[row + e] = qv;
        k_out[row + e] = kv * k_scale;
        decay_out[row + e] = head_decay[h];
    }
}

// In front of a selective state-space recurrence (one decay per head and token): dt = softplus(raw + dt_bias[h]);
// decay[t, h, :] = exp(-exp(A_log[h]) * dt) for each of the n_state key channels; v[t, h, :] = dt * x[t, h, :].
// raw: 32-bit rows [T, >= H]; x: [T, H * dv] (the convolved inputs). neg_rate[h] = exp(A_log[h]), made at load. One block per token.
__global__ void __launch_bounds__(WARPS * 32)
ssd_prep_kernel(const float* raw, int ld_raw, const void* __restrict__ dt_bias, int bias_dtype, const float* __restrict__ rate,
                const float* x, int ld_x, float* decay_out, float* v_out, int H, int n_state, int dv) {
    bl_pdl_trigger();
    bl_pdl_wait();
    __shared__ float dts[256];
    const int t = blockIdx.x;
    for (int h0 = 0; h0 < H; h0 += 256) {
        const int hn = min(256, H - h0);
        __syncthreads();
        for (int h = threadIdx.x; h < hn; h += WARPS * 32) {
            const float zz = raw[(size_t)t * ld_raw + h0 + h] + bl_load_any(dt_bias, bias_dtype, h0 + h);
            dts[h] = zz > 20.f ? zz : log1pf(expf(zz));
        }
        __syncthreads();
        for (int e = threadIdx.x; e < hn * n_state; e += WARPS * 32) {
            const int h = e / n_state;
            decay_out[((size_t)t * H + h0) * n_state + e] = expf(-rate[h0 + h] * dts[h]);
        }
        for (int e = threadIdx.x; e < hn * dv; e += WARPS * 32) {
            const int h = e / dv;
            v_out[((size_t)t * H + h0) * dv + e] = dts[h] * x[(size_t)t * ld_x + (size_t)h0 * dv + e];
        }
    }
}

// Behind such a recurrence: u = (o + skip[h] * x) * silu(z) (the gate comes BEFORE the norm), then an RMS norm over each of
// n_parts equal parts of the row (each part by its own root mean square), times w. One block per (token, part); a part may
// span several heads or a fraction of one. skip and x may be null (no skip term), z may be null (no gate). A thread keeps
// up to GN_KEEP of its values between the two passes (parts of up to GN_KEEP * 128 values are read once); the sum of squares
// is added in a fixed order (lanes, then warps).
constexpr int GN_KEEP = 16;
template <typename TY>
__global__ void __launch_bounds__(WARPS * 32)
gated_group_norm_kernel(const float* o, const float* x, int ld_x, const void* __restrict__ skip, int skip_dtype, int dv,
                        const float* z, int ld_z, const void* __restrict__ w, int w_dtype, TY* __restrict__ y, int n_parts,
                        int width, float eps) {
    bl_pdl_trigger();
    bl_pdl_wait();
    __shared__ float warp_ss[WARPS];
    const int t = blockIdx.x / n_parts, part = blockIdx.x % n_parts;
    const int per = width / n_parts, c0 = part * per;
    auto value = [&](int c) {
        float u = o[(size_t)t * width + c];
        if (x) u = fmaf(bl_load_any(skip, skip_dtype, c / dv), x[(size_t)t * ld_x + c], u);
        if (z) u *= bl_silu(z[(size_t)t * ld_z + c]);
        return u;
    };
    float keep[GN_KEEP];
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < GN_KEEP; ++j) {
        const int i = threadIdx.x + j * WARPS * 32;
        keep[j] = i < per ? value(c0 + i) : 0.f;
        ss += keep[j] * keep[j];
    }
    for (int i = threadIdx.x + GN_KEEP * WARPS * 32; i < per; i += WARPS * 32) { const float u = value(c0 + i); ss += u * u; }
    ss = bl_warp_sum(ss);
    if ((threadIdx.x & 31) == 0) warp_ss[threadIdx.x >> 5] = ss;
    __syncthreads();
    float total = 0.f;
#pragma unroll
    for (int k = 0; k < WARPS; ++k) total += warp_ss[k];
    const float inv = 1.0f / sqrtf(total / (float)per + eps);
#pragma unroll
    for (int j = 0; j < GN_KEEP; ++j) {
        const int i = threadIdx.x + j * WARPS * 32;
        if (i < per) bl_store(y + (size_t)t * width + c0 + i, keep[j] * inv * (w ? bl_load_any(w, w_dtype, c0 + i) : 1.f));
    }
    for (int i = threadIdx.x + GN_KEEP * WARPS * 32; i < per; i += WARPS * 32)
        bl_store(y + (size_t)t * width + c0 + i, value(c0 + i) * inv * (w ? bl_load_any(w, w_dtype, c0 + i) : 1.f));
}

}  // namespace

extern "C" int bl_recurrent_scan(int rule, const float* q, int ldq, const float* k, int ldk, const float* v, int ldv,
                                 const float* z, int ldz, const float* beta, int ldb, float q_scale, float* state, long long slot_stride, const int* slots, const int* cu_q, int R,
                                 float* out, int H, int G, int dk, int dv, void* stream) {
    return bl_recurrent_scan_parts(rule, q, ldq, k, ldk, v, ldv, z, ldz, beta, ldb, q_scale, state, slot_stride, slots, cu_q, R, out,
                                   H, G, dk, dv, 1, 0, R, nullptr, stream);
}

// Whether bl_recurrent_scan_parts can cut long portions of this rule and key size (else it runs them in one piece):
// 0, or the blocks that each part of one request's portion runs on in the first pass, H * ceil(columns / columns a
// block) (the delta rule's first pass has dk columns more, and its fold takes key sizes up to 128).
extern "C" int bl_recurrent_scan_can_split(int rule, int H, int dk, int dv) {
    if (rule != BL_RULE_GLA && rule != BL_RULE_DELTA && rule != BL_RULE_BONUS) return 0;
    if (rule == BL_RULE_DELTA && dk > FOLD_MAX_DK) return 0;
    for (int ks = 1; ks <= 32; ks *= 2)
        if (dk % (4 * ks) == 0 && dk / ks <= SCAN_VEC_ROWS) {
            const int cols_blk = WARPS * (32 / ks), cols = dv + (rule == BL_RULE_DELTA ? dk : 0);
            return H * ((cols + cols_blk - 1) / cols_blk);
        }
    return 0;
}

// Floats of scratch that bl_recurrent_scan_parts needs to cut n_cut of a step's R requests.
extern "C" long long bl_recurrent_scan_parts_scratch(int rule, int R, int n_cut, int nc, int H, int dk, int dv) {
    const long long per = rule == BL_RULE_DELTA ? (long long)dk * (2 * dv + dk) : (long long)dk * (dv + 1);
    return (R + 3) / 4 * 4 + (long long)n_cut * nc * H * per;
}

extern "C" int bl_recurrent_scan_parts(int rule, const float* q, int ldq, const float* k, int ldk, const float* v, int ldv,
                                       const float* z, int ldz, const float* beta, int ldb, float q_scale, float* state,
                                       long long slot_stride, const int* slots, const int* cu_q, int R, float* out, int H, int G,
                                       int dk, int dv, int nc, int n_cut, int busy, float* scratch, void* stream) {
    if (R <= 0) return 0;
    if (nc < 1 || (nc > 1 && (n_cut < 1 || n_cut > R || scratch == nullptr || !bl_recurrent_scan_can_split(rule, H, dk, dv) || (long long)R * nc > 65535)))
        BL_FAIL("bl_recurrent_scan_parts: %d parts for rule %d, %d key channels, %d requests", nc, rule, dk, R);
    if (H <= 0 || G <= 0 || H % G != 0 || dk <= 0 || dv <= 0) BL_FAIL("bl_recurrent_scan: bad sizes H=%d G=%d dk=%d dv=%d", H, G, dk, dv);
    if (dk > RKMAX * 32) BL_FAIL("bl_recurrent_scan: %d key channels, at most %d", dk, RKMAX * 32);
    if (R > 65535 || H > 65535) BL_FAIL("bl_recurrent_scan: %d requests or %d heads are too many for one launch", R, H);
    if ((rule == BL_RULE_DELTA || rule == BL_RULE_BONUS) && beta == nullptr) BL_FAIL("bl_recurrent_scan: rule %d needs beta", rule);
    int KS = 1;
    while ((dk + KS - 1) / KS > RKMAX) KS *= 2;
    // The kernel with 16-byte fetches where the key size splits evenly over the lanes. Sixteen rows a lane: eight, with a
    // butterfly of one more step, were measured and are no faster for one request (64 x 128 heads, 2,048 tokens: 534 us
    // against 570) and slower where it counts, 128 x 256 heads (752 against 678) and decode steps of 64 requests (115 us
    // against 67): a token's time is its chain of dependent instructions, not its arithmetic.
    int rk4 = 0;
    for (int ks = 1; ks <= 32 && rk4 == 0; ks *= 2)
        if (dk % (4 * ks) == 0 && dk / ks <= SCAN_VEC_ROWS) { KS = ks; rk4 = dk / (4 * ks); }
    if (rk4 == 0 && dk % (4 * KS) == 0) rk4 = dk / (4 * KS);
    const int CW = 32 / KS;
    struct Walk { int cols_blk, chunk; size_t smem; };
    auto walk_of = [&](int columns) {                  // of lanes with so many columns
        Walk k;
        k.cols_blk = WARPS * CW * columns;
        const size_t per_token = (size_t)(3 * dk + k.cols_blk + 4) * sizeof(float);
        k.chunk = (int)(SCAN_SMEM_BYTES / (2 * per_token));
        k.chunk = k.chunk < 1 ? 1 : (k.chunk > 16 ? 16 : k.chunk);
        k.smem = 2 * per_token * k.chunk;
        return k;
    };
    const Walk one = walk_of(1), four = walk_of(4);
    const int cols_blk = one.cols_blk, chunk = one.chunk;
    const size_t smem = one.smem;
    if (smem > 48 * 1024) BL_FAIL("bl_recurrent_scan: %d key channels need %zu bytes of shared memory a token", dk, smem / (2 * chunk));
    // 16-byte copies where every row of q, k and z starts on a 16-byte boundary
    const int vec = dk % 4 == 0 && ldq % 4 == 0 && ldk % 4 == 0 && ldz % 4 == 0 &&
                    (((uintptr_t)q | (uintptr_t)k | (uintptr_t)z) & 15) == 0;
    dim3 grid((dv + cols_blk - 1) / cols_blk, H, R * nc);
    // four columns a lane: where values, states and the parts' states between the passes are whole 16-byte pieces, too
    const bool fours = rk4 == 4 && vec && dv % 4 == 0 && ldv % 4 == 0 && slot_stride % 4 == 0 &&
                       (((uintptr_t)v | (uintptr_t)state | (uintptr_t)scratch) & 15) == 0 && four.smem <= 48 * 1024;
    cudaStream_t s = (cudaStream_t)stream;
    if (rule != BL_RULE_GLA && rule != BL_RULE_DELTA && rule != BL_RULE_BONUS) BL_FAIL("bl_recurrent_scan: unknown rule %d", rule);
    if (rk4 > 0) {                                     // a lane's rows are whole groups of four
        const bool dl = rule == BL_RULE_DELTA;
        if (dl && nc > 1 && ((uintptr_t)scratch & 15)) BL_FAIL("bl_recurrent_scan_parts: the delta rule's scratch must be 16-byte aligned (its folds read the transitions in such pieces)");
        int* places = n_cut < R ? reinterpret_cast<int*>(scratch) : nullptr;     // [R], up to a multiple of 16 bytes; null: r is r's place
        float* part_s = scratch ? scratch + (R + 3) / 4 * 4 : nullptr;           // [n_cut, nc, H, dk, dv]
        float* part_p = scratch ? part_s + (size_t)n_cut * nc * H * dk * dv : nullptr;   // [n_cut, nc, H, dk] or, delta rule, [n_cut, nc, H, dk, dk]
        // [n_cut, nc, H, dk, dv]; a fold with a decay per row leaves the starts in part_s
        float* part_start = scratch == nullptr ? nullptr : dl ? part_p + (size_t)n_cut * nc * H * dk * dk : part_s;
        // Two an SM, or the build for four: by the blocks that work side by side for most of the launch, not by those of a few
        // tokens beside a long portion that leave at once (2,000 tokens beside 31 running requests, in one piece: 7 heads of
        // 64 x 128 640 us counted by all, 507 so; 8 of 128 x 256 1,115 and 824; the delta rule 778 and 613, 1,215 and 934).
        const int two_an_sm = 2 * bl_device_sms();
        // Four columns a lane from four blocks of one column an SM on, when a second round of those would begin: 8 single tokens of 8
        // heads of 128 x 256 9.4 -> 6.3 us, 64 of them 56 -> 23; prompts of 401 to 57 tokens 249 -> 177 (delta rule 315 -> 238); 2,048
        // tokens in 32 parts of 7 heads of 64 x 128 103 -> 78. Below, a fourth of the blocks is too few: 8 single tokens of 7 heads of
        // 64 x 128 3.3 us against 4.1, 8 x 250 tokens 79 against 97.
        const long long fours_from = 4LL * bl_device_sms();
        const long long at_once[2] = {(long long)n_cut * nc, nc > 1 ? (long long)n_cut * nc + (busy > n_cut ? busy - n_cut : 0) : busy};
#define BL_SCAN_Q(D, R4, NC, KSC, DENSE, QUIET, CUT, GRID) BL_CUDA(bl_launch_dependent(recurrent_scan_vec_kernel<D, R4, NC, KSC, DENSE, QUIET, CUT>, GRID, \
        dim3(WARPS * 32), NC == 4 ? four.smem : smem, s, q, ldq, k, ldk, v, ldv, z, ldz, beta, ldb, q_scale, state, (size_t)slot_stride, slots, cu_q, out, H, G, \
        dk, dv, KS, NC == 4 ? four.chunk : chunk, vec, nc, n_cut, places, part_s, part_p, (const float*)part_start))
#define BL_SCAN_4(D, KSC, PASS, GRID) do { if (PASS == 1) BL_SCAN_Q(D, 4, 4, KSC, true, true, true, GRID); else BL_SCAN_Q(D, 4, 4, KSC, true, false, true, GRID); } while (0)
#define BL_SCAN(D, R4, PASS) do { \
        const int cols = D == BL_RULE_DELTA && PASS == 1 ? dv + dk : dv;         /* the delta rule's first pass makes its transition in dk more */ \
        const dim3 g((cols + cols_blk - 1) / cols_blk, H, R * nc), g4((cols + four.cols_blk - 1) / four.cols_blk, H, R * nc); \
        const long long blocks = at_once[PASS - 1] * g.x * g.y; \
        const bool dense = blocks > two_an_sm; \
        if (fours && blocks >= fours_from) { \
            if (KS == 4) BL_SCAN_4(D, 4, PASS, g4); else if (KS == 8) BL_SCAN_4(D, 8, PASS, g4); else BL_SCAN_4(D, 0, PASS, g4); } \
        else if (PASS == 1) { if (dense) BL_SCAN_Q(D, R4, 1, 0, true, true, true, g); else BL_SCAN_Q(D, R4, 1, 0, false, true, true, g); } \
        else if (dense) BL_SCAN_Q(D, R4, 1, 0, true, false, true, g); \
        else if (nc > 1) BL_SCAN_Q(D, R4, 1, 0, false, false, true, g); else BL_SCAN_Q(D, R4, 1, 0, false, false, false, g); } while (0)
        for (int pass = (nc > 1 ? 1 : 2); pass <= 2; ++pass) {
            if (pass == 2 && nc > 1 && dl && dv % 4 == 0 && slot_stride % 4 == 0 && (((uintptr_t)state | (uintptr_t)scratch) & 15) == 0) {
                // rows of up to 64 values a thread; 8 columns a block where P is large (every block of a head reads all of it)
                const bool wide = dk > 64;
                const dim3 g((dv + (wide ? 8 : 4) - 1) / (wide ? 8 : 4), H, R);
                if (wide) BL_CUDA(bl_launch_dependent(scan_fold_matrix4_kernel<2, 2>, g, dim3(2 * dk), 0, s, state, (size_t)slot_stride, slots, cu_q,
                                                      (const int*)places, (const float*)part_s, (const float*)part_p, part_start, H, dk, dv, nc));
                else BL_CUDA(bl_launch_dependent(scan_fold_matrix4_kernel<1, 1>, g, dim3(dk), 0, s, state, (size_t)slot_stride, slots, cu_q,
                                                 (const int*)places, (const float*)part_s, (const float*)part_p, part_start, H, dk, dv, nc));
            } else if (pass == 2 && nc > 1 && dl)
                BL_CUDA(bl_launch_dependent(scan_fold_matrix_kernel, dim3((dv + FOLD_COLS - 1) / FOLD_COLS, H, R), dim3(256), 0, s, state,
                                            (size_t)slot_stride, slots, cu_q, (const int*)places, (const float*)part_s, (const float*)part_p, part_start,
                                            H, dk, dv, nc));
            if (pass == 2 && nc > 1 && !dl)
                BL_CUDA(bl_launch_dependent(scan_fold_kernel, dim3((dk * dv + 255) / 256, H, R), dim3(256), 0, s, state, (size_t)slot_stride,
                                            slots, cu_q, (const int*)places, part_s, (const float*)part_p, H, dk, dv, nc));
            switch (rk4) {
#define BL_SCAN_RULE(R4) do { if (dl) BL_SCAN(BL_RULE_DELTA, R4, pass); else if (rule == BL_RULE_BONUS) BL_SCAN(BL_RULE_BONUS, R4, pass); \
                                  else BL_SCAN(BL_RULE_GLA, R4, pass); } while (0)
                case 1: BL_SCAN_RULE(1); break;
                case 2: BL_SCAN_RULE(2); break;
                case 3: BL_SCAN_RULE(3); break;
                default: BL_SCAN_RULE(4); break;
#undef BL_SCAN_RULE
            }
        }
#undef BL_SCAN
#undef BL_SCAN_4
#undef BL_SCAN_Q
        BL_CHECK_LAUNCH("bl_recurrent_scan");
        return 0;
    }
    if (nc > 1) BL_FAIL("bl_recurrent_scan_parts: %d key channels cannot be cut into parts", dk);
    if (rule == BL_RULE_GLA)
        BL_CUDA(bl_launch_dependent(recurrent_scan_kernel<BL_RULE_GLA>, grid, dim3(WARPS * 32), smem, s, q, ldq, k, ldk, v, ldv, z, ldz, beta, ldb, q_scale,
            state, (size_t)slot_stride, slots, cu_q, out, H, G, dk, dv, KS, chunk, vec));
    else if (rule == BL_RULE_DELTA)
        BL_CUDA(bl_launch_dependent(recurrent_scan_kernel<BL_RULE_DELTA>, grid, dim3(WARPS * 32), smem, s, q, ldq, k, ldk, v, ldv, z, ldz, beta, ldb, q_scale,
            state, (size_t)slot_stride, slots, cu_q, out, H, G, dk, dv, KS, chunk, vec));
    else
        BL_CUDA(bl_launch_dependent(recurrent_scan_kernel<BL_RULE_BONUS>, grid, dim3(WARPS * 32), smem, s, q, ldq, k, ldk, v, ldv, z, ldz, beta, ldb, q_scale,
            state, (size_t)slot_stride, slots, cu_q, out, H, G, dk, dv, KS, chunk, vec));
    BL_CHECK_LAUNCH("bl_recurrent_scan");
    return 0;
}

extern "C" int bl_head_norm_gate(const float* o, const void* w, int w_dtype, const float* gate, int ld_gate, int gate_kind,
                                 void* y, int y_dtype, int T, int H, int dv, float eps, void* stream) {
    return bl_head_norm_gate_ext(o, dv, w, w_dtype, 0, nullptr, gate, ld_gate, gate_kind, y, y_dtype, T, H, dv, eps, stream);
}

extern "C" int bl_head_norm_gate_ext(const float* o, int o_head_stride, const void* w, int w_dtype, int w_per_head, const float* floor,
                                     const float* gate, int ld_gate, int gate_kind, void* y, int y_dtype, int T, int H, int dv, float eps,
                                     void* stream) {
    if (T <= 0) return 0;
    if (H <= 0 || dv <= 0 || (gate && ld_gate < H * dv) || o_head_stride < dv + (floor ? 1 : 0))
        BL_FAIL("bl_head_norm_gate: bad sizes H=%d dv=%d gate stride %d head stride %d", H, dv, ld_gate, o_head_stride);
    if (gate && gate_kind != BL_GATE_SIGMOID && gate_kind != BL_GATE_SILU) BL_FAIL("bl_head_norm_gate: unknown gate %d", gate_kind);
    const int items = T * H, blocks = (items + WARPS - 1) / WARPS;
    cudaStream_t s = (cudaStream_t)stream;
    if (floor == nullptr && dv % 4 == 0 && dv <= 512 && o_head_stride % 4 == 0 && (gate == nullptr || ld_gate % 4 == 0) &&
        (((uintptr_t)o | (uintptr_t)gate) & 15) == 0 && ((uintptr_t)y & (y_dtype == BL_F32 ? 15 : 7)) == 0 && (y_dtype == BL_F32 || y_dtype == BL_BF16)) {
#define BL_HEADS4(TY, NV) BL_CUDA(bl_launch_dependent(head_norm_gate4_kernel<TY, NV>, dim3(blocks), dim3(WARPS * 32), 0, s, o, o_head_stride, w, w_dtype, \
        w_per_head, gate, ld_gate, gate_kind, (TY*)y, items, H, dv, eps))
#define BL_HEADS4_NV(TY) do { if (dv <= 128) BL_HEADS4(TY, 1); else if (dv <= 256) BL_HEADS4(TY, 2); else BL_HEADS4(TY, 4); } while (0)
        if (y_dtype == BL_F32) BL_HEADS4_NV(float); else BL_HEADS4_NV(__nv_bfloat16);
#undef BL_HEADS4_NV
#undef BL_HEADS4
        BL_CHECK_LAUNCH("bl_head_norm_gate");
        return 0;
    }
    if (y_dtype == BL_F32)
        BL_CUDA(bl_launch_dependent(head_norm_gate_kernel<float>, dim3(blocks), dim3(WARPS * 32), 0, s, o, o_head_stride, w, w_dtype, w_per_head,
                                    floor, gate, ld_gate, gate_kind, (float*)y, items, H, dv, eps));
    else if (y_dtype == BL_BF16)
        BL_CUDA(bl_launch_dependent(head_norm_gate_kernel<__nv_bfloat16>, dim3(blocks), dim3(WARPS * 32), 0, s, o, o_head_stride, w, w_dtype,
                                    w_per_head, floor, gate, ld_gate, gate_kind, (__nv_bfloat16*)y, items, H, dv, eps));
    else
        BL_FAIL("bl_head_norm_gate: unknown output dtype %d", y_dtype);
    BL_CHECK_LAUNCH("bl_head_norm_gate");
    return 0;
}

extern "C" int bl_memory_gates(const float* proj, int ld, int off_k, int off_v, int off_i, int off_f, const void* bias_i, int bi_dtype,
                               const void* bias_f, int bf_dtype, float cap, float* state, long long slot_stride, long long off_m,
                               const int* slots, const int* cu_q, int R, int T, float* gates, float* decay, float* k_out, float* v_out,
                               int H, int dk, int dv, void* stream) {
    if (R <= 0 || T <= 0) return 0;
    if (H <= 0 || dk <= 0 || dv <= 0 || !(cap > 0.f)) BL_FAIL("bl_memory_gates: bad sizes H=%d dk=%d dv=%d cap=%g", H, dk, dv, cap);
    if (R > 65535) BL_FAIL("bl_memory_gates: %d requests are too many for one launch", R);
    if (off_k + H * dk > ld || off_v + H * dv > ld || off_i + H > ld || off_f + H > ld) BL_FAIL("bl_memory_gates: columns do not fit rows of %d", ld);
    cudaStream_t s = (cudaStream_t)stream;
    BL_CUDA(bl_launch_dependent(memory_gate_chain_kernel, dim3(H, R), dim3(32), 0, s, proj, ld, off_i, off_f, bias_i, bi_dtype, bias_f, bf_dtype,
                                cap, state, (size_t)slot_stride, (size_t)off_m, slots, cu_q, gates, T, H));
    BL_CUDA(bl_launch_dependent(memory_expand_kernel, dim3(T), dim3(WARPS * 32), 0, s, proj, ld, off_k, off_v, (const float*)gates, decay, k_out,
                                v_out, T, H, dk, dv));
    BL_CHECK_LAUNCH("bl_memory_gates");
    return 0;
}

extern "C" int bl_shift_mix(const float* x, int ld, const float* mu, int n_mix, const float* prev, long long slot_stride,
                            const int* slots, const int* tok_req, const int* cu_q, void* out, int out_dtype, int T, int d, void* stream) {
    if (T <= 0) return 0;
    if (d <= 0 || ld < d || n_mix < 1) BL_FAIL("bl_shift_mix: bad sizes d=%d ld=%d mixes=%d", d, ld, n_mix);
    cudaStream_t s = (cudaStream_t)stream;
    const int vec = d % 4 == 0 && ld % 4 == 0 && slot_stride % 4 == 0 &&
                    (((uintptr_t)x | (uintptr_t)mu | (uintptr_t)prev | (uintptr_t)out) & 15) == 0;
    if (out_dtype == BL_F32)
        BL_CUDA(bl_launch_dependent(shift_mix_kernel<float>, dim3(T), dim3(WARPS * 32), 0, s, x, ld, mu, n_mix, prev,
                                    (size_t)slot_stride, slots, tok_req, cu_q, (float*)out, T, d, vec));
    else if (out_dtype == BL_BF16)
        BL_CUDA(bl_launch_dependent(shift_mix_kernel<__nv_bfloat16>, dim3(T), dim3(WARPS * 32), 0, s, x, ld, mu, n_mix, prev,
                                    (size_t)slot_stride, slots, tok_req, cu_q, (__nv_bfloat16*)out, T, d, vec));
    else
        BL_FAIL("bl_shift_mix: unknown output dtype %d", out_dtype);
    BL_CHECK_LAUNCH("bl_shift_mix");
    return 0;
}

extern "C" int bl_bonus_dot(const float* q, int ldq, const float* k, int ldk, const void* u, int u_dtype, float* out, int T, int H,
                            int dk, void* stream) {
    if (T <= 0) return 0;
    if (H <= 0 || dk <= 0 || ldq < H * dk || ldk < H * dk) BL_FAIL("bl_bonus_dot: bad sizes H=%d dk=%d", H, dk);
    const int items = T * H;
    BL_CUDA(bl_launch_dependent(bonus_dot_kernel, dim3((items + WARPS - 1) / WARPS), dim3(WARPS * 32), 0, (cudaStream_t)stream, q, ldq, k, ldk,
                                u, u_dtype, out, items, H, dk));
    BL_CHECK_LAUNCH("bl_bonus_dot");
    return 0;
}

extern "C" int bl_conv_silu_unit(const float* x, int ld, const float* taps, int n_taps, const float* tail, long long slot_stride,
                                 const int* slots, const int* tok_req, const int* cu_q, float* y, int T, int C, int unit_heads,
                                 int scaled_heads, int dk, float q_scale, float unit_eps, void* stream) {
    return bl_conv_silu_unit_bias(x, ld, taps, n_taps, tail, slot_stride, slots, tok_req, cu_q, y, T, C, unit_heads, scaled_heads, dk,
                                  q_scale, unit_eps, nullptr, BL_F32, stream);
}

// The same with a bias per channel (null: none) that the convolution's sum starts from.
extern "C" int bl_conv_silu_unit_bias(const float* x, int ld, const float* taps, int n_taps, const float* tail, long long slot_stride,
                                      const int* slots, const int* tok_req, const int* cu_q, float* y, int T, int C, int unit_heads,
                                      int scaled_heads, int dk, float q_scale, float unit_eps, const void* bias, int bias_dtype,
                                      void* stream) {
    if (T <= 0) return 0;
    if (n_taps < 1 || n_taps > MAX_TAPS) BL_FAIL("bl_conv_silu_unit: %d taps, 1..%d are built", n_taps, MAX_TAPS);
    if (C <= 0 || ld < C || unit_heads * dk > C || scaled_heads > unit_heads)
        BL_FAIL("bl_conv_silu_unit: bad sizes C=%d ld=%d heads=%d of %d", C, ld, unit_heads, dk);
    const int unit_cols = unit_heads * dk;
    if (n_taps == 4 && C % 4 == 0 && ld % 4 == 0 && slot_stride % 4 == 0 && unit_cols % 4 == 0 && unit_cols <= 8192 &&
        (((uintptr_t)x | (uintptr_t)taps | (uintptr_t)tail | (uintptr_t)y) & 15) == 0) {
        // several tokens a block where the launch then still has a block for every SM, and their unit heads fit its 48 KB
        if (T >= CONV_RUN * bl_device_sms() && CONV_RUN * unit_cols * (int)sizeof(float) <= 48 * 1024) {
            BL_CUDA(bl_launch_dependent(conv4_silu_unit_run_kernel, dim3((T + CONV_RUN - 1) / CONV_RUN), dim3(CONV4_THREADS),
                                        (size_t)CONV_RUN * unit_cols * sizeof(float), (cudaStream_t)stream, x, ld, (const float4*)taps, tail,
                                        (size_t)slot_stride, slots, tok_req, cu_q, y, T, C, unit_heads, scaled_heads, dk, q_scale, unit_eps, bias, bias_dtype));
            BL_CHECK_LAUNCH("bl_conv_silu_unit");
            return 0;
        }
        BL_CUDA(bl_launch_dependent(conv4_silu_unit_kernel, dim3(T), dim3(CONV4_THREADS), (size_t)unit_cols * sizeof(float),
                                    (cudaStream_t)stream, x, ld, (const float4*)taps, tail, (size_t)slot_stride, slots, tok_req, cu_q, y, C,
                                    unit_heads, scaled_heads, dk, q_scale, unit_eps, bias, bias_dtype));
        BL_CHECK_LAUNCH("bl_conv_silu_unit");
        return 0;
    }
    BL_CUDA(bl_launch_dependent(conv_silu_unit_kernel, dim3(T), dim3(WARPS * 32), 0, (cudaStream_t)stream, x, ld, taps, n_taps, tail,
                                (size_t)slot_stride, slots, tok_req, cu_q, y, C, unit_heads, scaled_heads, dk, q_scale, unit_eps, bias, bias_dtype));
    BL_CHECK_LAUNCH("bl_conv_silu_unit");
    return 0;
}

extern "C" int bl_conv_tail_update(const float* x, int ld, int n_taps, float* tail, long long slot_stride, const int* slots,
                                   const int* cu_q, int R, int C, void* stream) {
    if (R <= 0 || n_taps <= 1) return 0;
    if (n_taps > MAX_TAPS) BL_FAIL("bl_conv_tail_update: %d taps, 1..%d are built", n_taps, MAX_TAPS);
    if (R > 65535) BL_FAIL("bl_conv_tail_update: %d requests are too many for one launch", R);
    dim3 grid((C + 127) / 128, R);
    BL_CUDA(bl_launch_dependent(conv_tail_update_kernel, grid, dim3(128), 0, (cudaStream_t)stream, x, ld, n_taps, tail,
                                (size_t)slot_stride, slots, cu_q, C));
    BL_CHECK_LAUNCH("bl_conv_tail_update");
    return 0;
}

extern "C" int bl_rope_decay_prep(const float* proj, int ld, int off_k, const int* positions, const float* inv_freq, int rot_half,
                                  const float* head_decay, float k_scale, float* q_out, float* k_out, float* decay_out, int T, int H,
                                  int dk, void* stream) {
    if (T <= 0) return 0;
    if (H <= 0 || dk <= 0 || rot_half < 0 || 2 * rot_half > dk || off_k < H * dk || ld < off_k + H * dk)
        BL_FAIL("bl_rope_decay_prep: bad sizes H=%d dk=%d rotated pairs=%d off_k=%d ld=%d", H, dk, rot_half, off_k, ld);
    BL_CUDA(bl_launch_dependent(rope_decay_prep_kernel, dim3(T), dim3(WARPS * 32), 0, (cudaStream_t)stream, proj, ld, off_k, positions,
                                inv_freq, rot_half, head_decay, k_scale, q_out, k_out, decay_out, H, dk));
    BL_CHECK_LAUNCH("bl_rope_decay_prep");
    return 0;
}

extern "C" int bl_ssd_prep(const float* raw, int ld_raw, const void* dt_bias, int bias_dtype, const float* rate, const float* x,
                           int ld_x, float* decay_out, float* v_out, int T, int H, int n_state, int dv, void* stream) {
    if (T <= 0) return 0;
    if (H <= 0 || n_state <= 0 || dv <= 0 || ld_raw < H || ld_x < H * dv)
        BL_FAIL("bl_ssd_prep: bad sizes H=%d state=%d dv=%d ld_raw=%d ld_x=%d", H, n_state, dv, ld_raw, ld_x);
    BL_CUDA(bl_launch_dependent(ssd_prep_kernel, dim3(T), dim3(WARPS * 32), 0, (cudaStream_t)stream, raw, ld_raw, dt_bias, bias_dtype,
                                rate, x, ld_x, decay_out, v_out, H, n_state, dv));
    BL_CHECK_LAUNCH("bl_ssd_prep");
    return 0;
}

extern "C" int bl_gated_group_norm(const float* o, const float* x, int ld_x, const void* skip, int skip_dtype, int dv, const float* z,
                                   int ld_z, const void* w, int w_dtype, void* y, int y_dtype, int T, int width, int n_parts, float eps,
                                   void* stream) {
    if (T <= 0) return 0;
    if (width <= 0 || n_parts <= 0 || width % n_parts != 0 || (x && (dv <= 0 || width % dv != 0 || ld_x < width || !skip)) ||
        (z && ld_z < width))
        BL_FAIL("bl_gated_group_norm: bad sizes width=%d parts=%d dv=%d ld_x=%d ld_z=%d", width, n_parts, dv, ld_x, ld_z);
    if ((long long)T * n_parts > 2147483647LL) BL_FAIL("bl_gated_group_norm: %d rows in %d parts are more blocks than a launch takes", T, n_parts);
    const int blocks = T * n_parts;
    cudaStream_t s = (cudaStream_t)stream;
    if (y_dtype == BL_F32)
        BL_CUDA(bl_launch_dependent(gated_group_norm_kernel<float>, dim3(blocks), dim3(WARPS * 32), 0, s, o, x, ld_x, skip, skip_dtype, dv, z,
                                    ld_z, w, w_dtype, (float*)y, n_parts, width, eps));
    else if (y_dtype == BL_BF16)
        BL_CUDA(bl_launch_dependent(gated_group_norm_kernel<__nv_bfloat16>, dim3(blocks), dim3(WARPS * 32), 0, s, o, x, ld_x, skip, skip_dtype,
                                    dv, z, ld_z, w, w_dtype, (__nv_bfloat16*)y, n_parts, width, eps));
    else
        BL_FAIL("bl_gated_group_norm: unknown output dtype %d", y_dtype);
    BL_CHECK_LAUNCH("bl_gated_group_norm");
    return 0;
}
