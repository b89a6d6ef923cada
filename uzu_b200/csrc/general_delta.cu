// Generalized delta rule (per head a dim x dim f32 state S, key channel x value channel):
//     S <- diag(d) S - (a * u)(u^T S) + k v^T,   out = S^T r
// with decay d = exp(-e^-1/2 * sigmoid(.)), removal rate a = sigmoid(.), unit key u = k / sqrt(sum k^2 + 1e-6), all formed in f32 here
// from the raw projections. The value columns of a head are independent (u^T S is a per-column dot product).
//   general_delta_scan_kernel   passes of >= 4 tokens that bring a scratch: decay, rate * unit key and unit key of all tokens are formed in one
//                               parallel launch first (general_delta_prepare_kernel), then L lanes own a column and walk the tokens, two dot
//                               products and an update each, no barrier between tokens; the five vectors of a token come from shared memory,
//                               a batch of tokens ahead by cp.async. Bound: latency that nothing covers (one warp per scheduler).
//   general_delta_block_kernel  the same for passes of ten and more tokens, four per step, heads of 33..128 channels (column_block.cuh).
//   general_delta_kernel        the decode step and short passes: a CTA keeps a dim x 32 slice of the state in registers -- warp p owns PART
//                               key channels, lane c owns column c; partial sums meet in shared memory in warp order (a fixed order: one
//                               token at a time or several in one launch give the same bits).
#include <cstdlib>
#include <type_traits>

#include "column_block.cuh"
#include "common.cuh"

namespace uzu {


template <int PART>
__global__ void __launch_bounds__(1024) general_delta_kernel(const uzu_general_delta_args a) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ float gd_smem[];
    const uint32_t dim = a.dim, head = blockIdx.y;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, parts = blockDim.x >> 5;
    const uint32_t col = blockIdx.x * 32 + lane;
    const bool col_ok = col < dim;
    // shared memory: 2 x { d, au, u, k, r : dim each } + 2 x zpart[parts][32] + 2 x opart[parts][32] + 2 x ssq[32]
    float* vec = gd_smem;                                  // [2][5][dim]
    float* zpart = vec + 2 * 5 * dim;                      // [2][parts][32]
    float* opart = zpart + 2 * parts * 32;                 // [2][parts][32]
    float* ssq = opart + 2 * parts * 32;                   // [2][32]
    const uint32_t i0 = warp * PART;
    const uint32_t cnt = i0 < dim ? min((uint32_t)PART, dim - i0) : 0u;
    float* state = reinterpret_cast<float*>(a.state) + (size_t)head * dim * dim;
    float S[PART];
#pragma unroll
    for (int i = 0; i < PART; ++i) S[i] = ((uint32_t)i < cnt && col_ok) ? state[(size_t)(i0 + i) * dim + col] : 0.0f;

    const float* pr = reinterpret_cast<const float*>(a.r);
    const float* pk = reinterpret_cast<const float*>(a.k);
    const float* pv = reinterpret_cast<const float*>(a.v);
    const float* pa = reinterpret_cast<const float*>(a.rate_logit);
    const float* pd = reinterpret_cast<const float*>(a.decay_logit);
    const uint32_t hc = head * dim;
    const bool prep = tid < dim;
    const float rate_b = (prep && a.rate_bias) ? reinterpret_cast<const float*>(a.rate_bias)[hc + tid] : 0.0f;
    const float decay_b = (prep && a.decay_bias) ? reinterpret_cast<const float*>(a.decay_bias)[hc + tid] : 0.0f;
    // a token's inputs are requested three tokens ahead: the token-by-token chain never waits for memory
    struct Inputs { float k, r, a, d, v; };
    auto request = [&](uint32_t t) {
        Inputs q{0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
        if (t < a.rows) {
            if (prep) {
                q.k = pk[(size_t)t * a.k_stride + hc + tid];
                q.r = pr[(size_t)t * a.r_stride + hc + tid];
                q.a = pa[(size_t)t * a.rate_stride + hc + tid];
                q.d = pd[(size_t)t * a.decay_stride + hc + tid];
            }
            if (col_ok) q.v = pv[(size_t)t * a.v_stride + hc + col];
        }
        return q;
    };
    Inputs q0 = request(0), q1 = request(1), q2 = request(2);
    for (uint32_t t = 0; t < a.rows; ++t) {
        const uint32_t b = t & 1;
        float* vd = vec + (size_t)b * 5 * dim;
        float *vau = vd + dim, *vu = vau + dim, *vk = vu + dim, *vr = vk + dim;
        const Inputs cur = q0;
        q0 = q1;
        q1 = q2;
        q2 = request(t + 3);
        const float kk = cur.k, rr = cur.r, raw_a = cur.a, raw_d = cur.d, vv = cur.v;
        const float al = raw_a + rate_b, dl = raw_d + decay_b;
        const float sq = warp_sum(prep ? kk * kk : 0.0f);
        if (lane == 0) ssq[b * 32 + warp] = sq;
        __syncthreads();
        if (prep) {
            float total = 0.0f;
            for (uint32_t w = 0; w < parts; ++w) total += ssq[b * 32 + w];
            const float u = kk / sqrtf(total + 1e-6f);
            const float rate = 1.0f / (1.0f + expf(-al));
            const float decay = expf(-0.60653065971263342f * (1.0f / (1.0f + expf(-dl))));
            vd[tid] = decay;
            vau[tid] = rate * u;
            vu[tid] = u;
            vk[tid] = kk;
            vr[tid] = rr;
        }
        __syncthreads();
        float zp = 0.0f;
#pragma unroll
        for (int i = 0; i < PART; ++i)
            if ((uint32_t)i < cnt) zp = fmaf(vu[i0 + i], S[i], zp);
        zpart[(b * parts + warp) * 32 + lane] = zp;
        __syncthreads();
        float z = 0.0f;
        for (uint32_t w = 0; w < parts; ++w) z += zpart[(b * parts + w) * 32 + lane];
        float op = 0.0f;
#pragma unroll
        for (int i = 0; i < PART; ++i) {
            if ((uint32_t)i < cnt) {
                const float s = fmaf(vk[i0 + i], vv, fmaf(-vau[i0 + i], z, vd[i0 + i] * S[i]));
                S[i] = s;
                op = fmaf(s, vr[i0 + i], op);
            }
        }
        opart[(b * parts + warp) * 32 + lane] = op;
        __syncthreads();
        if (warp == 0 && col_ok) {
            float o = 0.0f;
            for (uint32_t w = 0; w < parts; ++w) o += opart[(b * parts + w) * 32 + lane];
            reinterpret_cast<float*>(a.out)[(size_t)t * a.heads * dim + hc + col] = o;
        }
    }
#pragma unroll
    for (int i = 0; i < PART; ++i)
        if ((uint32_t)i < cnt && col_ok) state[(size_t)(i0 + i) * dim + col] = S[i];
}

// One warp per (row, head): the per-token vectors of the recurrence for a whole pass at once, in place: decay_logit <- decay,
// rate_logit <- rate * unit key, unit <- unit key. Takes the transcendental functions out of the token-by-token chain of a prompt.
__global__ void __launch_bounds__(128) general_delta_prepare_kernel(const uzu_general_delta_args a) {
    pdl_launch_dependents();
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const uint32_t unit = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (unit >= a.rows * a.heads) return;
    const uint32_t row = unit / a.heads, h = unit % a.heads, hc = h * a.dim;
    const float* k = reinterpret_cast<const float*>(a.k) + (size_t)row * a.k_stride + hc;
    float* rate = reinterpret_cast<float*>(a.rate_logit) + (size_t)row * a.rate_stride + hc;
    float* decay = reinterpret_cast<float*>(a.decay_logit) + (size_t)row * a.decay_stride + hc;
    float* u = reinterpret_cast<float*>(a.unit) + (size_t)row * a.heads * a.dim + hc;
    const float* rb = a.rate_bias ? reinterpret_cast<const float*>(a.rate_bias) + hc : nullptr;
    const float* db = a.decay_bias ? reinterpret_cast<const float*>(a.decay_bias) + hc : nullptr;
    float ss = 0.0f;
    for (uint32_t i = lane; i < a.dim; i += 32) ss = fmaf(k[i], k[i], ss);
    const float inv = 1.0f / sqrtf(warp_sum(ss) + 1e-6f);
    for (uint32_t i = lane; i < a.dim; i += 32) {
        const float uu = k[i] * inv;
        const float al = rate[i] + (rb ? rb[i] : 0.0f), dl = decay[i] + (db ? db[i] : 0.0f);
        decay[i] = expf(-0.60653065971263342f * (1.0f / (1.0f + expf(-dl))));
        rate[i] = (1.0f / (1.0f + expf(-al))) * uu;
        u[i] = uu;
    }
}

// The tokens of a pass in order over ready-made vectors (decay in decay_logit, rate * unit key in rate_logit, unit key in `unit`): 4 warps per CTA,
// 32 / L columns per warp, grid (column blocks, heads). Bound: latency. 16 heads of 128 are 512 warps on 592 schedulers, and a warp's 20 shared 16-byte
// reads and its arithmetic of a token take 375 ns with nothing beside them; the dependent part (dot product over the lane's channels, log2 L shuffles, the
// update) is about a fifth of that. 1024 tokens, 16 heads of 128: 0.37 ms against 1.70 ms as a CTA per 32 columns with three barriers a token.
constexpr int GS_WARPS = 4;
template <int L, int NV>
constexpr int gs_batch() { return L * NV * 4 <= 128 ? 8 : (L * NV * 4 <= 256 ? 4 : 2); }

template <int L, int NV>
__global__ void __launch_bounds__(GS_WARPS * 32) general_delta_scan_kernel(const uzu_general_delta_args a, uint32_t vec) {
    constexpr int ROWF = L * NV * 4, BATCH = gs_batch<L, NV>(), CC = GS_WARPS * (32 / L);
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) float gs_smem[];
    float* vecs = gs_smem;                           // [2][BATCH][5][ROWF]: d, a * u, u, k, r
    float* vs = vecs + 2 * BATCH * 5 * ROWF;         // [2][BATCH][CC]
    const uint32_t dim = a.dim, h = blockIdx.y, hc = h * dim;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, part = lane % L;
    const uint32_t cl = warp * (32 / L) + lane / L, col0 = blockIdx.x * CC, col = col0 + cl;
    const bool col_ok = col < dim;
    const float* src[5] = {reinterpret_cast<const float*>(a.decay_logit) + hc, reinterpret_cast<const float*>(a.rate_logit) + hc,
                           reinterpret_cast<const float*>(a.unit) + hc, reinterpret_cast<const float*>(a.k) + hc, reinterpret_cast<const float*>(a.r) + hc};
    const uint32_t stride[5] = {a.decay_stride, a.rate_stride, a.heads * dim, a.k_stride, a.r_stride};
    const float* pv = reinterpret_cast<const float*>(a.v) + hc + col0;
    auto stage = [&](uint32_t tb, uint32_t buf) {
        const uint32_t nb = tb < a.rows ? min((uint32_t)BATCH, a.rows - tb) : 0u;
        float* dst = vecs + buf * BATCH * 5 * ROWF;
        if (vec) {                                   // rows and head offsets on 16-byte boundaries, dim a multiple of 4
            const uint32_t pieces = dim / 4;
#pragma unroll
            for (int w = 0; w < 5; ++w)
                for (uint32_t i = tid; i < nb * pieces; i += GS_WARPS * 32) {
                    const uint32_t r = i / pieces, c = (i - r * pieces) * 4;
                    gd_cp_async16(dst + (r * 5 + w) * ROWF + c, src[w] + (size_t)(tb + r) * stride[w] + c);
                }
        } else {
#pragma unroll
            for (int w = 0; w < 5; ++w)
                for (uint32_t i = tid; i < nb * dim; i += GS_WARPS * 32) {
                    const uint32_t r = i / dim, c = i - r * dim;
                    gd_cp_async4(dst + (r * 5 + w) * ROWF + c, src[w] + (size_t)(tb + r) * stride[w] + c);
                }
        }
        for (uint32_t i = tid; i < nb * CC; i += GS_WARPS * 32) {
            const uint32_t r = i / CC, c = i % CC;
            if (col0 + c < dim) gd_cp_async4(vs + (buf * BATCH + r) * CC + c, pv + (size_t)(tb + r) * a.v_stride + c);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (dim < (uint32_t)ROWF) {                      // channels past the head stay zero in both buffers
        const uint32_t tail = ROWF - dim;
        for (uint32_t i = tid; i < 2 * BATCH * 5 * tail; i += GS_WARPS * 32) vecs[i / tail * ROWF + dim + i % tail] = 0.0f;
    }
    stage(0, 0);
    float4 S[NV];
    float* state = reinterpret_cast<float*>(a.state) + (size_t)h * dim * dim + (col_ok ? col : 0u);
    auto at = [&](int i, int j) { return 4u * (i * L + part) + j; };
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        float s[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) s[j] = (col_ok && at(i, j) < dim) ? state[(size_t)at(i, j) * dim] : 0.0f;
        S[i] = make_float4(s[0], s[1], s[2], s[3]);
    }
    float* out = reinterpret_cast<float*>(a.out) + hc + col;
    const uint32_t out_stride = a.heads * dim;
    uint32_t buf = 0;
    for (uint32_t tb = 0; tb < a.rows; tb += BATCH, buf ^= 1) {
        const uint32_t nb = min((uint32_t)BATCH, a.rows - tb);
        stage(tb + BATCH, buf ^ 1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        const float* row = vecs + buf * BATCH * 5 * ROWF + part * 4;
        const float* v = vs + buf * BATCH * CC + cl;
        auto load_row = [&](float4 (&x)[NV], uint32_t r, int w) {
#pragma unroll
            for (int i = 0; i < NV; ++i) x[i] = *reinterpret_cast<const float4*>(row + (r * 5 + w) * ROWF + i * L * 4);
        };
        auto token = [&](uint32_t r) {               // one token; the lane's part of its read-out
            float4 u[NV], d[NV], au[NV], k[NV], rr[NV];
            load_row(u, r, 2);
            load_row(d, r, 0);
            load_row(au, r, 1);
            load_row(k, r, 3);
            load_row(rr, r, 4);
            const float vv = v[r * CC];
#pragma unroll
            for (int i = 0; i < NV; ++i) {           // what does not wait for the dot product: d S + k v
                d[i].x = fmaf(k[i].x, vv, d[i].x * S[i].x);
                d[i].y = fmaf(k[i].y, vv, d[i].y * S[i].y);
                d[i].z = fmaf(k[i].z, vv, d[i].z * S[i].z);
                d[i].w = fmaf(k[i].w, vv, d[i].w * S[i].w);
            }
            const float z = gd_lane_sum<L>(gd_dot<NV>(S, u));
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                S[i].x = fmaf(-au[i].x, z, d[i].x);
                S[i].y = fmaf(-au[i].y, z, d[i].y);
                S[i].z = fmaf(-au[i].z, z, d[i].z);
                S[i].w = fmaf(-au[i].w, z, d[i].w);
            }
            return gd_dot<NV>(S, rr);
        };
        if (nb == BATCH) {                           // straight-line code; the read-outs of the batch meet over the lanes all at once
            float o[BATCH];
#pragma unroll
            for (int j = 0; j < BATCH; ++j) o[j] = token(j);
            gd_transpose_sum<BATCH, L>(o, part);
            if (col_ok && part % (L / BATCH) == 0) out[(size_t)(tb + part / (L / BATCH)) * out_stride] = o[0];
        } else {
            for (uint32_t r = 0; r < nb; ++r) {
                const float o = gd_lane_sum<L>(token(r));
                if (part == 0 && col_ok) out[(size_t)(tb + r) * out_stride] = o;
            }
        }
        __syncthreads();
    }
    if (col_ok) {
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const float s[4] = {S[i].x, S[i].y, S[i].z, S[i].w};
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (at(i, j) < dim) state[(size_t)at(i, j) * dim] = s[j];
        }
    }
}

// The tokens of a pass four at a time, heads of 33..128 channels whose rows lie on 16-byte boundaries. With S the state at a block's start, P_j the
// product of the decays of its tokens before j and alpha = rate * unit key:
//     z_j = u_j . S_j = (u_j P_j) . S + sum_{i<j} -(u_j . (d_{i+1} .. d_{j-1} alpha_i)) z_i + (u_j . (d_{i+1} .. d_{j-1} k_i)) v_i
//     o_j = (r_j P_{j+1}) . S + sum_{i<=j} the same sums with r_j and one decay more
//     S' = P_4 S + sum_i (d_{i+1} .. d_3) (k_i v_i^T - alpha_i z_i^T)
// Producer warps (one per block) form the 17 vectors and the sums over channels, and invert the z_i system; decays are <= 1, so no product of them can
// grow. Consumer warps: see column_block.cuh; L lanes of four channels per group of Q columns.
// Bound: the shared-memory reads of a block (34 16-byte vector reads of each of four warps, in bursts) and the chain dot products -> lane sums -> exchange ->
// update: 1350 cycles a block, of which a scheduler issues 510 (16 heads of 128). More warps with fewer columns each read more and were slower (291 us), one reduction for both kinds of
// dot products instead of two was too (235 us). 1024 tokens with their preparation and copies: 16 heads of 128 206 us (386 token by token), 8 heads 0.20 ms
// (0.39), 32 heads 0.35 ms (0.57), 16 heads of 64 0.15 ms (0.24); 40 tokens 44 us (51).
template <int ROWF>
struct GbBlock {
    static constexpr int U = 0, A = 4 * ROWF, K = 8 * ROWF, R = 12 * ROWF, P = 16 * ROWF, T = 17 * ROWF, ZK = T + 12, OK = ZK + 16, OA = OK + 16, V = OA + 16;
    static constexpr int floats(int columns) { return V + 2 * CB_TOKENS * columns; }
};

template <int L, int NV, int Q>
__global__ void __launch_bounds__(CB_THREADS, 2) general_delta_block_kernel(const uzu_general_delta_args a) {
    constexpr int ROWF = L * NV * 4;
    using F = GbBlock<ROWF>;
    constexpr int GROUPS = 32 / L, CC = CB_WARPS * GROUPS * Q, U = CB_TOKENS * Q, SPAN = L / U, BLK = F::floats(CC);
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) float gb_smem[];
    float* zbuf = gb_smem + 2 * CB_BLOCKS * BLK;     // [2][CB_WARPS * GROUPS][U], twice each
    const uint32_t dim = a.dim, h = blockIdx.y, hc = h * dim, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, col0 = blockIdx.x * CC;
    const uint32_t steps = (a.rows + CB_BLOCKS * CB_TOKENS - 1) / (CB_BLOCKS * CB_TOKENS);

    if (warp >= CB_WARPS) {                          // producer of block `which` of every step
        const uint32_t which = warp - CB_WARPS, ch = 4 * lane;
        const bool ch_ok = ch < dim;
        const uint32_t stride[5] = {a.decay_stride, a.rate_stride, a.heads * dim, a.k_stride, a.r_stride};
        const float* src[5] = {reinterpret_cast<const float*>(a.decay_logit) + hc + ch, reinterpret_cast<const float*>(a.rate_logit) + hc + ch,
                               reinterpret_cast<const float*>(a.unit) + hc + ch, reinterpret_cast<const float*>(a.k) + hc + ch, reinterpret_cast<const float*>(a.r) + hc + ch};
        cb_f4 x[5][CB_TOKENS];                      // d, alpha, u, k, r; a token past the pass changes nothing (d = 1, the others 0)
        float v[CB_TOKENS];
        auto fetch = [&](uint32_t step) {
            const uint32_t t0 = (step * CB_BLOCKS + which) * CB_TOKENS;
#pragma unroll
            for (int j = 0; j < CB_TOKENS; ++j) {
                const bool ok = t0 + j < a.rows;
#pragma unroll
                for (int w = 0; w < 5; ++w) {
                    const float none = w == 0 ? 1.0f : 0.0f;
                    x[w][j] = ok && ch_ok ? cb_load4(src[w] + (size_t)(t0 + j) * stride[w]) : cb_set4(none);
                }
                v[j] = ok && lane < CC && col0 + lane < dim ? reinterpret_cast<const float*>(a.v)[(size_t)(t0 + j) * a.v_stride + hc + col0 + lane] : 0.0f;
            }
        };
        auto produce = [&](uint32_t step) {
            float* B = gb_smem + ((step & 1) * CB_BLOCKS + which) * BLK;
            const bool in_row = ch < (uint32_t)ROWF;
            auto put = [&](int off, const cb_f4& y) { if (in_row) cb_store4(B + off + ch, y); };
            cb_f4 (&d)[CB_TOKENS] = x[0];
            cb_f4 p = d[0];
            put(F::U, x[2][0]);
            put(F::R, cb_mul(x[4][0], p));
#pragma unroll
            for (int j = 1; j < CB_TOKENS; ++j) {
                put(F::U + j * ROWF, cb_mul(x[2][j], p));
                p = cb_mul(p, d[j]);
                put(F::R + j * ROWF, cb_mul(x[4][j], p));
            }
            put(F::P, p);
            // sums over the channels: [0, 6) u . -alpha, [6, 12) u . k (strictly lower), [12, 22) r . -alpha, [22, 32) r . k (with the diagonal)
            float s[32];
#pragma unroll
            for (int i = 0; i < CB_TOKENS; ++i) {
                cb_f4 al = cb_scale(x[1][i], cb_pack(-1.0f, -1.0f)), k = x[3][i];
#pragma unroll
                for (int j = i; j < CB_TOKENS; ++j) {
                    if (j > i) {
                        s[j * (j - 1) / 2 + i] = cb_dot(x[2][j], al);
                        s[6 + j * (j - 1) / 2 + i] = cb_dot(x[2][j], k);
                        al = cb_mul(al, d[j]);
                        k = cb_mul(k, d[j]);
                    }
                    s[12 + j * (j + 1) / 2 + i] = cb_dot(x[4][j], al);
                    s[22 + j * (j + 1) / 2 + i] = cb_dot(x[4][j], k);
                }
                put(F::A + i * ROWF, al);
                put(F::K + i * ROWF, k);
            }
            gd_transpose_sum<32, 32>(s, lane);
            float n[6], t[6];
#pragma unroll
            for (int e = 0; e < 6; ++e) n[e] = __shfl_sync(0xffffffffu, s[0], e);
            cb_invert(n, t);
            uint32_t j, i;
            if (lane == 0) {
                cb_store_solve(B + F::T, t);
            } else if (lane >= 6 && lane < 12) {
                cb_strict(lane - 6, j, i);
                B[F::ZK + j * 4 + i] = s[0];
            } else if (lane >= 12) {
                cb_lower(lane < 22 ? lane - 12 : lane - 22, j, i);
                B[(lane < 22 ? F::OA : F::OK) + j * 4 + i] = s[0];
            }
            if (lane < CC) {
#pragma unroll
                for (int j2 = 0; j2 < CB_TOKENS; ++j2) *reinterpret_cast<float2*>(B + F::V + 2 * (j2 * CC + lane)) = make_float2(v[j2], v[j2]);
            }
        };
        fetch(0);
        produce(0);
        fetch(1);
        for (uint32_t step = 0; step < steps; ++step) {
            __syncthreads();                         // step's blocks are ready, the other buffer is free
            if (step + 1 < steps) {
                produce(step + 1);
                fetch(step + 2);
            }
        }
        return;
    }

    const uint32_t part = lane % L, group = warp * GROUPS + lane / L, lc = group * Q, col = col0 + lc, ch = 4 * part;
    const uint32_t idx = part / SPAN, oj = idx / Q, oc = idx % Q;      // after a reduction the lane holds (token, column) oj, oc
    const bool first = part % SPAN == 0, owner = first && col + oc < dim;
    cb_f4 S[Q][NV];
    float* state = reinterpret_cast<float*>(a.state) + (size_t)h * dim * dim + col;
#pragma unroll
    for (int c = 0; c < Q; ++c)
#pragma unroll
        for (int n = 0; n < NV; ++n) {
            const uint32_t cn = ch + 4 * L * n;
            const float* p = state + (size_t)cn * dim + c;
            if (col + c < dim && cn < dim) S[c][n] = {cb_pack(p[0], p[dim]), cb_pack(p[2 * dim], p[3 * dim])};
            else S[c][n] = cb_set4(0.0f);
        }
    float* out = reinterpret_cast<float*>(a.out) + hc + col + oc;
    const uint32_t out_stride = a.heads * dim;
    for (uint32_t step = 0; step < steps; ++step) {
        __syncthreads();
        const uint32_t t_step = step * CB_BLOCKS * CB_TOKENS, nblocks = min((uint32_t)CB_BLOCKS, (a.rows - t_step + CB_TOKENS - 1) / CB_TOKENS);
        for (uint32_t b = 0; b < nblocks; ++b) {
            const float* B = gb_smem + ((step & 1) * CB_BLOCKS + b) * BLK;
            float* zb = zbuf + ((b & 1) * CB_WARPS * GROUPS + group) * U * 2;
            auto load = [&](cb_f4 (&y)[CB_TOKENS][NV], int off) {
#pragma unroll
                for (int j = 0; j < CB_TOKENS; ++j)
#pragma unroll
                    for (int n = 0; n < NV; ++n) y[j][n] = cb_load4(B + off + j * ROWF + ch + 4 * L * n);
            };
            cb_f4 x[CB_TOKENS][NV];
            float zp[U], op[U], vown[CB_TOKENS];
            cb_f2 v[CB_TOKENS][Q];
            load(x, F::U);
            cb_dots<NV, Q>(zp, x, S);
            load(x, F::R);
#pragma unroll
            for (int j = 0; j < CB_TOKENS; ++j) {
                vown[j] = B[F::V + 2 * (j * CC + lc + oc)];
                cb_load<Q>(v[j], B + F::V + 2 * (j * CC + lc));
            }
            const float4 zk = *reinterpret_cast<const float4*>(B + F::ZK + oj * 4);
            gd_transpose_sum<U, L>(zp, part);
            // the right-hand side of (token, column); a later token's value reaches no earlier one, not even as 0 * x
            const float r = cb_upto(zp[0], zk, vown, oj);
            if (first) *reinterpret_cast<float2*>(zb + 2 * idx) = make_float2(r, r);
            __syncwarp();                            // the buffer's next writer is two blocks on, behind another one of these
            cb_dots<NV, Q>(op, x, S);
            load(x, F::K);
#pragma unroll
            for (int n = 0; n < NV; ++n) {
                const cb_f4 p = cb_load4(B + F::P + ch + 4 * L * n);
#pragma unroll
                for (int c = 0; c < Q; ++c) S[c][n] = cb_mul(S[c][n], p);
            }
            cb_update<NV, Q>(S, x, v);
            cb_f2 z[CB_TOKENS][Q], rhs[CB_TOKENS][Q];
#pragma unroll
            for (int j = 0; j < CB_TOKENS; ++j) cb_load<Q>(rhs[j], zb + 2 * j * Q);
            cb_solve<Q>(z, rhs, B + F::T);
            load(x, F::A);
            cb_update<NV, Q>(S, x, z);
            gd_transpose_sum<U, L>(op, part);
            float zown[CB_TOKENS];
#pragma unroll
            for (int j = 0; j < CB_TOKENS; ++j) zown[j] = cb_pick<Q>(z[j], oc);
            float o = cb_upto(op[0], *reinterpret_cast<const float4*>(B + F::OK + oj * 4), vown, oj + 1);
            o = cb_upto(o, *reinterpret_cast<const float4*>(B + F::OA + oj * 4), zown, oj + 1);
            const uint32_t t = t_step + b * CB_TOKENS + oj;
            if (owner && t < a.rows) out[(size_t)t * out_stride] = o;
        }
    }
#pragma unroll
    for (int c = 0; c < Q; ++c)
#pragma unroll
        for (int n = 0; n < NV; ++n) {
            const uint32_t cn = ch + 4 * L * n;
            if (col + c >= dim || cn >= dim) continue;
            float* p = state + (size_t)cn * dim + c;
            p[0] = cb_lo(S[c][n].a);
            p[dim] = cb_hi(S[c][n].a);
            p[2 * dim] = cb_lo(S[c][n].b);
            p[3 * dim] = cb_hi(S[c][n].b);
        }
}

static void launch_general_delta_scan(uzu_command_buffer* cmd, const uzu_general_delta_args& a) {
    // 16-byte copies where every row of every vector starts on a 16-byte boundary
    const uint32_t vec = !((a.decay_logit | a.rate_logit | a.unit | a.k | a.r) & 15u) &&
                         !((a.decay_stride | a.rate_stride | a.k_stride | a.r_stride | a.dim) & 3u);
    auto go = [&](auto l_c, auto nv_c) {
        constexpr int L = decltype(l_c)::value, NV = decltype(nv_c)::value, CC = GS_WARPS * (32 / L), BATCH = gs_batch<L, NV>();
        constexpr size_t smem = ((size_t)2 * BATCH * 5 * L * NV * 4 + (size_t)2 * BATCH * CC) * sizeof(float);
        static std::atomic<uint64_t> done{0};
        if (smem > 48 * 1024) opt_in_dynamic_smem(cmd, general_delta_scan_kernel<L, NV>, (int)smem, done);
        launch(cmd, "general_delta_scan_kernel", general_delta_scan_kernel<L, NV>, dim3((a.dim + CC - 1) / CC, a.heads), dim3(GS_WARPS * 32), smem, a, vec);
    };
    // Four tokens at a time wherever a row's channels fit the lanes as float4, from ten tokens on. With the preparation, token by token / blocks, us: 16 heads of
    // 128, 5 tokens 10.4 / 11.5, 10 tokens 12.5 / 12.5, 16 tokens 15.0 / 12.8; 64 heads of 64, 9 tokens 11.6 / 12.5, 10 tokens 12.5 / 12.5, 64 tokens 27.8 / 23.7.
    // One column per lane group while such CTAs have an SM each (8 heads of 128, 1024 tokens: 166 us, 178 with two columns); more of them share an SM's issue
    // slots and shared memory, and two columns per lane group are faster in half the CTAs (10 heads 179 us, 272 with one; 16 heads 183, 273).
    if (vec && a.dim > 32 && a.dim <= 128 && a.rows >= 10) {
        auto blocks = [&](auto nv_c, auto q_c) {
            constexpr int L = 16, NV = decltype(nv_c)::value, Q = decltype(q_c)::value, GROUPS = CB_WARPS * (32 / L), CC = GROUPS * Q;
            constexpr size_t smem = ((size_t)2 * CB_BLOCKS * GbBlock<L * NV * 4>::floats(CC) + (size_t)4 * GROUPS * CB_TOKENS * Q) * sizeof(float);
            static std::atomic<uint64_t> done{0};
            if (smem > 48 * 1024) opt_in_dynamic_smem(cmd, general_delta_block_kernel<L, NV, Q>, (int)smem, done);
            launch(cmd, "general_delta_scan_kernel", general_delta_block_kernel<L, NV, Q>, dim3((a.dim + CC - 1) / CC, a.heads), dim3(CB_THREADS), smem, a);
        };
        auto one = std::integral_constant<int, 1>{};
        auto two = std::integral_constant<int, 2>{};
        const bool one_column = a.heads * ((a.dim + 7) / 8) <= (uint32_t)cmd->ctx->sm_count;
        if (a.dim <= 64) one_column ? blocks(one, one) : blocks(one, two);
        else one_column ? blocks(two, one) : blocks(two, two);
        return;
    }
    auto l8 = std::integral_constant<int, 8>{};
    if (a.dim <= 32) go(l8, std::integral_constant<int, 1>{});
    else if (a.dim <= 64) go(l8, std::integral_constant<int, 2>{});
    else if (a.dim <= 128) go(l8, std::integral_constant<int, 4>{});
    else if (a.dim <= 256) go(std::integral_constant<int, 16>{}, std::integral_constant<int, 4>{});
    else go(std::integral_constant<int, 32>{}, std::integral_constant<int, 4>{});
}

// one warp per (row, head)
// WIDE: a CTA per (row, head) instead of a warp: long heads (a norm over all heads at once)
template <bool WIDE>
__global__ void __launch_bounds__(WIDE ? 512 : 128) head_norm_gate_kernel(const uzu_head_norm_gate_args a) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ float red[32];
    const uint32_t lane = WIDE ? threadIdx.x : threadIdx.x & 31, step = WIDE ? blockDim.x : 32u;
    const uint32_t unit = WIDE ? blockIdx.x : blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (unit >= a.rows * a.heads) return;
    const uint32_t row = unit / a.heads, h = unit % a.heads;
    const float* x = reinterpret_cast<const float*>(a.x) + (size_t)row * a.x_stride + (size_t)h * a.dim;
    const float* gate = a.gate ? reinterpret_cast<const float*>(a.gate) + (size_t)row * a.gate_stride + (size_t)h * a.dim : nullptr;
    const float* sc = a.scales ? reinterpret_cast<const float*>(a.scales) + (size_t)h * a.dim : nullptr;
    float* out = reinterpret_cast<float*>(a.out) + (size_t)row * a.out_stride + (size_t)h * a.dim;
    float inv = 1.0f, pre = 1.0f;
    if (a.denom) {          // the row is first divided by max(|denom|, floor) + denom_epsilon
        float d = fabsf(reinterpret_cast<const float*>(a.denom)[(size_t)row * a.heads + h]);
        if (a.denom_floor) d = fmaxf(d, reinterpret_cast<const float*>(a.denom_floor)[(size_t)row * a.heads + h]);
        pre = 1.0f / (d + a.denom_epsilon);
    }
    if (a.normalize) {
        float ss = 0.0f;
        for (uint32_t i = lane; i < a.dim; i += step) { const float y = x[i] * pre; ss = fmaf(y, y, ss); }
        ss = WIDE ? block_sum(ss, red) : warp_sum(ss);
        inv = 1.0f / sqrtf(ss / (float)a.dim + a.epsilon);
    }
    const float out_scale = a.out_scale != 0.0f ? a.out_scale : 1.0f;
    for (uint32_t i = lane; i < a.dim; i += step) {
        float v = x[i] * pre * inv;
        if (sc) v *= sc[i];
        if (gate) v *= a.gate_op == 1 ? gate[i] / (1.0f + expf(-gate[i])) : 1.0f / (1.0f + expf(-gate[i]));
        out[i] = v * out_scale;
    }
}

}  // namespace uzu

extern "C" {
using namespace uzu;

void uzu_general_delta_encode(uzu_command_buffer* cmd, const uzu_general_delta_args* a) {
    if (!encodable(cmd, "general_delta")) return;
    if (!a->r || !a->k || !a->v || !a->rate_logit || !a->decay_logit || !a->state || !a->out || a->dim == 0 || a->dim > 512 || a->heads == 0) {
        cmd->record_error(UZU_ERROR_INVALID_ARGUMENT, "general_delta: null operand or head size outside 1..512");
        return;
    }
    if (a->rows == 0) return;
    // passes of several tokens with a scratch for the unit keys: the per-token vectors are formed for all tokens at once first
    if (a->unit != 0 && a->rows >= 4) {
        const uint32_t units = a->rows * a->heads;
        launch(cmd, "general_delta_prepare_kernel", general_delta_prepare_kernel, dim3((units + 3) / 4), dim3(128), 0, *a);
        launch_general_delta_scan(cmd, *a);
        return;
    }
    // key channels per warp: about 16 warps per CTA whatever the head size (4 channels up to 64, 8 at 128, ...), so that a thread's
    // token-by-token chain is short and the schedulers have other warps to issue from. Measured, 1024 tokens, 16 heads: head 128: 2.95 ms
    // with 16 channels per warp, 1.70 ms with 8, 1.74 ms with 4; head 64: 0.98 ms with 4, 1.37 ms with 8; head 48: 0.92 ms with 4.
    static const int part_env = [] { const char* e = getenv("UZU_DELTA_PART"); return e ? atoi(e) : 0; }();   // A/B runs: 4 | 8 | 16 | 32
    int part = 4;
    while (part * 16 < (int)a->dim) part *= 2;
    if (part_env == 4 || part_env == 8 || part_env == 16 || part_env == 32) part = part_env;
    while ((a->dim + part - 1) / part > 32) part *= 2;
    const uint32_t parts = (a->dim + part - 1) / part;
    const size_t smem = ((size_t)2 * 5 * a->dim + (size_t)4 * parts * 32 + 64) * sizeof(float);
    const dim3 grid((a->dim + 31) / 32, a->heads), block(parts * 32);
    auto go = [&](auto kernel, std::atomic<uint64_t>& done) {
        if (smem > 48 * 1024) opt_in_dynamic_smem(cmd, kernel, (int)smem, done);
        launch(cmd, "general_delta_kernel", kernel, grid, block, smem, *a);
    };
    static std::atomic<uint64_t> done[4];
    if (part == 4) go(general_delta_kernel<4>, done[0]);
    else if (part == 8) go(general_delta_kernel<8>, done[1]);
    else if (part == 16) go(general_delta_kernel<16>, done[2]);
    else go(general_delta_kernel<32>, done[3]);
}

void uzu_head_norm_gate_encode(uzu_command_buffer* cmd, const uzu_head_norm_gate_args* a) {
    if (!encodable(cmd, "head_norm_gate")) return;
    if (!a->x || !a->out || a->dim == 0 || a->heads == 0) {
        cmd->record_error(UZU_ERROR_INVALID_ARGUMENT, "head_norm_gate: null operand");
        return;
    }
    if (a->rows == 0) return;
    uzu_head_norm_gate_args b = *a;
    if (!b.x_stride) b.x_stride = b.heads * b.dim;
    if (!b.gate_stride) b.gate_stride = b.heads * b.dim;
    if (!b.out_stride) b.out_stride = b.heads * b.dim;
    const uint32_t units = b.rows * b.heads;
    if (b.dim > 512)
        launch(cmd, "head_norm_gate_kernel", head_norm_gate_kernel<true>, dim3(units), dim3(b.dim > 2048 ? 512 : 256), 0, b);
    else
        launch(cmd, "head_norm_gate_kernel", head_norm_gate_kernel<false>, dim3((units + 3) / 4), dim3(128), 0, b);
}

}  // extern "C"
