// Gated delta rule with one decay per head, for any head sizes, f32 throughout. Per head a state S [dim, vdim]:
//     S <- g S;  S <- S + k (beta (v - S^T k))^T;  o = S^T q
// with q, k, v behind a short causal convolution per channel and silu, q and k unit vectors, g = exp(-exp(A) softplus(.)), beta = sigmoid(.).
//
// A column of S (one value channel) needs no other column: S^T k and S^T q are dot products along it. So L neighbouring lanes own a column --
// lane part p holds the key channels {4 (i L + p) .. + 3}, NV float4 in registers -- and a token costs two dot products, two shuffle
// reductions over L lanes and no barrier at all. q and k rows are read from shared memory as float4 with the L parts side by side (128
// contiguous bytes at L = 8: no bank conflict, the columns of a warp share the read).
//   gated_delta_block_kernel the tokens of a longer pass four at a time, keys of 33..128 channels (column_block.cuh). Sums in another order than token by
//                            token: how a prompt is cut shows in an element's last bits.
//   gated_delta_kernel       the tokens of a pass in order, 4 warps per CTA, grid (column blocks, heads). The prepared q / k / v / decay / beta
//                            rows arrive by cp.async one batch ahead. Passes that all go this way give the same bits however they are cut.
//   delta_prepare_kernel     convolution, silu, unit vectors and gates of all tokens of a pass at once, a warp per (a few tokens, head).
//   gated_delta_step_kernel  one token with everything between the projections in one launch: a cluster of CL CTAs per head, each CTA owning
//                            vdim / CL columns; the state is requested before the previous kernel's results are waited for; the head's sum
//                            of squares meets through distributed shared memory in rank order; norm weight and silu gate applied on the way out.
// The convolution's earlier inputs live in a ring of `taps` rows indexed by position % taps: the step kernel writes the slot of its own token
// while all CTAs read the other taps - 1 slots, so no ordering between the CTAs is needed (several value heads may share a key head).
#include <type_traits>

#include "column_block.cuh"
#include "common.cuh"

namespace uzu {

namespace {

constexpr float kUnitEps = 1e-6f;

__device__ __forceinline__ float gd_silu(float x) { return x / (1.0f + expf(-x)); }
__device__ __forceinline__ float gd_sigmoid(float x) { return 1.0f / (1.0f + expf(-x)); }
__device__ __forceinline__ float gd_decay(float a_log, float a) {
    const float softplus = fmaxf(a, 0.0f) + log1pf(expf(-fabsf(a)));
    return expf(-expf(a_log) * softplus);
}

__device__ __forceinline__ uint32_t gd_prefix(const uzu_delta_prepare_args& a) {
    return a.dynamic_position ? *reinterpret_cast<const uint32_t*>(a.dynamic_position) : a.prefix;
}

// silu of the convolution of channel c at row t of the pass (position prefix + t)
__device__ __forceinline__ float gd_conv(const uzu_delta_prepare_args& a, uint32_t channels, uint32_t prefix, uint32_t t, uint32_t c) {
    const float* proj = reinterpret_cast<const float*>(a.proj) + c;
    const float* w = reinterpret_cast<const float*>(a.conv) + (size_t)c * a.taps;
    const float* ring = reinterpret_cast<const float*>(a.ring) + c;
    float y = 0.0f;
    for (uint32_t j = 0; j < a.taps; ++j) {
        const uint32_t back = a.taps - 1 - j;                    // tokens before the current one
        float x = 0.0f;
        if (back <= t) x = proj[(size_t)(t - back) * a.stride];
        else if (back <= prefix + t) x = ring[(size_t)((prefix + t - back) % a.taps) * channels];
        y = fmaf(w[j], x, y);
    }
    return gd_silu(y);
}

// the convolution of channel c at position `prefix` without its last tap (all inputs come from the ring), and that tap's weight
__device__ __forceinline__ void gd_conv_past(const uzu_delta_prepare_args& a, uint32_t channels, uint32_t prefix, uint32_t c, float& past, float& tap) {
    const float* w = reinterpret_cast<const float*>(a.conv) + (size_t)c * a.taps;
    const float* ring = reinterpret_cast<const float*>(a.ring) + c;
    past = 0.0f;
    for (uint32_t j = 0; j + 1 < a.taps; ++j) {
        const uint32_t back = a.taps - 1 - j;
        if (back <= prefix) past = fmaf(w[j], ring[(size_t)((prefix - back) % a.taps) * channels], past);
    }
    tap = w[a.taps - 1];
}

}  // namespace

// A warp per (block of GP_ROWS tokens, unit): units [0, kv_heads) queries, [kv_heads, 2 kv_heads) keys, then the value heads, then one unit for
// the gates. NC = channels of a head per lane; the convolution's window of a channel slides through registers, so an input is read once.
constexpr int GP_ROWS = 8;

template <int TAPS, int NC>
__global__ void __launch_bounds__(128) delta_prepare_window_kernel(const uzu_delta_prepare_args a) {
    pdl_launch_dependents();
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t units = 2 * a.kv_heads + a.heads + 1, blocks = (a.rows + GP_ROWS - 1) / GP_ROWS;
    const uint32_t item = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (item >= blocks * units) return;
    const uint32_t t0 = item / units * GP_ROWS, unit = item % units, nr = min((uint32_t)GP_ROWS, a.rows - t0);
    const uint32_t kd = a.kv_heads * a.dim, channels = 2 * kd + a.heads * a.vdim, dim4 = (a.dim + 3) & ~3u;
    if (unit == units - 1) {
        pdl_wait();
        for (uint32_t i = lane; i < nr * a.heads; i += 32) {
            const uint32_t t = t0 + i / a.heads, h = i % a.heads;
            const float* row = reinterpret_cast<const float*>(a.proj) + (size_t)t * a.stride;
            reinterpret_cast<float*>(a.decay)[(size_t)t * a.heads + h] =
                gd_decay(reinterpret_cast<const float*>(a.a_log)[h], row[a.a_offset + h] + reinterpret_cast<const float*>(a.dt_bias)[h]);
            reinterpret_cast<float*>(a.beta)[(size_t)t * a.heads + h] = gd_sigmoid(row[a.b_offset + h]);
        }
        return;
    }
    const bool is_q = unit < a.kv_heads, is_v = unit >= 2 * a.kv_heads;
    const uint32_t head = is_q ? unit : (is_v ? unit - 2 * a.kv_heads : unit - a.kv_heads), n = is_v ? a.vdim : a.dim;
    const uint32_t c0 = is_q ? head * a.dim : (is_v ? 2 * kd + head * a.vdim : kd + head * a.dim);
    const uint32_t pad = is_v ? n : dim4;                        // q / k rows are padded to whole float4
    float* out = reinterpret_cast<float*>(is_q ? a.q : (is_v ? a.v : a.k)) + ((size_t)t0 * (is_v ? a.heads : a.kv_heads) + head) * pad;
    const size_t out_stride = (size_t)(is_v ? a.heads : a.kv_heads) * pad;
    const float* proj = reinterpret_cast<const float*>(a.proj) + (size_t)t0 * a.stride + c0;
    float w[NC][TAPS], x[NC][TAPS + GP_ROWS - 1];
#pragma unroll
    for (int i = 0; i < NC; ++i) {
        const uint32_t c = lane + 32u * i;
#pragma unroll
        for (int j = 0; j < TAPS; ++j) w[i][j] = c < n ? reinterpret_cast<const float*>(a.conv)[(size_t)(c0 + c) * TAPS + j] : 0.0f;
    }
    pdl_wait();
    const uint32_t prefix = gd_prefix(a);
#pragma unroll
    for (int i = 0; i < NC; ++i) {
        const uint32_t c = lane + 32u * i;
#pragma unroll
        for (int j = 0; j < TAPS + GP_ROWS - 1; ++j) {
            const int t = j - (TAPS - 1);                        // row relative to the block's first
            float v = 0.0f;
            if (c < n) {
                if (t >= 0 || (uint32_t)(-t) <= t0) { if (t < (int)nr) v = proj[(ptrdiff_t)t * a.stride + c]; }
                else if ((uint32_t)(-t) <= prefix + t0)
                    v = reinterpret_cast<const float*>(a.ring)[(size_t)((prefix + t0 + t) % TAPS) * channels + c0 + c];
            }
            x[i][j] = v;
        }
    }
#pragma unroll
    for (int r = 0; r < GP_ROWS; ++r) {
        if ((uint32_t)r >= nr) break;
        float y[NC], f = 1.0f;
#pragma unroll
        for (int i = 0; i < NC; ++i) {
            float s = 0.0f;
#pragma unroll
            for (int j = 0; j < TAPS; ++j) s = fmaf(w[i][j], x[i][r + j], s);
            y[i] = gd_silu(s);
        }
        if (!is_v) {
            float ss = 0.0f;
#pragma unroll
            for (int i = 0; i < NC; ++i) ss = fmaf(y[i], y[i], ss);      // (channels past the head hold zero)
            f = 1.0f / sqrtf(warp_sum(ss) + kUnitEps);
            if (is_q) f *= 1.0f / sqrtf((float)a.dim);
        }
#pragma unroll
        for (int i = 0; i < NC; ++i) {
            const uint32_t c = lane + 32u * i;
            if (c < pad) out[(size_t)r * out_stride + c] = y[i] * f;
        }
    }
}

// the same for any number of taps and any head size: a warp per (token, unit), every input read once per tap
__global__ void __launch_bounds__(128) delta_prepare_kernel(const uzu_delta_prepare_args a) {
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t units = 2 * a.kv_heads + a.heads + 1;
    const uint32_t item = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (item >= a.rows * units) return;
    const uint32_t t = item / units, unit = item % units;
    const uint32_t kd = a.kv_heads * a.dim, channels = 2 * kd + a.heads * a.vdim, dim4 = (a.dim + 3) & ~3u;
    const uint32_t prefix = gd_prefix(a);
    if (unit < 2 * a.kv_heads) {
        const bool is_q = unit < a.kv_heads;
        const uint32_t head = is_q ? unit : unit - a.kv_heads;
        const uint32_t c0 = (is_q ? 0u : kd) + head * a.dim;
        float* out = reinterpret_cast<float*>(is_q ? a.q : a.k) + ((size_t)t * a.kv_heads + head) * dim4;
        constexpr int KEEP = 8;
        float x[KEEP], ss = 0.0f;
#pragma unroll
        for (int i = 0; i < KEEP; ++i) {
            const uint32_t c = lane + 32u * i;
            x[i] = c < a.dim ? gd_conv(a, channels, prefix, t, c0 + c) : 0.0f;
            ss = fmaf(x[i], x[i], ss);
        }
        for (uint32_t c = lane + 32u * KEEP; c < a.dim; c += 32) {          // long heads: the rest waits in the output row
            const float y = gd_conv(a, channels, prefix, t, c0 + c);
            out[c] = y;
            ss = fmaf(y, y, ss);
        }
        float f = 1.0f / sqrtf(warp_sum(ss) + kUnitEps);
        if (is_q) f *= 1.0f / sqrtf((float)a.dim);
#pragma unroll
        for (int i = 0; i < KEEP; ++i) {
            const uint32_t c = lane + 32u * i;
            if (c < dim4) out[c] = x[i] * f;                               // the pad channels hold zero
        }
        for (uint32_t c = lane + 32u * KEEP; c < dim4; c += 32) out[c] = c < a.dim ? out[c] * f : 0.0f;
    } else if (unit < 2 * a.kv_heads + a.heads) {
        const uint32_t h = unit - 2 * a.kv_heads;
        float* out = reinterpret_cast<float*>(a.v) + ((size_t)t * a.heads + h) * a.vdim;
        for (uint32_t c = lane; c < a.vdim; c += 32) out[c] = gd_conv(a, channels, prefix, t, 2 * kd + h * a.vdim + c);
    } else {
        const float* row = reinterpret_cast<const float*>(a.proj) + (size_t)t * a.stride;
        for (uint32_t h = lane; h < a.heads; h += 32) {
            reinterpret_cast<float*>(a.decay)[(size_t)t * a.heads + h] =
                gd_decay(reinterpret_cast<const float*>(a.a_log)[h], row[a.a_offset + h] + reinterpret_cast<const float*>(a.dt_bias)[h]);
            reinterpret_cast<float*>(a.beta)[(size_t)t * a.heads + h] = gd_sigmoid(row[a.b_offset + h]);
        }
    }
}

constexpr int GD_WARPS = 4;

template <int L, int NV>
constexpr int gd_batch() { return L * NV * 4 <= 256 ? 16 : (L * NV * 4 <= 512 ? 8 : 4); }

// the pass's last inputs of the convolution go to the ring (the launch before the scan was its last reader); all threads of the grid take part
__device__ __forceinline__ void gd_ring_store(const uzu_delta_prepare_args& a) {
    const uint32_t channels = 2 * a.kv_heads * a.dim + a.heads * a.vdim, prefix = gd_prefix(a), keep = min(a.rows, a.taps - 1);
    const uint32_t threads = gridDim.x * gridDim.y * blockDim.x, me = (blockIdx.y * gridDim.x + blockIdx.x) * blockDim.x + threadIdx.x;
    const float* proj = reinterpret_cast<const float*>(a.proj);
    float* ring = reinterpret_cast<float*>(a.ring);
    for (uint32_t i = me; i < keep * channels; i += threads) {
        const uint32_t t = a.rows - keep + i / channels, c = i % channels;
        ring[(size_t)((prefix + t) % a.taps) * channels + c] = proj[(size_t)t * a.stride + c];
    }
}

template <int L, int NV>
__global__ void __launch_bounds__(GD_WARPS * 32) gated_delta_kernel(const uzu_gated_delta_args ga) {
    constexpr int ROWF = L * NV * 4, BATCH = gd_batch<L, NV>(), CC = GD_WARPS * (32 / L), U = BATCH < 8 ? BATCH : 8;
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) float gd_smem[];
    float* qs = gd_smem;                             // [2][BATCH][ROWF]
    float* ks = qs + 2 * BATCH * ROWF;               // [2][BATCH][ROWF]
    float* vs = ks + 2 * BATCH * ROWF;               // [2][BATCH][CC]
    float* gs = vs + 2 * BATCH * CC;                 // [2][BATCH] decay
    float* bs = gs + 2 * BATCH;                      // [2][BATCH] beta
    const uzu_delta_prepare_args& a = ga.prep;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, part = lane % L;
    const uint32_t h = blockIdx.y, kvh = h / (a.heads / a.kv_heads), dim4 = (a.dim + 3) & ~3u, pieces = dim4 / 4;
    const uint32_t cl = warp * (32 / L) + lane / L, col0 = blockIdx.x * CC, col = col0 + cl;
    const bool col_ok = col < a.vdim;
    const float* pq = reinterpret_cast<const float*>(a.q) + (size_t)kvh * dim4;
    const float* pk = reinterpret_cast<const float*>(a.k) + (size_t)kvh * dim4;
    const float* pv = reinterpret_cast<const float*>(a.v) + (size_t)h * a.vdim + col0;
    const float* pg = reinterpret_cast<const float*>(a.decay) + h;
    const float* pb = reinterpret_cast<const float*>(a.beta) + h;
    const size_t qk_stride = (size_t)a.kv_heads * dim4, v_stride = (size_t)a.heads * a.vdim;
    auto stage = [&](uint32_t tb, uint32_t buf) {
        const uint32_t nb = tb < a.rows ? min((uint32_t)BATCH, a.rows - tb) : 0u;
        float* q = qs + buf * BATCH * ROWF;
        float* k = ks + buf * BATCH * ROWF;
        for (uint32_t i = tid; i < nb * pieces; i += GD_WARPS * 32) {
            const uint32_t r = i / pieces, c = (i - r * pieces) * 4;
            gd_cp_async16(q + r * ROWF + c, pq + (size_t)(tb + r) * qk_stride + c);
            gd_cp_async16(k + r * ROWF + c, pk + (size_t)(tb + r) * qk_stride + c);
        }
        for (uint32_t i = tid; i < nb * CC; i += GD_WARPS * 32) {
            const uint32_t r = i / CC, c = i % CC;
            if (col0 + c < a.vdim) gd_cp_async4(vs + (buf * BATCH + r) * CC + c, pv + (size_t)(tb + r) * v_stride + c);
        }
        if (tid < nb) {
            gd_cp_async4(gs + buf * BATCH + tid, pg + (size_t)(tb + tid) * a.heads);
            gd_cp_async4(bs + buf * BATCH + tid, pb + (size_t)(tb + tid) * a.heads);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (dim4 < (uint32_t)ROWF) {                     // channels past the head stay zero in both buffers
        const uint32_t tail = ROWF - dim4;
        for (uint32_t i = tid; i < 2 * BATCH * tail; i += GD_WARPS * 32) {
            const uint32_t r = i / tail, c = dim4 + i % tail;
            qs[r * ROWF + c] = 0.0f;
            ks[r * ROWF + c] = 0.0f;
        }
    }
    stage(0, 0);
    gd_ring_store(a);
    float4 S[NV];
    float* state = reinterpret_cast<float*>(ga.state) + ((size_t)h * a.vdim + (col_ok ? col : 0u)) * dim4;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const uint32_t c = 4u * (i * L + part);
        S[i] = (col_ok && c < dim4) ? *reinterpret_cast<const float4*>(state + c) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    float* out = reinterpret_cast<float*>(ga.out) + (size_t)h * a.vdim + col;
    uint32_t buf = 0;
    for (uint32_t tb = 0; tb < a.rows; tb += BATCH, buf ^= 1) {
        const uint32_t nb = min((uint32_t)BATCH, a.rows - tb);
        stage(tb + BATCH, buf ^ 1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        const float* q = qs + buf * BATCH * ROWF + part * 4;
        const float* k = ks + buf * BATCH * ROWF + part * 4;
        const float* v = vs + buf * BATCH * CC + cl;
        const float* g = gs + buf * BATCH;
        const float* b = bs + buf * BATCH;
        auto load_row = [&](float4 (&x)[NV], const float* row) {
#pragma unroll
            for (int i = 0; i < NV; ++i) x[i] = *reinterpret_cast<const float4*>(row + i * L * 4);
        };
        uint32_t r0 = 0;
        for (; r0 + U <= nb; r0 += U) {              // U tokens in straight-line code: the next token's rows are read during this token's reduction
            float gr[U], bg[U], bv[U], o[U];
            float4 kc[NV], qc[NV], kn[NV], qn[NV];
            load_row(kc, k + r0 * ROWF);
            load_row(qc, q + r0 * ROWF);
#pragma unroll
            for (int j = 0; j < U; ++j) {
                const float beta = b[r0 + j];
                gr[j] = g[r0 + j];
                bg[j] = -beta * gr[j];
                bv[j] = beta * v[(r0 + j) * CC];
            }
#pragma unroll
            for (int j = 0; j < U; ++j) {
                if (j + 1 < U) {
                    load_row(kn, k + (r0 + j + 1) * ROWF);
                    load_row(qn, q + (r0 + j + 1) * ROWF);
                }
                const float z = gd_lane_sum<L>(gd_dot<NV>(S, kc));
                gd_update<NV>(S, kc, gr[j], fmaf(bg[j], z, bv[j]));
                o[j] = gd_dot<NV>(S, qc);
                if (j + 1 < U) {
#pragma unroll
                    for (int i = 0; i < NV; ++i) { kc[i] = kn[i]; qc[i] = qn[i]; }
                }
            }
            // the U read-outs meet over the lanes of a column all at once: at every level a lane keeps half of the values
            gd_transpose_sum<U, L>(o, part);
            if (col_ok && part % (L / U) == 0) out[(size_t)(tb + r0 + part / (L / U)) * v_stride] = o[0];
        }
        for (; r0 < nb; ++r0) {
            float4 k4[NV], q4[NV];
            load_row(k4, k + r0 * ROWF);
            load_row(q4, q + r0 * ROWF);
            const float gr = g[r0], beta = b[r0];
            const float z = gd_lane_sum<L>(gd_dot<NV>(S, k4));
            gd_update<NV>(S, k4, gr, fmaf(-beta * gr, z, beta * v[r0 * CC]));
            const float o = gd_lane_sum<L>(gd_dot<NV>(S, q4));
            if (part == 0 && col_ok) out[(size_t)(tb + r0) * v_stride] = o;
        }
        __syncthreads();
    }
    if (col_ok) {
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const uint32_t c = 4u * (i * L + part);
            if (c < dim4) *reinterpret_cast<float4*>(state + c) = S[i];
        }
    }
}

constexpr int GS_THREADS = 256;

// The same tokens four at a time, keys of 33..128 channels (column_block.cuh). With S the state at a block's start and p_j the product of the decays of
// its tokens before j, what token j writes is
//     w_j = beta_j v_j - beta_j g_j p_j (k_j . S) - sum_{i<j} beta_j g_j (g_{i+1} .. g_{j-1}) (k_j . k_i) w_i
//     o_j = p_{j+1} (q_j . S) + sum_{i<=j} (g_{i+1} .. g_j) (q_j . k_i) w_i,      S' = p_4 S + sum_i (g_{i+1} .. g_3) k_i w_i^T
// Producer warps (one per block) pass the q and k rows on, form the products k_j . k_i and q_j . k_i and invert the w_i system; consumer warps take the
// dot products with S, L lanes of four channels per group of Q columns. A decay is at most 1, so no product of them can grow.
// Bound: the chain dot products -> lane sums -> exchange -> update, 1200 cycles a block with one consumer warp per scheduler, which issues 420. 509 tokens, 16 heads of
// 128 x 128: 78 us against 96 us token by token.
template <int ROWF>
struct GdBlock {
    static constexpr int K = 0, R = 4 * ROWF, T = 8 * ROWF, C = T + 12, PO = C + 4, BETA = PO + 4, QS = BETA + 4, OW = QS + 8, V = OW + 16;
    static constexpr int floats(int columns) { return V + CB_TOKENS * columns; }
};

template <int L, int NV, int Q>
__global__ void __launch_bounds__(CB_THREADS, 2) gated_delta_block_kernel(const uzu_gated_delta_args ga) {
    constexpr int ROWF = L * NV * 4;
    using F = GdBlock<ROWF>;
    constexpr int GROUPS = 32 / L, CC = CB_WARPS * GROUPS * Q, U = CB_TOKENS * Q, SPAN = L / U, BLK = F::floats(CC);
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) float gd_smem[];
    float* wbuf = gd_smem + 2 * CB_BLOCKS * BLK;     // [2][CB_WARPS * GROUPS][U], twice each
    const uzu_delta_prepare_args& a = ga.prep;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t h = blockIdx.y, kvh = h / (a.heads / a.kv_heads), dim4 = (a.dim + 3) & ~3u, col0 = blockIdx.x * CC;
    const uint32_t steps = (a.rows + CB_BLOCKS * CB_TOKENS - 1) / (CB_BLOCKS * CB_TOKENS);
    const size_t qk_stride = (size_t)a.kv_heads * dim4, v_stride = (size_t)a.heads * a.vdim;
    gd_ring_store(a);

    if (warp >= CB_WARPS) {                          // producer of block `which` of every step
        const uint32_t which = warp - CB_WARPS, ch = 4 * lane;
        const bool ch_ok = ch < dim4;
        const float* pq = reinterpret_cast<const float*>(a.q) + (size_t)kvh * dim4 + ch;
        const float* pk = reinterpret_cast<const float*>(a.k) + (size_t)kvh * dim4 + ch;
        const float* pv = reinterpret_cast<const float*>(a.v) + (size_t)h * a.vdim + col0 + lane;
        const float* pg = reinterpret_cast<const float*>(a.decay) + h;
        const float* pb = reinterpret_cast<const float*>(a.beta) + h;
        cb_f4 q[CB_TOKENS], k[CB_TOKENS];
        float v[CB_TOKENS], g[CB_TOKENS], beta[CB_TOKENS];        // a token past the pass changes nothing: g = 1, the others 0
        auto fetch = [&](uint32_t step) {
            const uint32_t t0 = (step * CB_BLOCKS + which) * CB_TOKENS;
#pragma unroll
            for (int j = 0; j < CB_TOKENS; ++j) {
                const uint32_t t = t0 + j;
                const bool ok = t < a.rows;
                q[j] = ok && ch_ok ? cb_load4(pq + t * qk_stride) : cb_set4(0.0f);
                k[j] = ok && ch_ok ? cb_load4(pk + t * qk_stride) : cb_set4(0.0f);
                v[j] = ok && lane < CC && col0 + lane < a.vdim ? pv[t * v_stride] : 0.0f;
                g[j] = ok ? pg[(size_t)t * a.heads] : 1.0f;
                beta[j] = ok ? pb[(size_t)t * a.heads] : 0.0f;
            }
        };
        auto produce = [&](uint32_t step) {
            float* B = gd_smem + ((step & 1) * CB_BLOCKS + which) * BLK;
            if (ch < (uint32_t)ROWF) {
#pragma unroll
                for (int j = 0; j < CB_TOKENS; ++j) {
                    cb_store4(B + F::K + j * ROWF + ch, k[j]);
                    cb_store4(B + F::R + j * ROWF + ch, q[j]);
                }
            }
            float s[16];                             // [0, 6) k . k below the diagonal, [6, 16) q . k with it
#pragma unroll
            for (int j = 0; j < CB_TOKENS; ++j)
#pragma unroll
                for (int i = 0; i <= j; ++i) {
                    if (i < j) s[j * (j - 1) / 2 + i] = cb_dot(k[j], k[i]);
                    s[6 + j * (j + 1) / 2 + i] = cb_dot(q[j], k[i]);
                }
            gd_transpose_sum<16, 32>(s, lane);
            float n[6], t[6];
#pragma unroll
            for (int e = 0; e < 6; ++e) n[e] = __shfl_sync(0xffffffffu, s[0], 2 * e);
            const float g12 = g[1] * g[2], p3 = g[0] * g12;
            n[0] *= -beta[1] * g[1];
            n[1] *= -beta[2] * g12;
            n[2] *= -beta[2] * g[2];
            n[3] *= -beta[3] * (g12 * g[3]);
            n[4] *= -beta[3] * (g[2] * g[3]);
            n[5] *= -beta[3] * g[3];
            cb_invert(n, t);
            if (lane == 0) {
                cb_store_solve(B + F::T, t);
                const float p1 = g[0], p2 = g[0] * g[1], p4 = p3 * g[3];
                *reinterpret_cast<float4*>(B + F::PO) = make_float4(p1, p2, p3, p4);
                *reinterpret_cast<float4*>(B + F::C) = make_float4(-beta[0] * p1, -beta[1] * p2, -beta[2] * p3, -beta[3] * p4);
                *reinterpret_cast<float4*>(B + F::BETA) = make_float4(beta[0], beta[1], beta[2], beta[3]);
                const float q0 = g12 * g[3], q1 = g[2] * g[3];
                *reinterpret_cast<float4*>(B + F::QS) = make_float4(q0, q0, q1, q1);
                *reinterpret_cast<float4*>(B + F::QS + 4) = make_float4(g[3], g[3], p4, p4);
            } else if (lane >= 12 && (lane & 1) == 0) {
                uint32_t j, i;
                cb_lower(lane / 2 - 6, j, i);
                float f = 1.0f;                      // g_{i+1} .. g_j
#pragma unroll
                for (uint32_t l = 1; l < CB_TOKENS; ++l)
                    if (l > i && l <= j) f *= g[l];
                B[F::OW + j * 4 + i] = s[0] * f;
            }
            if (lane < CC) {
#pragma unroll
                for (int j = 0; j < CB_TOKENS; ++j) B[F::V + j * CC + lane] = v[j];
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
    const bool first = part % SPAN == 0, owner = first && col + oc < a.vdim;
    cb_f4 S[Q][NV];
    float* state = reinterpret_cast<float*>(ga.state) + ((size_t)h * a.vdim + col) * dim4 + ch;
#pragma unroll
    for (int c = 0; c < Q; ++c)
#pragma unroll
        for (int n = 0; n < NV; ++n) S[c][n] = col + c < a.vdim && ch + 4 * L * n < dim4 ? cb_load4(state + (size_t)c * dim4 + 4 * L * n) : cb_set4(0.0f);
    float* out = reinterpret_cast<float*>(ga.out) + (size_t)h * a.vdim + col + oc;
    for (uint32_t step = 0; step < steps; ++step) {
        __syncthreads();
        const uint32_t t_step = step * CB_BLOCKS * CB_TOKENS, nblocks = min((uint32_t)CB_BLOCKS, (a.rows - t_step + CB_TOKENS - 1) / CB_TOKENS);
        for (uint32_t b = 0; b < nblocks; ++b) {
            const float* B = gd_smem + ((step & 1) * CB_BLOCKS + b) * BLK;
            float* wb = wbuf + ((b & 1) * CB_WARPS * GROUPS + group) * U * 2;
            cb_f4 k[CB_TOKENS][NV], q[CB_TOKENS][NV];
#pragma unroll
            for (int j = 0; j < CB_TOKENS; ++j)
#pragma unroll
                for (int n = 0; n < NV; ++n) k[j][n] = cb_load4(B + F::K + j * ROWF + ch + 4 * L * n);
#pragma unroll
            for (int j = 0; j < CB_TOKENS; ++j)
#pragma unroll
                for (int n = 0; n < NV; ++n) q[j][n] = cb_load4(B + F::R + j * ROWF + ch + 4 * L * n);
            float zp[U], op[U];
            cb_dots<NV, Q>(zp, k, S);
            const float bv = B[F::BETA + oj] * B[F::V + oj * CC + lc + oc], cj = B[F::C + oj], po = B[F::PO + oj];
            const cb_f4 qs0 = cb_load4(B + F::QS), qs1 = cb_load4(B + F::QS + 4);
            gd_transpose_sum<U, L>(zp, part);
            if (first) {
                const float r = fmaf(cj, zp[0], bv);
                *reinterpret_cast<float2*>(wb + 2 * idx) = make_float2(r, r);
            }
            __syncwarp();                            // the buffer's next writer is two blocks on, behind another one of these
            cb_dots<NV, Q>(op, q, S);
#pragma unroll
            for (int c = 0; c < Q; ++c)
#pragma unroll
                for (int n = 0; n < NV; ++n) S[c][n] = cb_scale(S[c][n], qs1.b);
            cb_f2 w[CB_TOKENS][Q], y[CB_TOKENS][Q];
#pragma unroll
            for (int j = 0; j < CB_TOKENS; ++j) cb_load<Q>(y[j], wb + 2 * j * Q);
            cb_solve<Q>(w, y, B + F::T);
#pragma unroll
            for (int c = 0; c < Q; ++c) {            // the last token's write has decayed by nothing
                y[0][c] = cb_mul2(w[0][c], qs0.a);
                y[1][c] = cb_mul2(w[1][c], qs0.b);
                y[2][c] = cb_mul2(w[2][c], qs1.a);
                y[3][c] = w[3][c];
            }
            cb_update<NV, Q>(S, k, y);
            gd_transpose_sum<U, L>(op, part);
            float wown[CB_TOKENS];
#pragma unroll
            for (int j = 0; j < CB_TOKENS; ++j) wown[j] = cb_pick<Q>(w[j], oc);
            // up to the token itself: a later token's value reaches no earlier one, not even as 0 * x
            const float o = cb_upto(po * op[0], *reinterpret_cast<const float4*>(B + F::OW + oj * 4), wown, oj + 1);
            const uint32_t t = t_step + b * CB_TOKENS + oj;
            if (owner && t < a.rows) out[t * v_stride] = o;
        }
    }
#pragma unroll
    for (int c = 0; c < Q; ++c)
#pragma unroll
        for (int n = 0; n < NV; ++n)
            if (col + c < a.vdim && ch + 4 * L * n < dim4) cb_store4(state + (size_t)c * dim4 + 4 * L * n, S[c][n]);
}

// CL CTAs (one cluster) per head, ceil(vdim / CL) columns each, GS_THREADS / L columns at a time
template <int CL, int L, int NV>
__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(GS_THREADS) gated_delta_step_kernel(const uzu_gated_delta_step_args sa) {
    constexpr int ROWF = L * NV * 4, CPP = GS_THREADS / L;
    extern __shared__ __align__(16) float gd_smem[];
    __shared__ float red_q[GS_THREADS / 32], red_k[GS_THREADS / 32], red_o[32], ss_parts[CL];
    const uzu_delta_prepare_args& a = sa.prep;
    pdl_launch_dependents();
    if constexpr (CL > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");     // "this CTA runs": awaited before the first remote store
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, part = tid % L;
    const uint32_t h = blockIdx.x / CL, rank = blockIdx.x % CL, group = a.heads / a.kv_heads, kvh = h / group;
    const uint32_t per = (a.vdim + CL - 1) / CL, col0 = min(a.vdim, rank * per), ncols = min(a.vdim, col0 + per) - col0;
    const uint32_t kd = a.kv_heads * a.dim, channels = 2 * kd + a.heads * a.vdim, dim4 = (a.dim + 3) & ~3u;
    float* qs = gd_smem;             // [ROWF]
    float* ks = qs + ROWF;           // [ROWF]
    float* vs = ks + ROWF;           // [per]
    float* os = vs + per;            // [per]
    float* state = reinterpret_cast<float*>(sa.state) + ((size_t)h * a.vdim + col0) * dim4;
    float4 S[NV];
    auto load_state = [&](uint32_t cl) {
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const uint32_t c = 4u * (i * L + part);
            S[i] = (cl < ncols && c < dim4) ? *reinterpret_cast<const float4*>(state + (size_t)cl * dim4 + c) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
    };
    load_state(tid / L);             // nothing in front of this kernel writes the state or the ring: requested before the wait
    // ... and so is what the convolution takes from earlier tokens: all but the last tap
    const uint32_t prefix = gd_prefix(a), v0 = 2 * kd + h * a.vdim + col0;
    constexpr int QK = (2 * ROWF + GS_THREADS - 1) / GS_THREADS;      // q / k channels of a thread
    float qk_past[QK], qk_tap[QK], v_past = 0.0f, v_tap = 0.0f;
    auto qk_channel = [&](uint32_t i) { return (i < ROWF ? 0u : kd - ROWF) + kvh * a.dim + i; };      // (i counts q channels, then k channels)
    auto in_head = [&](uint32_t i) { return i < 2 * ROWF && (i < ROWF ? i : i - ROWF) < a.dim; };
#pragma unroll
    for (int u = 0; u < QK; ++u) {
        const uint32_t i = tid + u * GS_THREADS;
        qk_past[u] = qk_tap[u] = 0.0f;
        if (in_head(i)) gd_conv_past(a, channels, prefix, qk_channel(i), qk_past[u], qk_tap[u]);
    }
    if (tid < ncols) gd_conv_past(a, channels, prefix, v0 + tid, v_past, v_tap);
    const float a_log = reinterpret_cast<const float*>(a.a_log)[h], dt_bias = reinterpret_cast<const float*>(a.dt_bias)[h];
    const float norm0 = tid < ncols ? reinterpret_cast<const float*>(sa.norm)[(size_t)h * a.vdim + col0 + tid] : 0.0f;
    pdl_wait();
    const float* proj = reinterpret_cast<const float*>(a.proj);
    const float* gate = proj + sa.gate_offset + (size_t)h * a.vdim + col0;
    const float gate0 = tid < ncols ? gate[tid] : 0.0f;
    float* ring = reinterpret_cast<float*>(a.ring) + (size_t)(prefix % a.taps) * channels;        // the slot of this token: nobody reads it here
    float sq = 0.0f, sk = 0.0f;
#pragma unroll
    for (int u = 0; u < QK; ++u) {
        const uint32_t i = tid + u * GS_THREADS;
        float y = 0.0f;
        if (in_head(i)) {
            const float x = proj[qk_channel(i)];
            y = gd_silu(fmaf(qk_tap[u], x, qk_past[u]));
            if (rank == 0 && h % group == 0 && a.taps > 1) ring[qk_channel(i)] = x;
        }
        if (i < 2 * ROWF) qs[i] = y;                                     // ks follows qs
        if (i < ROWF) sq = fmaf(y, y, sq);
        else sk = fmaf(y, y, sk);
    }
    for (uint32_t i = tid; i < ncols; i += GS_THREADS) {
        if (i >= GS_THREADS) gd_conv_past(a, channels, prefix, v0 + i, v_past, v_tap);
        const float x = proj[v0 + i];
        vs[i] = gd_silu(fmaf(v_tap, x, v_past));
        if (a.taps > 1) ring[v0 + i] = x;
    }
    const float g = gd_decay(a_log, proj[a.a_offset + h] + dt_bias);
    const float beta = gd_sigmoid(proj[a.b_offset + h]);
    sq = warp_sum(sq);
    sk = warp_sum(sk);
    if (lane == 0) { red_q[warp] = sq; red_k[warp] = sk; }
    __syncthreads();
    float tq = 0.0f, tk = 0.0f;
#pragma unroll
    for (int w = 0; w < GS_THREADS / 32; ++w) { tq += red_q[w]; tk += red_k[w]; }
    const float fq = (1.0f / sqrtf(tq + kUnitEps)) * (1.0f / sqrtf((float)a.dim)), fk = 1.0f / sqrtf(tk + kUnitEps);
    float4 q4[NV], k4[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const float4 q = *reinterpret_cast<const float4*>(qs + 4 * (i * L + part)), k = *reinterpret_cast<const float4*>(ks + 4 * (i * L + part));
        q4[i] = make_float4(q.x * fq, q.y * fq, q.z * fq, q.w * fq);
        k4[i] = make_float4(k.x * fk, k.y * fk, k.z * fk, k.w * fk);
    }
    for (uint32_t cb = 0; cb < ncols; cb += CPP) {
        const uint32_t cl = cb + tid / L;
        if (cb) load_state(cl);
        const float z = gd_lane_sum<L>(gd_dot<NV>(S, k4));
        const float u = beta * ((cl < ncols ? vs[cl] : 0.0f) - g * z);
        gd_update<NV>(S, k4, g, u);
        const float o = gd_lane_sum<L>(gd_dot<NV>(S, q4));
        if (cl < ncols) {
            if (part == 0) os[cl] = o;
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                const uint32_t c = 4u * (i * L + part);
                if (c < dim4) *reinterpret_cast<float4*>(state + (size_t)cl * dim4 + c) = S[i];
            }
        }
    }
    __syncthreads();
    float ss = 0.0f;
    for (uint32_t i = tid; i < ncols; i += GS_THREADS) ss = fmaf(os[i], os[i], ss);
    ss = block_sum(ss, red_o);
    if constexpr (CL > 1) {
        asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
        if (tid < CL) {
            const uint32_t local = (uint32_t)__cvta_generic_to_shared(&ss_parts[rank]);
            uint32_t remote;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(tid));
            asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(remote), "f"(ss) : "memory");
        }
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        ss = 0.0f;
#pragma unroll
        for (int c = 0; c < CL; ++c) ss += ss_parts[c];
    }
    const float inv = 1.0f / sqrtf(ss / (float)a.vdim + sa.epsilon);
    float* out = reinterpret_cast<float*>(sa.out) + (size_t)h * a.vdim + col0;
    if (tid < ncols) out[tid] = os[tid] * inv * norm0 * gd_silu(gate0);
    const float* norm = reinterpret_cast<const float*>(sa.norm) + (size_t)h * a.vdim + col0;
    for (uint32_t i = tid + GS_THREADS; i < ncols; i += GS_THREADS) out[i] = os[i] * inv * norm[i] * gd_silu(gate[i]);
}

static const char* delta_prepare_check(const uzu_delta_prepare_args& a, bool scratch) {
    if (!a.proj || !a.conv || !a.ring || !a.a_log || !a.dt_bias || (scratch && (!a.q || !a.k || !a.v || !a.decay || !a.beta))) return "null operand";
    if (a.heads == 0 || a.kv_heads == 0 || a.heads % a.kv_heads || a.dim == 0 || a.dim > 1024 || a.vdim == 0 || a.vdim > 4096 || a.taps == 0)
        return "kv_heads must divide heads, dim must be in 1..1024, vdim in 1..4096, taps positive";
    if (scratch && ((a.q & 15) || (a.k & 15))) return "the q / k rows must be 16-byte aligned";
    const uint64_t channels = 2ull * a.kv_heads * a.dim + (uint64_t)a.heads * a.vdim;
    if (a.stride < channels || a.a_offset + a.heads > a.stride || a.b_offset + a.heads > a.stride) return "a projection row is shorter than its parts";
    return nullptr;
}

// lanes per value column and float4 of key channels per lane, by head size
template <typename F>
static void by_key_size(uint32_t dim, F&& f) {
    if (dim <= 32) f(std::integral_constant<int, 8>{}, std::integral_constant<int, 1>{});
    else if (dim <= 64) f(std::integral_constant<int, 8>{}, std::integral_constant<int, 2>{});
    else if (dim <= 128) f(std::integral_constant<int, 8>{}, std::integral_constant<int, 4>{});
    else if (dim <= 256) f(std::integral_constant<int, 16>{}, std::integral_constant<int, 4>{});
    else if (dim <= 512) f(std::integral_constant<int, 32>{}, std::integral_constant<int, 4>{});
    else f(std::integral_constant<int, 32>{}, std::integral_constant<int, 8>{});
}

// Blocks of four tokens for keys of 33..128 channels from the pass length on at which they are no slower. One column per lane group while such CTAs have an SM
// each (8 heads of 128 x 128, 1024 tokens: 105 us, 144 with two columns); more of them share an SM's issue slots and shared memory, and two columns per
// lane group are faster in half the CTAs (16 heads 144 us, 158 with one). Token by token / blocks, us: one column, 8 heads of 128, 3 tokens 4.8 / 5.2, 12 tokens
// 6.3 / 6.3, 24 tokens 8.4 / 7.3; two columns, 16 heads of 128, 2 tokens 4.2 / 6.3, 16 tokens 6.8 / 7.2, 36 tokens 11.3 / 10.4; 32 heads of 128, 9 tokens 6.4 / 8.3, 33 tokens
// 12.5 / 13.4, 36 tokens 14.1 / 13.5.
void launch_gated_delta_scan(uzu_command_buffer* cmd, const uzu_gated_delta_args& a) {
    const bool one_column = a.prep.heads * ((a.prep.vdim + 7) / 8) <= (uint32_t)cmd->ctx->sm_count;
    if (a.prep.dim > 32 && a.prep.dim <= 128 && a.prep.rows >= (one_column ? 12u : 36u)) {
        auto blocks = [&](auto nv_c, auto q_c) {
            constexpr int L = 16, NV = decltype(nv_c)::value, Q = decltype(q_c)::value, GROUPS = CB_WARPS * (32 / L), CC = GROUPS * Q;
            constexpr size_t smem = ((size_t)2 * CB_BLOCKS * GdBlock<L * NV * 4>::floats(CC) + (size_t)4 * GROUPS * CB_TOKENS * Q) * sizeof(float);
            static std::atomic<uint64_t> done{0};
            if (smem > 48 * 1024) opt_in_dynamic_smem(cmd, gated_delta_block_kernel<L, NV, Q>, (int)smem, done);
            launch(cmd, "gated_delta_kernel", gated_delta_block_kernel<L, NV, Q>, dim3((a.prep.vdim + CC - 1) / CC, a.prep.heads), dim3(CB_THREADS), smem, a);
        };
        auto one = std::integral_constant<int, 1>{};
        auto two = std::integral_constant<int, 2>{};
        if (a.prep.dim <= 64) one_column ? blocks(one, one) : blocks(one, two);
        else one_column ? blocks(two, one) : blocks(two, two);
        return;
    }
    by_key_size(a.prep.dim, [&](auto l_c, auto nv_c) {
        constexpr int L = decltype(l_c)::value, NV = decltype(nv_c)::value, CC = GD_WARPS * (32 / L), BATCH = gd_batch<L, NV>();
        constexpr size_t smem = ((size_t)4 * BATCH * L * NV * 4 + (size_t)2 * BATCH * CC + 4 * BATCH) * sizeof(float);
        static std::atomic<uint64_t> done{0};
        if (smem > 48 * 1024) opt_in_dynamic_smem(cmd, gated_delta_kernel<L, NV>, (int)smem, done);
        launch(cmd, "gated_delta_kernel", gated_delta_kernel<L, NV>, dim3((a.prep.vdim + CC - 1) / CC, a.prep.heads), dim3(GD_WARPS * 32), smem, a);
    });
}

}  // namespace uzu

extern "C" {
using namespace uzu;

void uzu_delta_prepare_encode(uzu_command_buffer* cmd, const uzu_delta_prepare_args* a) {
    if (!encodable(cmd, "delta_prepare")) return;
    if (const char* err = delta_prepare_check(*a, true)) {
        cmd->record_error(UZU_ERROR_INVALID_ARGUMENT, std::string("delta_prepare: ") + err);
        return;
    }
    if (a->rows == 0) return;
    const uint32_t units = 2 * a->kv_heads + a->heads + 1, widest = std::max(a->dim, a->vdim);
    if (a->rows >= 4 && a->taps >= 2 && a->taps <= 4 && widest <= 256) {
        const uint32_t blocks = (a->rows + GP_ROWS - 1) / GP_ROWS;
        auto go = [&](auto kernel) { launch(cmd, "delta_prepare_kernel", kernel, dim3((blocks * units + 3) / 4), dim3(128), 0, *a); };
        auto by_width = [&](auto taps_c) {
            constexpr int T = decltype(taps_c)::value;
            if (widest <= 32) go(delta_prepare_window_kernel<T, 1>);
            else if (widest <= 64) go(delta_prepare_window_kernel<T, 2>);
            else if (widest <= 128) go(delta_prepare_window_kernel<T, 4>);
            else go(delta_prepare_window_kernel<T, 8>);
        };
        if (a->taps == 2) by_width(std::integral_constant<int, 2>{});
        else if (a->taps == 3) by_width(std::integral_constant<int, 3>{});
        else by_width(std::integral_constant<int, 4>{});
        return;
    }
    const uint32_t items = a->rows * units;
    launch(cmd, "delta_prepare_kernel", delta_prepare_kernel, dim3((items + 3) / 4), dim3(128), 0, *a);
}

void uzu_gated_delta_encode(uzu_command_buffer* cmd, const uzu_gated_delta_args* a) {
    if (!encodable(cmd, "gated_delta")) return;
    const char* err = delta_prepare_check(a->prep, true);
    if (!err && (!a->state || !a->out || (a->state & 15))) err = "null or unaligned state, or null output";
    if (err) {
        cmd->record_error(UZU_ERROR_INVALID_ARGUMENT, std::string("gated_delta: ") + err);
        return;
    }
    if (a->prep.rows == 0) return;
    launch_gated_delta_scan(cmd, *a);
}

void uzu_gated_delta_step_encode(uzu_command_buffer* cmd, const uzu_gated_delta_step_args* a) {
    if (!encodable(cmd, "gated_delta_step")) return;
    const char* err = delta_prepare_check(a->prep, false);
    if (!err && (!a->state || !a->out || !a->norm || (a->state & 15))) err = "null operand or unaligned state";
    if (!err && a->prep.rows != 1) err = "one token per launch";
    if (!err && (uint64_t)a->gate_offset + (uint64_t)a->prep.heads * a->prep.vdim > a->prep.stride) err = "a projection row is shorter than its parts";
    if (err) {
        cmd->record_error(UZU_ERROR_INVALID_ARGUMENT, std::string("gated_delta_step: ") + err);
        return;
    }
    by_key_size(a->prep.dim, [&](auto l_c, auto nv_c) {
        constexpr int L = decltype(l_c)::value, NV = decltype(nv_c)::value;
        auto go = [&](auto cl_c) {
            constexpr int CL = decltype(cl_c)::value;
            const size_t smem = ((size_t)2 * L * NV * 4 + (size_t)2 * ((a->prep.vdim + CL - 1) / CL)) * sizeof(float);
            launch(cmd, "gated_delta_step_kernel", gated_delta_step_kernel<CL, L, NV>, dim3(a->prep.heads * CL), dim3(GS_THREADS), smem, *a);
        };
        // one pass over a CTA's columns where a cluster of four can do that; a head of few columns needs no cluster
        if (a->prep.vdim > (uint32_t)(GS_THREADS / L)) go(std::integral_constant<int, 4>{});
        else go(std::integral_constant<int, 1>{});
    });
}

}  // extern "C"
