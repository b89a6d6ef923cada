// DeltaNet prefill: the decode recurrence (DeltaNetConvUpdate + DeltaNetUpdate, backends/cpu/kernel/gdn/{conv_update.rs:8-55,
// update.rs:13-144}) applied to the m tokens of a pass, in three launches whatever m is:
//   delta_net_conv_kernel    causal conv + SiLU (bf16-rounded, like the conv kernel), unit q and k vectors, q scaled by Dk^-0.5, decay and
//                            beta of all tokens at once into f32 scratch rows (a warp per 8 tokens and head, the conv window in registers);
//   the gated delta scan     (gated_delta.cu) a value column of the state needs no other column, so a few lanes own one and walk the tokens,
//                            four at a time; 128 CTAs for 16 heads of 128 columns;
//   delta_net_gate_kernel    RMS norm of each head's row, norm weight, SiLU(z), bf16 store; the rolling conv state moves on here, when all
//                            readers of the old one are done.
// Bound: latency of the scan (one warp per scheduler walks the tokens, nothing covers its waits), not bytes. As ONE CTA per
// head with the state in shared memory and ten barriers per token a 509-token pass of 16 heads took 2.87 ms per layer; an 8-layer prompt
// (6 such layers) 17.7 ms, 3.05 ms now.
// Same formulas and rounding points as the single-token kernels (this file is built with -fmad=false like deltanet.cu); sums run in another
// order, so parity with the oracle's sequential sums is at tolerance level, as for the decode kernel.
// Requires head_k_dim = 128, head_v_dim <= 128, <= 7 conv taps. Passes of 2 and 3 tokens keep the one-launch kernel below (a CTA per head,
// about 6 us a token: three launches cost as much), where every k head has one v head.
#include <cstdlib>

#include "common.cuh"

namespace uzu {

constexpr int DP_THREADS = 256;
constexpr int DP_DK = 128;
constexpr int DP_MAX_TAPS = 7;

struct DeltaPrefillParams {
    uzu_delta_net_fused_update_args f;   // per-token arguments; update.in_proj / update.out / conv.in_out point at row 0
    uint32_t rows;                       // tokens
    uint32_t in_stride, out_stride;      // elements between consecutive rows of the projection / the output
};

__device__ __forceinline__ float dp_block_sum(float v, float* red, int nwarps) {
    v = warp_sum(v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    float t = 0.0f;
    for (int w = 0; w < nwarps; ++w) t += red[w];     // fixed order: every thread gets the same bits
    return t;
}

__global__ void __launch_bounds__(DP_THREADS) delta_net_prefill_kernel(const DeltaPrefillParams p) {
    extern __shared__ __align__(16) float dp_smem[];
    const uzu_delta_net_update_args& a = p.f.update;
    const uzu_delta_net_conv_update_args& c = p.f.conv;
    const uint32_t DV = a.head_v_dim;
    float* S = dp_smem;                        // [DV][128]
    float* sq = S + (size_t)DV * DP_DK;        // [128]
    float* sk = sq + DP_DK;                    // [128]
    float* sv = sk + DP_DK;                    // [128]
    float* so = sv + DP_DK;                    // [128]
    float* red = so + DP_DK;                   // [8]

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t hv = blockIdx.x, hk = hv;   // num_v_heads == num_k_heads
    const uint32_t conv_dim = 2 * a.key_dim + a.value_dim;
    const uint32_t taps = c.kernel_size - 1;
    float* gstate = reinterpret_cast<float*>(a.state) + (size_t)hv * DV * DP_DK;

    // recurrent state -> shared memory
    for (uint32_t i = tid; i < DV * DP_DK / 4; i += DP_THREADS) reinterpret_cast<float4*>(S)[i] = reinterpret_cast<const float4*>(gstate)[i];

    // conv channels of this thread: threads 0..127 own q_j and k_j (j = tid), threads 128..255 own v_i (i = tid - 128)
    const bool qk_thread = tid < DP_DK, v_thread = tid >= DP_DK && (uint32_t)(tid - DP_DK) < DV;
    const uint32_t ch0 = qk_thread ? hk * DP_DK + tid : 2 * a.key_dim + hv * DV + (tid - DP_DK);   // q channel or v channel
    const uint32_t ch1 = a.key_dim + hk * DP_DK + tid;                                               // k channel (q/k threads)
    float w0[DP_MAX_TAPS + 1], w1[DP_MAX_TAPS + 1], st0[DP_MAX_TAPS], st1[DP_MAX_TAPS];
    float b0 = 0.0f, b1 = 0.0f;
    const float* cw = reinterpret_cast<const float*>(c.conv_weight);
    float* cs = reinterpret_cast<float*>(c.state);
#pragma unroll
    for (int t = 0; t <= DP_MAX_TAPS; ++t) {
        w0[t] = w1[t] = 0.0f;
        if (t < DP_MAX_TAPS) st0[t] = st1[t] = 0.0f;
    }
    if (qk_thread || v_thread) {
#pragma unroll
        for (int t = 0; t <= DP_MAX_TAPS; ++t)
            if ((uint32_t)t <= taps) w0[t] = cw[(size_t)ch0 * c.kernel_size + t];
#pragma unroll
        for (int t = 0; t < DP_MAX_TAPS; ++t)
            if ((uint32_t)t < taps) st0[t] = cs[(size_t)ch0 * c.state_stride + t];
        if (c.has_bias) b0 = reinterpret_cast<const float*>(c.bias)[ch0];
    }
    if (qk_thread) {
#pragma unroll
        for (int t = 0; t <= DP_MAX_TAPS; ++t)
            if ((uint32_t)t <= taps) w1[t] = cw[(size_t)ch1 * c.kernel_size + t];
#pragma unroll
        for (int t = 0; t < DP_MAX_TAPS; ++t)
            if ((uint32_t)t < taps) st1[t] = cs[(size_t)ch1 * c.state_stride + t];
        if (c.has_bias) b1 = reinterpret_cast<const float*>(c.bias)[ch1];
    }
    // one conv step (conv_update.rs:25-54): acc = bias + sum_t state[t]*w[t] + x*w[taps]; out = bf16(SiLU(acc)); state shifts in x
    auto conv_step = [&](float x, const float (&w)[DP_MAX_TAPS + 1], float (&st)[DP_MAX_TAPS], float bias) {
        float acc = bias;
#pragma unroll
        for (int t = 0; t < DP_MAX_TAPS; ++t)
            if ((uint32_t)t < taps) acc += st[t] * w[t];
        float wl = 0.0f;
#pragma unroll
        for (int t = 0; t <= DP_MAX_TAPS; ++t)
            if ((uint32_t)t == taps) wl = w[t];
        acc += x * wl;
#pragma unroll
        for (int t = 0; t < DP_MAX_TAPS - 1; ++t)
            if ((uint32_t)(t + 1) < taps) st[t] = st[t + 1];
#pragma unroll
        for (int t = 0; t < DP_MAX_TAPS; ++t)
            if ((uint32_t)t == taps - 1) st[t] = x;
        return bf2f(f2bf(act_f32(UZU_ACT_SILU, acc)));
    };

    const float a_log = reinterpret_cast<const float*>(a.a_log)[hv], dt_bias = reinterpret_cast<const float*>(a.dt_bias)[hv];
    const float nw = tid < (int)DV ? reinterpret_cast<const float*>(a.norm_weight)[tid] : 0.0f;
    const float qscale = 1.0f / sqrtf((float)DP_DK);
    __syncthreads();

    for (uint32_t t = 0; t < p.rows; ++t) {
        const __nv_bfloat16* row = reinterpret_cast<const __nv_bfloat16*>(a.in_proj) + (size_t)t * p.in_stride;
        // ---- 1. conv + SiLU ----
        float qv = 0.0f, kv = 0.0f;
        if (qk_thread) {
            qv = conv_step(bf2f(row[ch0]), w0, st0, b0);
            kv = conv_step(bf2f(row[ch1]), w1, st1, b1);
        } else if (v_thread) {
            sv[tid - DP_DK] = conv_step(bf2f(row[ch0]), w0, st0, b0);
        }
        // ---- 2. q / k normalisation, k.q, gate scalars (update.rs:60-95) ----
        const float qn = dp_block_sum(qv * qv, red, DP_THREADS / 32);
        const float kn = dp_block_sum(kv * kv, red, DP_THREADS / 32);
        const float qi = 1.0f / sqrtf(qn + 1e-6f), ki = 1.0f / sqrtf(kn + 1e-6f);
        float qq = 0.0f, kk = 0.0f;
        if (qk_thread) {
            qq = qv * qi;
            qq = qq * qscale;
            kk = kv * ki;
            sq[tid] = qq;
            sk[tid] = kk;
        }
        const float kq = dp_block_sum(kk * qq, red, DP_THREADS / 32);     // also orders the sq / sk / sv writes before the reads below
        const float beta_raw = bf2f(row[conv_dim + a.value_dim + hv]);
        const float beta = 1.0f / (1.0f + expf(-beta_raw));
        const float a_raw = bf2f(row[conv_dim + a.value_dim + a.num_v_heads + hv]);
        const float sp_in = a_raw + dt_bias;
        const float sp = sp_in > 20.0f ? sp_in : logf(1.0f + expf(sp_in));
        const float decay = expf(-expf(a_log) * sp);
        // ---- 3. state update, one warp per row ----
        const float4 q4 = *reinterpret_cast<const float4*>(&sq[lane * 4]);
        const float4 k4 = *reinterpret_cast<const float4*>(&sk[lane * 4]);
        for (uint32_t i = warp; i < DV; i += DP_THREADS / 32) {
            float4* srow = reinterpret_cast<float4*>(S + (size_t)i * DP_DK) + lane;
            const float4 s = *srow;
            float sqa = s.x * q4.x + s.y * q4.y + s.z * q4.z + s.w * q4.w;
            float ska = s.x * k4.x + s.y * k4.y + s.z * k4.z + s.w * k4.w;
            sqa = warp_sum(sqa);
            ska = warp_sum(ska);
            const float retrieved = decay * ska;
            const float delta = beta * (sv[i] - retrieved);
            if (lane == 0) so[i] = decay * sqa + delta * kq;
            float4 ns;
            ns.x = decay * s.x + k4.x * delta;
            ns.y = decay * s.y + k4.y * delta;
            ns.z = decay * s.z + k4.z * delta;
            ns.w = decay * s.w + k4.w * delta;
            *srow = ns;
        }
        __syncthreads();
        // ---- 4. RMS norm * norm_weight * SiLU(z) (update.rs:120-143) ----
        const float ov = tid < (int)DV ? so[tid] : 0.0f;
        const float ss = dp_block_sum(ov * ov, red, DP_THREADS / 32);
        const float inv_rms = 1.0f / sqrtf(ss / (float)DV + a.norm_epsilon);
        if (tid < (int)DV) {
            const float z = bf2f(row[conv_dim + hv * DV + tid]);
            const float zs = act_f32(UZU_ACT_SILU, z);
            reinterpret_cast<__nv_bfloat16*>(a.out)[(size_t)t * p.out_stride + hv * DV + tid] = f2bf(ov * inv_rms * nw * zs);
        }
        __syncthreads();                                        // so / sv / sq / sk are rewritten by the next token
    }

    // state and rolling conv state back to global memory
    for (uint32_t i = tid; i < DV * DP_DK / 4; i += DP_THREADS) reinterpret_cast<float4*>(gstate)[i] = reinterpret_cast<const float4*>(S)[i];
    if (qk_thread || v_thread) {
#pragma unroll
        for (int t = 0; t < DP_MAX_TAPS; ++t)
            if ((uint32_t)t < taps) cs[(size_t)ch0 * c.state_stride + t] = st0[t];
    }
    if (qk_thread) {
#pragma unroll
        for (int t = 0; t < DP_MAX_TAPS; ++t)
            if ((uint32_t)t < taps) cs[(size_t)ch1 * c.state_stride + t] = st1[t];
    }
}

// ---- four tokens and more ------------------------------------------------------------------------------------------------------------
struct DeltaScanParams {
    DeltaPrefillParams p;
    float *q, *k, *v, *o, *decay, *beta;   // f32 rows [rows, key_dim] x 2, [rows, value_dim] x 2, [rows, num_v_heads] x 2
};
constexpr int DP_BLOCK = 8;                // tokens per warp: an input is read once per block, plus the window before it

// units: q heads, k heads, v heads, then one for the gates
template <int TAPS>
__global__ void __launch_bounds__(128) delta_net_conv_kernel(const DeltaScanParams s) {
    pdl_launch_dependents();
    pdl_wait();
    const uzu_delta_net_update_args& a = s.p.f.update;
    const uzu_delta_net_conv_update_args& c = s.p.f.conv;
    const uint32_t lane = threadIdx.x & 31, rows = s.p.rows;
    const uint32_t units = 2 * a.num_k_heads + a.num_v_heads + 1, blocks = (rows + DP_BLOCK - 1) / DP_BLOCK;
    const uint32_t item = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (item >= blocks * units) return;
    const uint32_t t0 = item / units * DP_BLOCK, unit = item % units, nr = min((uint32_t)DP_BLOCK, rows - t0);
    const __nv_bfloat16* in = reinterpret_cast<const __nv_bfloat16*>(a.in_proj);
    const uint32_t conv_dim = 2 * a.key_dim + a.value_dim;
    if (unit == units - 1) {
        for (uint32_t i = lane; i < nr * a.num_v_heads; i += 32) {
            const uint32_t t = t0 + i / a.num_v_heads, h = i % a.num_v_heads;
            const __nv_bfloat16* row = in + (size_t)t * s.p.in_stride + conv_dim + a.value_dim;
            const float sp_in = bf2f(row[a.num_v_heads + h]) + reinterpret_cast<const float*>(a.dt_bias)[h];
            const float sp = sp_in > 20.0f ? sp_in : logf(1.0f + expf(sp_in));
            s.decay[(size_t)t * a.num_v_heads + h] = expf(-expf(reinterpret_cast<const float*>(a.a_log)[h]) * sp);
            s.beta[(size_t)t * a.num_v_heads + h] = 1.0f / (1.0f + expf(-bf2f(row[h])));
        }
        return;
    }
    const bool is_q = unit < a.num_k_heads, is_v = unit >= 2 * a.num_k_heads;
    const uint32_t head = is_q ? unit : (is_v ? unit - 2 * a.num_k_heads : unit - a.num_k_heads);
    const uint32_t width = is_v ? a.head_v_dim : DP_DK, ch0 = (is_q ? 0u : is_v ? 2 * a.key_dim : a.key_dim) + head * width;
    float* out = (is_q ? s.q : is_v ? s.v : s.k) + (size_t)t0 * (is_v ? a.value_dim : a.key_dim) + head * width;
    const uint32_t out_stride = is_v ? a.value_dim : a.key_dim;
    constexpr int NC = DP_DK / 32;
    float w[NC][TAPS + 1], x[NC][TAPS], bias[NC];
#pragma unroll
    for (int i = 0; i < NC; ++i) {
        const uint32_t ci = lane + 32u * i, ch = ch0 + ci;
        const bool ok = ci < width;
        bias[i] = ok && c.has_bias ? reinterpret_cast<const float*>(c.bias)[ch] : 0.0f;
#pragma unroll
        for (int j = 0; j <= TAPS; ++j) w[i][j] = ok ? reinterpret_cast<const float*>(c.conv_weight)[(size_t)ch * (TAPS + 1) + j] : 0.0f;
#pragma unroll
        for (int j = 0; j < TAPS; ++j) {              // input of token t0 - TAPS + j: from the pass, or from the rolling state before it
            const uint32_t t = t0 + j;
            x[i][j] = !ok ? 0.0f : t >= (uint32_t)TAPS ? bf2f(in[(size_t)(t - TAPS) * s.p.in_stride + ch])
                                                       : reinterpret_cast<const float*>(c.state)[(size_t)ch * c.state_stride + t];
        }
    }
    for (uint32_t r = 0; r < nr; ++r) {
        float y[NC], ss = 0.0f;
#pragma unroll
        for (int i = 0; i < NC; ++i) {
            const uint32_t ci = lane + 32u * i;
            const float now = ci < width ? bf2f(in[(size_t)(t0 + r) * s.p.in_stride + ch0 + ci]) : 0.0f;
            float acc = bias[i];
#pragma unroll
            for (int j = 0; j < TAPS; ++j) acc += x[i][j] * w[i][j];
            acc += now * w[i][TAPS];
#pragma unroll
            for (int j = 0; j + 1 < TAPS; ++j) x[i][j] = x[i][j + 1];
            x[i][TAPS - 1] = now;
            y[i] = bf2f(f2bf(act_f32(UZU_ACT_SILU, acc)));
            ss += y[i] * y[i];
        }
        float f = 1.0f, g = 1.0f;
        if (!is_v) {
            f = 1.0f / sqrtf(warp_sum(ss) + 1e-6f);
            if (is_q) g = 1.0f / sqrtf((float)DP_DK);
        }
#pragma unroll
        for (int i = 0; i < NC; ++i) {
            const uint32_t ci = lane + 32u * i;
            if (ci < width) out[(size_t)r * out_stride + ci] = y[i] * f * g;
        }
    }
}

// a warp per (token, v head); the blocks behind them move the rolling conv state on by the pass's last inputs, a thread per channel
__global__ void __launch_bounds__(128) delta_net_gate_kernel(const DeltaScanParams s, uint32_t gate_blocks) {
    pdl_launch_dependents();
    pdl_wait();
    const uzu_delta_net_update_args& a = s.p.f.update;
    const uzu_delta_net_conv_update_args& c = s.p.f.conv;
    const uint32_t lane = threadIdx.x & 31, conv_dim = 2 * a.key_dim + a.value_dim;
    const __nv_bfloat16* in = reinterpret_cast<const __nv_bfloat16*>(a.in_proj);
    if (blockIdx.x >= gate_blocks) {
        const uint32_t ch = (blockIdx.x - gate_blocks) * blockDim.x + threadIdx.x, taps = c.kernel_size - 1;
        if (ch >= conv_dim) return;
        float* st = reinterpret_cast<float*>(c.state) + (size_t)ch * c.state_stride;
        for (uint32_t j = 0; j < taps; ++j) {         // ascending: a short pass shifts the old inputs down first
            const uint32_t t = s.p.rows + j;          // input of token rows - taps + j
            st[j] = t >= taps ? bf2f(in[(size_t)(t - taps) * s.p.in_stride + ch]) : st[t];
        }
        return;
    }
    const uint32_t item = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (item >= s.p.rows * a.num_v_heads) return;
    const uint32_t t = item / a.num_v_heads, h = item % a.num_v_heads, DV = a.head_v_dim;
    const float* o = s.o + (size_t)t * a.value_dim + h * DV;
    const __nv_bfloat16* z = in + (size_t)t * s.p.in_stride + conv_dim + h * DV;
    __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(a.out) + (size_t)t * s.p.out_stride + h * DV;
    constexpr int NC = 4;
    float y[NC], ss = 0.0f;
#pragma unroll
    for (int i = 0; i < NC; ++i) {
        const uint32_t ci = lane + 32u * i;
        y[i] = ci < DV ? o[ci] : 0.0f;
        ss += y[i] * y[i];
    }
    const float inv_rms = 1.0f / sqrtf(warp_sum(ss) / (float)DV + a.norm_epsilon);
#pragma unroll
    for (int i = 0; i < NC; ++i) {
        const uint32_t ci = lane + 32u * i;
        if (ci < DV) out[ci] = f2bf(y[i] * inv_rms * reinterpret_cast<const float*>(a.norm_weight)[ci] * act_f32(UZU_ACT_SILU, bf2f(z[ci])));
    }
}

size_t delta_net_prefill_scratch_bytes(uint32_t rows, uint32_t key_dim, uint32_t value_dim, uint32_t v_heads) {
    return ((size_t)rows * (2 * (size_t)key_dim + 2 * (size_t)value_dim + 2 * (size_t)v_heads)) * sizeof(float);
}

static void encode_delta_net_scan(uzu_command_buffer* cmd, const DeltaPrefillParams& p, float* scratch) {
    const uzu_delta_net_update_args& a = p.f.update;
    DeltaScanParams s{p};
    s.q = scratch;                                   // key_dim is a multiple of 128: q and k rows stay 16-byte aligned
    s.k = s.q + (size_t)p.rows * a.key_dim;
    s.v = s.k + (size_t)p.rows * a.key_dim;
    s.o = s.v + (size_t)p.rows * a.value_dim;
    s.decay = s.o + (size_t)p.rows * a.value_dim;
    s.beta = s.decay + (size_t)p.rows * a.num_v_heads;
    const uint32_t units = 2 * a.num_k_heads + a.num_v_heads + 1, items = (p.rows + DP_BLOCK - 1) / DP_BLOCK * units;
    auto conv = [&](auto kernel) { launch(cmd, "delta_net_conv_kernel", kernel, dim3((items + 3) / 4), dim3(128), 0, s); };
    switch (p.f.conv.kernel_size - 1) {
        case 1: conv(delta_net_conv_kernel<1>); break;
        case 2: conv(delta_net_conv_kernel<2>); break;
        case 3: conv(delta_net_conv_kernel<3>); break;
        case 4: conv(delta_net_conv_kernel<4>); break;
        case 5: conv(delta_net_conv_kernel<5>); break;
        case 6: conv(delta_net_conv_kernel<6>); break;
        default: conv(delta_net_conv_kernel<7>); break;
    }
    uzu_gated_delta_args g{};
    g.prep.q = (uint64_t)s.q; g.prep.k = (uint64_t)s.k; g.prep.v = (uint64_t)s.v; g.prep.decay = (uint64_t)s.decay; g.prep.beta = (uint64_t)s.beta;
    g.prep.rows = p.rows; g.prep.heads = a.num_v_heads; g.prep.kv_heads = a.num_k_heads; g.prep.dim = DP_DK; g.prep.vdim = a.head_v_dim;
    g.prep.taps = 1;                                 // no convolution ring to advance
    g.state = a.state; g.out = (uint64_t)s.o;
    // an ordinary launch: started beside the convolution's last CTAs, two of the scan's would share an SM here and there (110 us instead of 78 for 509 tokens of 16 heads)
    const bool pdl = cmd->use_pdl;
    cmd->use_pdl = false;
    launch_gated_delta_scan(cmd, g);
    cmd->use_pdl = pdl;
    const uint32_t gate_blocks = (p.rows * a.num_v_heads + 3) / 4, conv_dim = 2 * a.key_dim + a.value_dim;
    launch(cmd, "delta_net_gate_kernel", delta_net_gate_kernel, dim3(gate_blocks + (conv_dim + 127) / 128), dim3(128), 0, s, gate_blocks);
}

static int g_delta_prefill = -1;   // -1: follow UZU_DELTA_PREFILL_KERNEL, 0 / 1: forced

// true = handled: the whole m-token recurrence of one DeltaNet layer. `scratch`: delta_net_prefill_scratch_bytes of f32 rows, 16-byte aligned
bool encode_delta_net_prefill(uzu_command_buffer* cmd, const uzu_delta_net_fused_update_args& f, uint32_t rows, uint32_t in_stride, uint32_t out_stride,
                              uint64_t scratch) {
    static const bool env_enabled = [] { const char* e = getenv("UZU_DELTA_PREFILL_KERNEL"); return !e || atoi(e) != 0; }();   // default on
    if (!(g_delta_prefill < 0 ? env_enabled : g_delta_prefill != 0)) return false;
    const uzu_delta_net_update_args& a = f.update;
    const uzu_delta_net_conv_update_args& c = f.conv;
    if (rows < 2 || a.head_k_dim != DP_DK || a.head_v_dim == 0 || a.head_v_dim > 128) return false;
    if (a.num_k_heads == 0 || a.num_v_heads % a.num_k_heads || a.key_dim != a.num_k_heads * DP_DK || a.value_dim != a.num_v_heads * a.head_v_dim) return false;
    if (c.kernel_size < 2 || c.kernel_size - 1 > (uint32_t)DP_MAX_TAPS || c.conv_dim != 2 * a.key_dim + a.value_dim || c.in_out != a.in_proj) return false;
    if (!a.in_proj || !a.a_log || !a.dt_bias || !a.norm_weight || !a.state || !a.out || !c.conv_weight || !c.state || (c.has_bias && !c.bias)) return false;
    if ((a.state & 15u)) return false;
    if (rows >= 4 && scratch) {
        encode_delta_net_scan(cmd, DeltaPrefillParams{f, rows, in_stride, out_stride}, reinterpret_cast<float*>(scratch));
        return true;
    }
    if (a.num_v_heads != a.num_k_heads || (a.head_v_dim & 3u)) return false;
    const size_t smem = ((size_t)a.head_v_dim * DP_DK + 4 * DP_DK + 8) * sizeof(float);
    static std::atomic<uint64_t> smem_opt_in{0};
    opt_in_dynamic_smem(cmd, delta_net_prefill_kernel, (int)((int)(((size_t)128 * DP_DK + 4 * DP_DK + 8) * sizeof(float))), smem_opt_in);
    DeltaPrefillParams p{f, rows, in_stride, out_stride};
    delta_net_prefill_kernel<<<a.num_v_heads, DP_THREADS, smem, cmd->ctx->stream>>>(p);
    after_launch(cmd, "delta_net_prefill_kernel");
    return true;
}

}  // namespace uzu

extern "C" void uzu_debug_set_delta_prefill(int mode) { uzu::g_delta_prefill = mode; }
