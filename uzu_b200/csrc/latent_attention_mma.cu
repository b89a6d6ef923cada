// Latent attention of a prompt's rows on the tensor pipe, for bf16 caches (latent_attention.cu serves decoded rows, f32 caches and odd sizes).
//
// All heads of all tokens score against the same cache rows, so a CTA takes 32 consecutive (token, head) rows and walks the keys in tiles of 64,
// staged once. Queries and softmax weights are f32: each is the sum of THREE bf16 numbers (8 + 8 + 8 bits, exact to the last bit of f32), so that
// with exact bf16 products and f32 accumulation the scores and sums keep f32 precision; the cache's own rows are bf16.
//   8 warps = 2 row groups of 16 x 4 shares. Scores: a share is 16 keys, mma.sync.m16n8k16 over rank + rot channels, three planes. The row maxima and
//   the planes of the weights meet in shared memory. Sums: a share is a quarter of the rank columns, weights by ldmatrix from the planes, rows by
//   ldmatrix.trans from the same key tile (a cache row is key and value). The pipe cuts what it adds to an accumulator off at its last bit, so no
//   chain is longer than four leading products: they are summed by rounded additions. The first half of the next tile is requested while the second half of
//   this one is multiplied.
// A weight of zero does not hide a row that is not finite (0 x NaN), so tiles that some row sees in part are looked over first, and one with infinities or
// NaN is summed key by key for the rows that see them: no token reaches an earlier one, none from before the window comes back.
// Bound: mma.sync issue, three products per score and sum. 1024 tokens x 16 heads, rank 512 + 64: 0.26 ms (210 TFLOP/s of the three planes) against 1.99 ms with a token and 8 heads per CTA
// on the FMA pipe; error against 64 bits 2.3e-7 (3.1e-7 there).
#include <algorithm>
#include <type_traits>

#include "common.cuh"

namespace uzu {

namespace {

constexpr uint32_t LM_ROWS = 32, LM_KEYS = 64, LM_PLD = LM_KEYS + 8, LM_THREADS = 256;

__device__ __forceinline__ void lm_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void lm_ldmatrix(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void lm_ldmatrix_trans(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
// (x0, x1) = the sum of three bf16 pairs
__device__ __forceinline__ void lm_split3(float x0, float x1, uint32_t (&w)[3]) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(x0, x1);
        w[i] = *reinterpret_cast<const uint32_t*>(&h);
        x0 -= __uint_as_float(w[i] << 16);
        x1 -= __uint_as_float(w[i] & 0xFFFF0000u);
    }
}

// A number of any size: beyond bf16's largest one the leading part is cut off instead of rounded, and an infinity has no rest.
__device__ __forceinline__ uint32_t lm_leading(float& x) {
    uint32_t h = __bfloat16_as_ushort(__float2bfloat16_rn(x));
    if ((h & 0x7F80u) == 0x7F80u && x == x) h = __float_as_uint(x) >> 16;
    x = fabsf(x) == INFINITY ? 0.0f : x - __uint_as_float(h << 16);
    return h;
}
// either half of a word is an infinity or NaN
__device__ __forceinline__ uint32_t lm_not_finite(uint32_t w) { return (uint32_t)((w & 0x7F80u) == 0x7F80u) | (uint32_t)((w & 0x7F800000u) == 0x7F800000u); }
// lm_split3 for numbers of any size
__device__ __forceinline__ void lm_split3_any(float x0, float x1, uint32_t (&w)[3]) {
    lm_split3(x0, x1, w);
    if (lm_not_finite(w[0])) {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const uint32_t lo = lm_leading(x0);
            w[i] = lo | lm_leading(x1) << 16;
        }
    }
}

}  // namespace

// NB: most 16-column blocks of a quarter of the rank
template <int NB>
__global__ void __launch_bounds__(LM_THREADS, 1) latent_attention_mma_kernel(const uzu_latent_attention_args a) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) uint8_t lm_raw[];
    __shared__ float s_part[4][LM_ROWS];
    const uint32_t width = a.rank + a.rot_dim, ld = width + 8, steps = width / 16, nb = a.rank / 64;
    const uint32_t q_plane = LM_ROWS * ld * 2, p_plane = LM_ROWS * LM_PLD * 2;
    const uint32_t sq = (uint32_t)__cvta_generic_to_shared(lm_raw), sk = sq + 3 * q_plane, sp = sk + LM_KEYS * ld * 2;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, quad = lane >> 2, tq = lane & 3, rg = warp & 1, share = warp >> 1;
    const uint32_t total = a.rows * a.heads, row0 = (gridDim.x - 1u - blockIdx.x) * LM_ROWS;      // the rows with the most keys first
    const uint32_t last_t = (min(row0 + LM_ROWS, total) - 1u) / a.heads, nkeys = a.prefix + last_t + 1u;
    const uint32_t first_keys = a.prefix + row0 / a.heads + 1u;
    const uint32_t last_lo = a.window && nkeys > a.window ? nkeys - a.window : 0u;
    const uint32_t t_begin = (a.window && first_keys > a.window ? first_keys - a.window : 0u) / LM_KEYS, t_end = (nkeys + LM_KEYS - 1) / LM_KEYS;
    const __nv_bfloat16* cache = reinterpret_cast<const __nv_bfloat16*>(a.cache);

    auto load_half = [&](uint32_t t, uint32_t half) {                    // 32 rows of tile t; rows past the last key are zero, never read
        const uint32_t pieces = width / 8;
        for (uint32_t i = tid; i < 32u * pieces; i += LM_THREADS) {
            const uint32_t r = i / pieces + half * 32u, c = i % pieces, key = t * LM_KEYS + r;
            const bool ok = key < nkeys;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(sk + (r * ld + c * 8) * 2), "l"(cache + (size_t)(ok ? key : 0u) * width + c * 8), "r"(ok ? 16u : 0u)
                         : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    load_half(t_begin, 0);
    load_half(t_begin, 1);
    {   // the query rows as three planes
        const float* q = reinterpret_cast<const float*>(a.query) + (size_t)row0 * width;
        const uint32_t pairs = width / 2;
        constexpr int BATCH = 6;                                         // requests in flight
        for (uint32_t i0 = tid; i0 < LM_ROWS * pairs; i0 += BATCH * LM_THREADS) {
            float2 x[BATCH];
#pragma unroll
            for (int u = 0; u < BATCH; ++u) {
                const uint32_t i = i0 + u * LM_THREADS, r = i / pairs, c = i % pairs * 2;
                x[u] = r < LM_ROWS && row0 + r < total ? *reinterpret_cast<const float2*>(q + (size_t)r * width + c) : make_float2(0.0f, 0.0f);
            }
#pragma unroll
            for (int u = 0; u < BATCH; ++u) {
                const uint32_t i = i0 + u * LM_THREADS, r = i / pairs, c = i % pairs * 2;
                if (r >= LM_ROWS) break;
                uint32_t w[3];
                lm_split3_any(x[u].x, x[u].y, w);
#pragma unroll
                for (int p = 0; p < 3; ++p) asm volatile("st.shared.u32 [%0], %1;" ::"r"(sq + p * q_plane + (r * ld + c) * 2), "r"(w[p]) : "memory");
            }
        }
    }
    float o[NB][2][4];
#pragma unroll
    for (int b = 0; b < NB; ++b)
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int c = 0; c < 4; ++c) o[b][h][c] = 0.0f;
    const uint32_t lr = rg * 16 + quad, ra = row0 + lr, rb = ra + 8;     // this thread's rows: lr and lr + 8 of the tile
    const uint32_t lim_a = ra < total ? a.prefix + ra / a.heads + 1u : 0u, lim_b = rb < total ? a.prefix + rb / a.heads + 1u : 0u;
    const uint32_t lo_a = a.window && lim_a > a.window ? lim_a - a.window : 0u, lo_b = a.window && lim_b > a.window ? lim_b - a.window : 0u;
    float m_a = -INFINITY, m_b = -INFINITY, l_a = 0.0f, l_b = 0.0f;      // running maximum; this lane's share of the weight sums
    const uint32_t q_addr = sq + ((rg * 16 + (lane & 15)) * ld + (lane >> 4) * 8) * 2;
    const uint32_t k_addr = sk + ((share * 16 + (lane >> 4) * 8 + (lane & 7)) * ld + ((lane >> 3) & 1) * 8) * 2;
    const uint32_t p_addr = sp + ((rg * 16 + (lane & 15)) * LM_PLD + (lane >> 4) * 8) * 2;
    const uint32_t v_addr = sk + ((lane & 15) * ld + share * (a.rank / 4) + (lane >> 4) * 8) * 2;

    auto tile = [&](const uint32_t t, auto part_c) {                     // part: not every row sees the whole tile
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        bool key_by_key = false;
        __syncthreads();
        if constexpr (decltype(part_c)::value) {
            uint32_t bad = 0;
            for (uint32_t r = warp; r < LM_KEYS; r += LM_THREADS / 32)
                for (uint32_t c = lane; c < a.rank / 8; c += 32) {
                    uint32_t x[4];
                    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(x[0]), "=r"(x[1]), "=r"(x[2]), "=r"(x[3]) : "r"(sk + (r * ld + c * 8) * 2));
#pragma unroll
                    for (int j = 0; j < 4; ++j) bad |= lm_not_finite(x[j]);
                }
            key_by_key = __syncthreads_or((int)bad) != 0;
        }
        // ---- scores of 16 rows x 16 keys ----
        float s[2][4], low[2][4];                                        // [8 keys]: the leading plane | the other two
#pragma unroll
        for (int i = 0; i < 8; ++i) s[i >> 2][i & 3] = low[i >> 2][i & 3] = 0.0f;
#pragma unroll 1
        for (uint32_t k0 = 0; k0 < steps; k0 += 4) {
            float part[2][4];
#pragma unroll
            for (int i = 0; i < 8; ++i) part[i >> 2][i & 3] = 0.0f;
#pragma unroll
            for (uint32_t kk = 0; kk < 4; ++kk) {
                const uint32_t ks = k0 + kk;
                if (ks >= steps) continue;
                uint32_t kf[4], qf[3][4];
                lm_ldmatrix(kf, k_addr + ks * 32);
#pragma unroll
                for (int p = 0; p < 3; ++p) lm_ldmatrix(qf[p], q_addr + p * q_plane + ks * 32);
                lm_mma(part[0], qf[0], kf[0], kf[1]);
                lm_mma(part[1], qf[0], kf[2], kf[3]);
#pragma unroll
                for (int p = 1; p < 3; ++p) {
                    lm_mma(low[0], qf[p], kf[0], kf[1]);
                    lm_mma(low[1], qf[p], kf[2], kf[3]);
                }
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) s[i >> 2][i & 3] += part[i >> 2][i & 3];
        }
        float x[2][4], mx_a = -INFINITY, mx_b = -INFINITY;
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const uint32_t key = t * LM_KEYS + share * 16 + n * 8 + 2 * tq + (c & 1);
                const bool sees = c < 2 ? key < lim_a && key >= lo_a : key < lim_b && key >= lo_b;
                x[n][c] = sees ? (s[n][c] + low[n][c]) * a.scale : -INFINITY;
                if (c < 2) mx_a = fmaxf(mx_a, x[n][c]);
                else mx_b = fmaxf(mx_b, x[n][c]);
            }
        mx_a = fmaxf(mx_a, __shfl_xor_sync(0xffffffffu, mx_a, 1)); mx_a = fmaxf(mx_a, __shfl_xor_sync(0xffffffffu, mx_a, 2));
        mx_b = fmaxf(mx_b, __shfl_xor_sync(0xffffffffu, mx_b, 1)); mx_b = fmaxf(mx_b, __shfl_xor_sync(0xffffffffu, mx_b, 2));
        if (tq == 0) { s_part[share][lr] = mx_a; s_part[share][lr + 8] = mx_b; }
        __syncthreads();
        float top_a = m_a, top_b = m_b;
#pragma unroll
        for (int i = 0; i < 4; ++i) { top_a = fmaxf(top_a, s_part[i][lr]); top_b = fmaxf(top_b, s_part[i][lr + 8]); }
        const float base_a = top_a == -INFINITY ? 0.0f : top_a, base_b = top_b == -INFINITY ? 0.0f : top_b;
        const float c_a = expf(m_a - base_a), c_b = expf(m_b - base_b);
        const bool moved = __any_sync(0xffffffffu, top_a != m_a || top_b != m_b);
        m_a = top_a;
        m_b = top_b;
        l_a *= c_a;
        l_b *= c_b;
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            const float e0 = expf(x[n][0] - base_a), e1 = expf(x[n][1] - base_a), e2 = expf(x[n][2] - base_b), e3 = expf(x[n][3] - base_b);
            l_a += e0 + e1;
            l_b += e2 + e3;
            uint32_t wa[3], wb[3];
            lm_split3(e0, e1, wa);
            lm_split3(e2, e3, wb);
            const uint32_t dst = sp + (lr * LM_PLD + share * 16 + n * 8 + 2 * tq) * 2;
#pragma unroll
            for (int p = 0; p < 3; ++p) {
                asm volatile("st.shared.u32 [%0], %1;" ::"r"(dst + p * p_plane), "r"(wa[p]) : "memory");
                asm volatile("st.shared.u32 [%0], %1;" ::"r"(dst + p * p_plane + 8 * LM_PLD * 2), "r"(wb[p]) : "memory");
            }
        }
        if (moved) {
#pragma unroll
            for (int b = 0; b < NB; ++b)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    o[b][h][0] *= c_a; o[b][h][1] *= c_a;
                    o[b][h][2] *= c_b; o[b][h][3] *= c_b;
                }
        }
        __syncthreads();
        // ---- weighted sums of 16 rows x a quarter of the rank ----
        if (key_by_key) {
            for (uint32_t k = 0; k < LM_KEYS; ++k) {
                const uint32_t key = t * LM_KEYS + k;
                const bool sees_a = key < lim_a && key >= lo_a, sees_b = key < lim_b && key >= lo_b;
                float w_a = 0.0f, w_b = 0.0f;
#pragma unroll
                for (int p = 2; p >= 0; --p) {
                    uint16_t ha, hb;
                    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(ha) : "r"(sp + p * p_plane + (lr * LM_PLD + k) * 2));
                    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(hb) : "r"(sp + p * p_plane + ((lr + 8) * LM_PLD + k) * 2));
                    w_a += bf16_bits_to_f32(ha);
                    w_b += bf16_bits_to_f32(hb);
                }
#pragma unroll
                for (int b = 0; b < NB; ++b) {
                    if ((uint32_t)b >= nb) continue;
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        uint32_t v;
                        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(sk + (k * ld + share * (a.rank / 4) + b * 16 + h * 8 + 2 * tq) * 2));
                        const float v0 = __uint_as_float(v << 16), v1 = __uint_as_float(v & 0xFFFF0000u);
                        if (sees_a) { o[b][h][0] = fmaf(w_a, v0, o[b][h][0]); o[b][h][1] = fmaf(w_a, v1, o[b][h][1]); }
                        if (sees_b) { o[b][h][2] = fmaf(w_b, v0, o[b][h][2]); o[b][h][3] = fmaf(w_b, v1, o[b][h][3]); }
                    }
                }
            }
            __syncthreads();
            if (t + 1 < t_end) load_half(t + 1, 0);
        } else {
#pragma unroll
            for (uint32_t half = 0; half < 2; ++half) {
                if (half) {
                    __syncthreads();                                         // every warp is done with the tile's first 32 keys
                    if (t + 1 < t_end) load_half(t + 1, 0);
                }
                uint32_t pf[2][3][4];
#pragma unroll
                for (int i = 0; i < 6; ++i) lm_ldmatrix(pf[i / 3][i % 3], p_addr + (i % 3) * p_plane + (half * 2 + i / 3) * 32);
#pragma unroll
                for (int b = 0; b < NB; ++b) {
                    if ((uint32_t)b >= nb) continue;
                    float part[2][4];
#pragma unroll
                    for (int i = 0; i < 8; ++i) part[i >> 2][i & 3] = 0.0f;
#pragma unroll
                    for (int ks = 0; ks < 2; ++ks) {
                        uint32_t vf[4];
                        lm_ldmatrix_trans(vf, v_addr + (half * 2 + ks) * 16 * ld * 2 + b * 32);
#pragma unroll
                        for (int p = 2; p >= 0; --p) {
                            lm_mma(part[0], pf[ks][p], vf[0], vf[1]);
                            lm_mma(part[1], pf[ks][p], vf[2], vf[3]);
                        }
                    }
#pragma unroll
                    for (int i = 0; i < 8; ++i) o[b][i >> 2][i & 3] += part[i >> 2][i & 3];
                }
            }
        }
        __syncthreads();
        if (t + 1 < t_end) load_half(t + 1, 1);
    };
    for (uint32_t t = t_begin; t < t_end; ++t) {
        if ((t + 1) * LM_KEYS > first_keys || t * LM_KEYS < last_lo) tile(t, std::true_type{});
        else tile(t, std::false_type{});
    }
    // a row's weight sum: over the quad's lanes, then over the four shares in order
    l_a += __shfl_xor_sync(0xffffffffu, l_a, 1); l_a += __shfl_xor_sync(0xffffffffu, l_a, 2);
    l_b += __shfl_xor_sync(0xffffffffu, l_b, 1); l_b += __shfl_xor_sync(0xffffffffu, l_b, 2);
    if (tq == 0) { s_part[share][lr] = l_a; s_part[share][lr + 8] = l_b; }
    __syncthreads();
    auto inverse = [&](uint32_t row, uint32_t r, float m) {
        float l = 0.0f;
#pragma unroll
        for (int i = 0; i < 4; ++i) l += s_part[i][r];
        const uint32_t t = row / a.heads, head = row % a.heads;
        if (a.sinks) l += expf(reinterpret_cast<const float*>(a.sinks)[head] - m);
        float inv = 1.0f / l;
        if (a.head_gate) inv *= 1.0f / (1.0f + expf(-reinterpret_cast<const float*>(a.head_gate)[(size_t)t * a.head_gate_stride + head]));
        return inv;
    };
    const float i_a = ra < total ? inverse(ra, lr, m_a) : 0.0f, i_b = rb < total ? inverse(rb, lr + 8, m_b) : 0.0f;
    float* out = reinterpret_cast<float*>(a.out) + share * (a.rank / 4) + 2 * tq;
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        if ((uint32_t)b >= nb) continue;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t c = b * 16 + h * 8;
            if (ra < total) *reinterpret_cast<float2*>(out + (size_t)ra * a.rank + c) = make_float2(o[b][h][0] * i_a, o[b][h][1] * i_a);
            if (rb < total) *reinterpret_cast<float2*>(out + (size_t)rb * a.rank + c) = make_float2(o[b][h][2] * i_b, o[b][h][3] * i_b);
        }
    }
}

static size_t latent_mma_smem(uint32_t width) { return ((size_t)3 * LM_ROWS * (width + 8) + (size_t)LM_KEYS * (width + 8) + (size_t)3 * LM_ROWS * LM_PLD) * 2; }

// bf16 rows of whole 16-byte pieces, a rank of whole 64 columns, sixteen tokens and more (fewer are cut into key splits over many CTAs), and enough keys: a
// tile of 64 costs the same however few are seen, and the FMA kernel takes a CTA per token and 8 heads and two to three keys a microsecond. 16 heads, FMA /
// this one, us: rank 64, 32 tokens 8.9 / 10.3, 48 tokens 10.9 / 10.3; rank 512, 32 tokens 15 / 25, 96 tokens 50 / 33, 20 tokens behind 100 44 / 33.
bool latent_attention_mma_applicable(const uzu_latent_attention_args& a) {
    const uint32_t width = a.rank + a.rot_dim;
    const uint64_t ctas = std::max<uint64_t>((uint64_t)a.rows * ((a.heads + 7) / 8), 148), keys = (uint64_t)(a.window ? std::min(a.prefix, a.window) : a.prefix) + a.rows;
    if (keys * ctas < (a.rank <= 128 ? 52u : a.heads < 8 ? 112u : 96u) * 148ull) return false;
    if (a.cache_dt != UZU_DT_BF16 || a.dynamic_position || a.splits > 1 || a.rows < 16) return false;
    if (a.rank % 64u || width % 16u || (a.cache & 15u) || (a.query & 7u) || (a.out & 7u)) return false;
    return (uint64_t)a.rows * a.heads < 0x80000000ull && latent_mma_smem(width) <= 225u * 1024u;
}

void encode_latent_attention_mma(uzu_command_buffer* cmd, const uzu_latent_attention_args& a) {
    const size_t smem = latent_mma_smem(a.rank + a.rot_dim);
    const dim3 grid((a.rows * a.heads + LM_ROWS - 1) / LM_ROWS);
    auto go = [&](auto kernel, std::atomic<uint64_t>& done) {
        opt_in_dynamic_smem(cmd, kernel, 225 * 1024, done);
        launch(cmd, "latent_attention_mma_kernel", kernel, grid, dim3(LM_THREADS), smem, a);
    };
    static std::atomic<uint64_t> done[3];
    if (a.rank <= 128) go(latent_attention_mma_kernel<2>, done[0]);
    else if (a.rank <= 256) go(latent_attention_mma_kernel<4>, done[1]);
    else go(latent_attention_mma_kernel<8>, done[2]);
}

}  // namespace uzu
