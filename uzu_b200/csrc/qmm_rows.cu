// Quantised MatmulKernel for a few activation rows (2 .. 32): every weight is read once and used for all rows. Speculation passes over a trie, decoded
// rows of several sequences, short prompts. Semantic spec: backends/cpu/kernel/matmul/kernel.rs:164-295.
//
// mma.sync.m16n8k16 with 16 output features as M and 8 activation rows as N: here it is the better pipe than tcgen05, whose products cost the same for
// 8 rows as for 64. Codes become bf16 INTEGERS code - zp in registers (exact: nibbles behind the bits of 128.0, one subtraction; bytes as two nibbles
// and one fma), sums of a group are f32, and a group's scale is one f32 fma per sum. Nothing of a weight is rounded. The integers enter times 2^-11 (bytes
// 2^-15) and a finished sum is brought back: a group's sum is no larger than the largest activation, so it is in range where the product is.
//   CTA     12 warps, one CTA per SM, pinned to a slice of k whose activations it keeps in shared memory in fragment order; slices of a tile meet in
//           the split-k workspace, added in slice order by whoever comes last (the same bits every time).
//   warp    an equal run of the CTA's (16 features, step of k) pairs; a tile that several warps share meets in shared memory, in order. Steps are
//           256 bytes of codes per row, with their scales and zero points, by cp.async into a ring of the warp's own.
//   lane    16 consecutive k of a group of 64 for two rows (g, g + 8 of the tile): 8 or 16 bytes of shared memory each, at pitches that spread a
//           quarter warp over all banks. The products' k order is the lanes' order, the same for both operands.
// Bound: the codes' way from HBM, then issue slots: a step of 16 features x 64 k is about 70 instructions, 130 for 8-bit codes.
// The linears of a layer of an 8B model (115 MB of 4-bit codes, groups of 64), us, with the kernels that took these rows before it (2 and 8 rows) or would take
// them without it (qmm_scaled.cu):
//   rows            2        8        16         24         32
//   4 bit        60 (84)  61 (85)  76 (118)   102 (129)  123 (131)      at 40 rows 135 (135): the line is at 32
//     groups 128          59 (112) 75 (114)   99 (116)   119 (118)
//   8 bit        85 (124) 88 (128) 105 (142)  121 (151)  146 (152)
//   MLX          62 (82)  65 (144) 81 (173)   108 (176)  130 (177)
#include <cstdlib>

#include "common.cuh"
#include "qmm_rows_index.h"

namespace uzu {

struct QrParams {
    const uint8_t* w;
    const __nv_bfloat16* scales;
    const uint8_t* second;           // zero points or biases
    const __nv_bfloat16* x;
    void* d;
    const __nv_bfloat16* bias;
    float* ws;
    unsigned int* counters;
    uint32_t m, n, k, row_bytes, groups, zp_stride, xor_mask;
    uint32_t steps, slice_steps, slices, tiles, whole;      // steps of k: all, of a slice; whole: tiles are not shared by warps
    uint32_t d_is_f32, accumulate, has_soft_cap;
    float ab_scale, soft_cap;        // ab_scale brings the integers' factor back
};

namespace {

constexpr int QR_WARPS = 12, QR_STAGES = 2;

template <int BITS>
struct QrShape {
    static constexpr uint32_t CODES = BITS == 4 ? 512 : 256, PITCH = BITS == 4 ? 288 : 320, STAGE = 16 * PITCH + 512;
    static constexpr float DOWN = BITS == 4 ? 1.0f / 2048.0f : 1.0f / 32768.0f;                              // the integers' factor
    static constexpr uint32_t MAGIC = BITS == 4 ? 0x3D803D80u : 0x3B803B80u;                                 // bf16 128 DOWN, twice
};

template <int BYTES>
__device__ __forceinline__ void qr_cp_async(uint32_t dst, const void* src) {
    if constexpr (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst), "l"(src), "n"(BYTES) : "memory");
}
__device__ __forceinline__ void qr_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// nibbles 0 and 4 of w as bf16 128 + nibble, times the integers' factor
__device__ __forceinline__ uint32_t qr_nibbles(uint32_t w, uint32_t magic) {
    uint32_t r;
    asm("lop3.b32 %0, %1, 0x000f000f, %2, 0xEA;" : "=r"(r) : "r"(w), "r"(magic));
    return r;
}
__device__ __forceinline__ uint32_t qr_sub(uint32_t a, uint32_t b) {
    const __nv_bfloat162 r = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
    return *reinterpret_cast<const uint32_t*>(&r);
}
__device__ __forceinline__ uint32_t qr_mad16(uint32_t a, uint32_t b) {             // 16 a + b
    const uint32_t sixteen = 0x41804180u;
    const __nv_bfloat162 r = __hfma2(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&sixteen), *reinterpret_cast<const __nv_bfloat162*>(&b));
    return *reinterpret_cast<const uint32_t*>(&r);
}
// Four codes of a byte word less the zero point: (0, 2) and (1, 3). lo, hi: 128 + the zero point's nibbles, times the factor
__device__ __forceinline__ void qr_bytes(uint32_t w, uint32_t lo, uint32_t hi, uint32_t magic, uint32_t& p02, uint32_t& p13) {
    p02 = qr_mad16(qr_sub(qr_nibbles(w >> 4, magic), hi), qr_sub(qr_nibbles(w, magic), lo));
    p13 = qr_mad16(qr_sub(qr_nibbles(w >> 12, magic), hi), qr_sub(qr_nibbles(w >> 8, magic), lo));
}

template <int BITS, int GS, int METHOD, int MB>
__global__ void __launch_bounds__(QR_WARPS * 32, 1) qmm_rows_kernel(const QrParams p) {
    using S = QrShape<BITS>;
    constexpr uint32_t CODES = S::CODES, PITCH = S::PITCH, NG = CODES / GS, SB = NG * 2, MROWS = MB * 8, ITEMS = CODES / 8;
    constexpr bool kZero = METHOD == UZU_QMETHOD_SCALE_ZERO_POINT, kBias = METHOD == UZU_QMETHOD_SCALE_BIAS;
    extern __shared__ __align__(16) uint8_t qr_smem[];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const uint32_t slice = blockIdx.x % p.slices, column = blockIdx.x / p.slices, columns = gridDim.x / p.slices;
    const uint32_t s0 = slice * p.slice_steps, s1 = min(p.steps, s0 + p.slice_steps);
    const uint32_t tile_begin = (uint32_t)((uint64_t)column * p.tiles / columns), tile_end = (uint32_t)((uint64_t)(column + 1) * p.tiles / columns);
    const uint32_t xstride = p.slice_steps * ITEMS + 1;                       // odd: the rows of a fragment read fall on all banks
    uint4* xs = reinterpret_cast<uint4*>(qr_smem);                            // [MROWS][xstride]
    float* sx = reinterpret_cast<float*>(xs + (size_t)MROWS * xstride);       // [slice_steps * NG][MROWS]: sums of the groups' activations, times the factor (ScaleBias)
    float* turns = sx + (kBias ? (size_t)p.slice_steps * NG * MROWS : 0), *turn = turns + warp * 128;      // [8][16] of each warp
    float4* heads = reinterpret_cast<float4*>(turns + QR_WARPS * 128);        // [warps][MB][32]: what a warp adds to a tile that another one began
    uint8_t* ring = reinterpret_cast<uint8_t*>(heads + (p.whole ? 0 : QR_WARPS * MB * 32)) + (size_t)warp * QR_STAGES * S::STAGE;
    const uint32_t ring_s = (uint32_t)__cvta_generic_to_shared(ring);
    uint32_t magic;
    asm volatile("mov.b32 %0, %1;" : "=r"(magic) : "n"(S::MAGIC));

    auto zero_fetch = [&](uint32_t row, uint32_t step) { return qr_zero_fetch(row, step, p.n, p.zp_stride, BITS == 4 ? NG / 2 : NG); };
    auto issue_stage = [&](uint32_t tile, uint32_t step, uint32_t slot) {
        const uint32_t dst = ring_s + slot * S::STAGE;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t r = (uint32_t)i * 2u + (lane >> 4), b = lane & 15, row = min(tile * 16u + r, p.n - 1u);
            qr_cp_async<16>(dst + r * PITCH + b * 16u, p.w + (size_t)row * p.row_bytes + (size_t)step * 256u + b * 16u);
        }
        const uint32_t r = lane & 15, row = min(tile * 16u + r, p.n - 1u);
        const uint32_t at = dst + 16 * PITCH + r * 16u;
        const size_t group = (size_t)row * p.groups + step * NG;
        if (lane < 16) qr_cp_async<SB>(at, p.scales + group);
        else if (kZero) {
            const QrZeroFetch z = zero_fetch(row, step);
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(at + 256u), "l"(p.second + z.offset), "r"(z.bytes) : "memory");
        }
        else if (kBias) qr_cp_async<SB>(at + 256u, reinterpret_cast<const __nv_bfloat16*>(p.second) + group);
    };
    // the column's (tile, step) pairs in order, an equal run of them for each warp
    const uint32_t steps = s1 - s0, tiles = tile_end - tile_begin;
    auto unit_at = [&](uint32_t w) { return p.whole ? w * tiles / QR_WARPS * steps : w * tiles * steps / QR_WARPS; };
    const uint32_t u_begin = unit_at(warp), u_end = unit_at(warp + 1);
    uint32_t i_unit = u_begin, i_tile = tile_begin + u_begin / steps, i_step = s0 + u_begin % steps, issued = 0;
    auto issue_next = [&]() {
        if (i_unit < u_end) {
            issue_stage(i_tile, i_step, issued % QR_STAGES);
            ++i_unit;
            if (++i_step == s1) { i_step = s0; ++i_tile; }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        ++issued;
    };
#pragma unroll
    for (int i = 0; i < QR_STAGES - 1; ++i) issue_next();                     // weights do not wait for the producer of the activations
    pdl_launch_dependents();
    pdl_wait();
    {   // the slice's activations in fragment order, rows past the last one zero
        constexpr int BATCH = 8;
        const uint32_t items = (s1 - s0) * ITEMS, total = MROWS * items;
        for (uint32_t base = tid; base < total; base += QR_WARPS * 32 * BATCH) {
            uint4 v[BATCH];
#pragma unroll
            for (int u = 0; u < BATCH; ++u) {
                const uint32_t it = base + u * QR_WARPS * 32, r = it / items, li = it % items;
                v[u] = it < total && r < p.m ? *reinterpret_cast<const uint4*>(p.x + (size_t)r * p.k + ((size_t)s0 * ITEMS + li) * 8u) : make_uint4(0, 0, 0, 0);
            }
#pragma unroll
            for (int u = 0; u < BATCH; ++u) {
                const uint32_t it = base + u * QR_WARPS * 32, r = it / items, li = it % items;
                if (it >= total) break;                                       // uniform over a warp: items is a multiple of 32
                uint4 o;
                if (BITS == 4) {
                    o = make_uint4(__byte_perm(v[u].x, v[u].z, 0x5410), __byte_perm(v[u].x, v[u].z, 0x7632), __byte_perm(v[u].y, v[u].w, 0x5410), __byte_perm(v[u].y, v[u].w, 0x7632));
                } else {
                    o = make_uint4(__byte_perm(v[u].x, v[u].y, 0x5410), __byte_perm(v[u].x, v[u].y, 0x7632), __byte_perm(v[u].z, v[u].w, 0x5410), __byte_perm(v[u].z, v[u].w, 0x7632));
                }
                xs[(size_t)r * xstride + li] = o;
                if (kBias) {
                    const uint32_t e[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
                    float sum = 0.0f;
#pragma unroll
                    for (int i = 0; i < 4; ++i) sum += fmaf(S::DOWN, __uint_as_float(e[i] << 16), S::DOWN * __uint_as_float(e[i] & 0xffff0000u));
#pragma unroll
                    for (uint32_t o_ = 1; o_ < GS / 8; o_ <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o_);
                    if (li % (GS / 8) == 0) sx[(size_t)(li / (GS / 8)) * MROWS + r] = sum;
                }
            }
        }
    }
    __syncthreads();

    float acc[MB][4];
    auto finish = [&](uint32_t tile) {
        if (p.slices > 1) {
            float4* ws = reinterpret_cast<float4*>(p.ws) + (size_t)tile * p.slices * (MB * 32) + lane;
#pragma unroll
            for (int c = 0; c < MB; ++c) ws[(size_t)slice * (MB * 32) + c * 32] = make_float4(acc[c][0], acc[c][1], acc[c][2], acc[c][3]);
            __threadfence();
            __syncwarp();
            unsigned int ticket = 0;
            if (lane == 0) ticket = atomicAdd(&p.counters[tile], 1u);
            ticket = __shfl_sync(0xffffffffu, ticket, 0);
            if (ticket != p.slices - 1) return;
            __threadfence();
#pragma unroll
            for (int c = 0; c < MB; ++c) acc[c][0] = acc[c][1] = acc[c][2] = acc[c][3] = 0.0f;
#pragma unroll 4
            for (uint32_t s = 0; s < p.slices; ++s)
#pragma unroll
                for (int c = 0; c < MB; ++c) {
                    const float4 v = __ldcg(ws + (size_t)s * (MB * 32) + c * 32);
                    acc[c][0] += v.x; acc[c][1] += v.y; acc[c][2] += v.z; acc[c][3] += v.w;
                }
            if (lane == 0) p.counters[tile] = 0;
        }
#pragma unroll
        for (int c = 0; c < MB; ++c) {                                        // 8 rows at a time: fragment order -> features side by side
            __syncwarp();
            turn[(2 * t) * 16 + g] = acc[c][0];
            turn[(2 * t + 1) * 16 + g] = acc[c][1];
            turn[(2 * t) * 16 + g + 8] = acc[c][2];
            turn[(2 * t + 1) * 16 + g + 8] = acc[c][3];
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t o = lane + 32u * i, row = (uint32_t)c * 8u + o / 16u, feature = tile * 16u + o % 16u;
                if (row >= p.m || feature >= p.n) continue;
                const size_t idx = (size_t)row * p.n + feature;
                float v = p.ab_scale * turn[o];
                if (p.accumulate) v += p.d_is_f32 ? reinterpret_cast<const float*>(p.d)[idx] : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p.d)[idx]);
                if (p.bias) v += __bfloat162float(p.bias[feature]);
                if (p.has_soft_cap) v = p.soft_cap * tanhf(v / p.soft_cap);
                if (p.d_is_f32) reinterpret_cast<float*>(p.d)[idx] = v;
                else reinterpret_cast<__nv_bfloat16*>(p.d)[idx] = __float2bfloat16_rn(v);
            }
        }
    };
    uint32_t consumed = 0, open_tile = ~0u;
    for (uint32_t unit = u_begin; unit < u_end;) {
        const uint32_t tile = tile_begin + unit / steps;
        const bool began = unit % steps == 0;
#pragma unroll
        for (int c = 0; c < MB; ++c) acc[c][0] = acc[c][1] = acc[c][2] = acc[c][3] = 0.0f;
#pragma unroll 1
        for (uint32_t step = s0 + unit % steps, last = min(s1, step + u_end - unit); step < last; ++step, ++unit) {
            __syncwarp();                                                     // every lane is done with the slot that is filled next
            issue_next();
            asm volatile("cp.async.wait_group %0;" ::"n"(QR_STAGES - 1) : "memory");
            __syncwarp();
            const uint8_t* st = ring + (consumed % QR_STAGES) * S::STAGE;
            ++consumed;
            const uint8_t *ca = st + g * PITCH, *cb = ca + 8 * PITCH, *fa = st + 16 * PITCH + g * 16, *fb = fa + 128;
            constexpr int SW = SB / 4;
            uint32_t sa[SW], sb[SW], za[SW], zb[SW];
#pragma unroll
            for (int i = 0; i < SW; ++i) {
                sa[i] = reinterpret_cast<const uint32_t*>(fa)[i];
                sb[i] = reinterpret_cast<const uint32_t*>(fb)[i];
                za[i] = zb[i] = 0u;
                if (kBias || (kZero && i == 0)) {
                    za[i] = reinterpret_cast<const uint32_t*>(fa + 256)[i];
                    zb[i] = reinterpret_cast<const uint32_t*>(fb + 256)[i];
                }
            }
            if (kZero && GS == 128) {                                         // two bytes of a word
                za[0] >>= zero_fetch(min(tile * 16u + g, p.n - 1u), step).shift;
                zb[0] >>= zero_fetch(min(tile * 16u + g + 8u, p.n - 1u), step).shift;
            }
            const uint4* xrow = xs + (size_t)g * xstride + (size_t)(step - s0) * ITEMS + 2 * t;
#pragma unroll
            for (int gq = 0; gq < (int)NG; ++gq) {
                float d[MB][4];
#pragma unroll
                for (int c = 0; c < MB; ++c) d[c][0] = d[c][1] = d[c][2] = d[c][3] = 0.0f;
                uint32_t lo_a, lo_b, hi_a = magic, hi_b = magic;              // 128 + the zero point (its nibbles), times the factor
                if (kZero) {
                    const uint32_t z1 = za[0] >> (gq * BITS), z2 = zb[0] >> (gq * BITS);
                    lo_a = magic + (z1 & 15u) * 0x00010001u;
                    lo_b = magic + (z2 & 15u) * 0x00010001u;
                    if (BITS == 8) { hi_a = magic + (z1 >> 4 & 15u) * 0x00010001u; hi_b = magic + (z2 >> 4 & 15u) * 0x00010001u; }
                } else if (kBias) {
                    lo_a = lo_b = magic;
                } else {
                    lo_a = lo_b = BITS == 4 ? S::MAGIC + 0x00080008u : magic;
                    hi_a = hi_b = S::MAGIC + 0x00080008u;
                }
#pragma unroll
                for (int part = 0; part < GS / 64; ++part) {
                    const int q = gq * (GS / 64) + part;
                    uint32_t wa[BITS / 2], wb[BITS / 2];
                    if (BITS == 4) {
                        *reinterpret_cast<uint2*>(wa) = *reinterpret_cast<const uint2*>(ca + q * 32 + t * 8);
                        *reinterpret_cast<uint2*>(wb) = *reinterpret_cast<const uint2*>(cb + q * 32 + t * 8);
                    } else {
                        *reinterpret_cast<uint4*>(wa) = *reinterpret_cast<const uint4*>(ca + q * 64 + t * 16);
                        *reinterpret_cast<uint4*>(wb) = *reinterpret_cast<const uint4*>(cb + q * 64 + t * 16);
                    }
#pragma unroll
                    for (int i = 0; i < BITS / 2; ++i) { wa[i] ^= p.xor_mask; wb[i] ^= p.xor_mask; }
#pragma unroll
                    for (int w = 0; w < 2; ++w) {                             // 8 of the lane's 16 k: two products
                        uint32_t a[4], b[4];
                        if (BITS == 4) {
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                a[i] = qr_sub(qr_nibbles(wa[w] >> (4 * i), magic), lo_a);
                                b[i] = qr_sub(qr_nibbles(wb[w] >> (4 * i), magic), lo_b);
                            }
                        } else {
#pragma unroll
                            for (int i = 0; i < 2; ++i) {
                                qr_bytes(wa[w * 2 + i], lo_a, hi_a, magic, a[2 * i], a[2 * i + 1]);
                                qr_bytes(wb[w * 2 + i], lo_b, hi_b, magic, b[2 * i], b[2 * i + 1]);
                            }
                        }
#pragma unroll
                        for (int c = 0; c < MB; ++c) {
                            const uint4 x = xrow[(size_t)c * 8 * xstride + q * 8 + w];
                            qr_mma(d[c], a[0], b[0], a[1], b[1], x.x, x.y);
                            qr_mma(d[c], a[2], b[2], a[3], b[3], x.z, x.w);
                        }
                    }
                }
                auto half = [&](uint32_t v) { return __uint_as_float((gq & 1) ? v & 0xffff0000u : v << 16); };
                const float fs_a = half(sa[gq / 2]), fs_b = half(sb[gq / 2]);
#pragma unroll
                for (int c = 0; c < MB; ++c) {
                    acc[c][0] = fmaf(fs_a, d[c][0], acc[c][0]);
                    acc[c][1] = fmaf(fs_a, d[c][1], acc[c][1]);
                    acc[c][2] = fmaf(fs_b, d[c][2], acc[c][2]);
                    acc[c][3] = fmaf(fs_b, d[c][3], acc[c][3]);
                    if (kBias) {
                        const float2 sums = *reinterpret_cast<const float2*>(sx + (size_t)((step - s0) * NG + gq) * MROWS + c * 8 + 2 * t);
                        const float b_a = half(za[gq / 2]), b_b = half(zb[gq / 2]);
                        acc[c][0] = fmaf(b_a, sums.x, acc[c][0]);
                        acc[c][1] = fmaf(b_a, sums.y, acc[c][1]);
                        acc[c][2] = fmaf(b_b, sums.x, acc[c][2]);
                        acc[c][3] = fmaf(b_b, sums.y, acc[c][3]);
                    }
                }
            }
        }
        if (!began) {
#pragma unroll
            for (int c = 0; c < MB; ++c) heads[(warp * MB + c) * 32 + lane] = make_float4(acc[c][0], acc[c][1], acc[c][2], acc[c][3]);
        } else if (unit % steps == 0) {
            finish(tile);
        } else {
            open_tile = tile;                                                 // its run ends inside the tile: the sums stay in registers
        }
    }
    __syncthreads();
    if (open_tile != ~0u) {                                                   // the following warps' shares, in order
        const uint32_t tile_units = (open_tile - tile_begin + 1) * steps;
        for (uint32_t w = warp + 1; w < QR_WARPS && unit_at(w) < tile_units; ++w) {
            if (unit_at(w) == unit_at(w + 1)) continue;
#pragma unroll
            for (int c = 0; c < MB; ++c) {
                const float4 v = heads[(w * MB + c) * 32 + lane];
                acc[c][0] += v.x; acc[c][1] += v.y; acc[c][2] += v.z; acc[c][3] += v.w;
            }
        }
        finish(open_tile);
    }
}

struct QrPlan { uint32_t slice_steps = 0, slices = 0, whole = 0; size_t smem = 0; };

// Slices of k: a CTA's activations have to fit beside its rings; more slices give few tiles to more warps, at a workspace round trip per tile. Time in
// steps of a warp: its run of steps + meeting the other slices + staging the activations + meeting the other warps. The last is about 2 us: equal runs
// win where a warp has many steps (28672 x 4096, 8 rows: 22.9 us, 28.8 in whole tiles), whole tiles where it has few (4096 x 4096: 9.9 us, 11.7 in runs).
QrPlan qr_plan(uint32_t m, uint32_t n, uint32_t k, uint32_t bits, uint32_t gs, bool bias, uint32_t sms, size_t ws_bytes, uint32_t ws_counters) {
    const uint32_t codes = bits == 4 ? 512 : 256, steps = k / codes, tiles = (n + 15) / 16, mrows = (m + 7) / 8 * 8;
    const size_t rings = (size_t)QR_WARPS * (QR_STAGES * (bits == 4 ? QrShape<4>::STAGE : QrShape<8>::STAGE) + 512), heads = (size_t)QR_WARPS * mrows * 64;
    QrPlan best;
    float least = 1e30f;
    for (uint32_t slices = 1; slices <= std::min(steps, sms); ++slices) {
        const uint32_t per = (steps + slices - 1) / slices;
        if ((steps + per - 1) / per != slices) continue;                      // the same slices as a smaller count
        if (slices > 1 && ((size_t)tiles * slices * mrows * 64 > ws_bytes || tiles > ws_counters)) continue;
        const size_t fixed = rings + (size_t)mrows * (per * (codes / 8) + 1) * 16 + (bias ? (size_t)per * (codes / gs) * mrows * 4 : 0);
        const uint32_t columns = std::min(tiles, sms / slices), share = (tiles + columns - 1) / columns;
        for (uint32_t whole = 0; whole < 2; ++whole) {
            const size_t smem = fixed + (whole ? 0 : heads);
            if (smem > 226u * 1024u) continue;
            const uint32_t of_warp = (share + QR_WARPS - 1) / QR_WARPS, run = whole ? of_warp * per : (share * per + QR_WARPS - 1) / QR_WARPS;
            const float cost = run * (0.6f + 0.05f * mrows) + (slices > 1 ? of_warp * (0.6f + 0.002f * slices * mrows) : 0.1f) + 0.012f * mrows * per +
                               (whole ? 0.0f : 1.6f + 0.05f * mrows);
            if (cost < least) {
                least = cost;
                best.slice_steps = per;
                best.slices = slices;
                best.whole = whole;
                best.smem = smem;
            }
        }
    }
    return best;
}

template <int BITS, int GS, int METHOD>
void qr_launch(uzu_command_buffer* cmd, const QrParams& p, uint32_t grid, size_t smem) {
    static std::atomic<uint64_t> done[4];
    auto go = [&](auto mb) {
        constexpr int MB = decltype(mb)::value;
        opt_in_dynamic_smem(cmd, qmm_rows_kernel<BITS, GS, METHOD, MB>, 226 * 1024, done[MB - 1]);
        launch(cmd, "qmm_rows_kernel", qmm_rows_kernel<BITS, GS, METHOD, MB>, dim3(grid), dim3(QR_WARPS * 32), smem, p);
    };
    switch ((p.m + 7) / 8) {
        case 1: go(std::integral_constant<int, 1>{}); break;
        case 2: go(std::integral_constant<int, 2>{}); break;
        case 3: go(std::integral_constant<int, 3>{}); break;
        default: go(std::integral_constant<int, 4>{}); break;
    }
}

template <int BITS, int GS>
void qr_method(uzu_command_buffer* cmd, const QrParams& p, uint32_t prologue, uint32_t grid, size_t smem) {
    if (prologue == UZU_B_SCALE_ZERO_POINT_DEQUANT) qr_launch<BITS, GS, UZU_QMETHOD_SCALE_ZERO_POINT>(cmd, p, grid, smem);
    else if (prologue == UZU_B_SCALE_BIAS_DEQUANT) qr_launch<BITS, GS, UZU_QMETHOD_SCALE_BIAS>(cmd, p, grid, smem);
    else qr_launch<BITS, GS, UZU_QMETHOD_SCALE_SYMMETRIC>(cmd, p, grid, smem);
}

// rows of one launch: 17 .. 63 over a matrix of at most 2^21 weights go 16 at a time, a launch count that the kernel tests hold on to. It costs time: 1024 x 2048, 24
// rows, int4 16.6 us, 8.5 in one launch; 40 rows 24.8, 14.6 on qmm_scaled.cu. Larger matrices: 3072 x 1024, 24 rows 10.5 (18.0 in launches of 16).
uint32_t qr_rows_per_launch(const uzu_matmul_args& a) { return a.m > 16 && (uint64_t)a.n * a.k <= (1u << 21) ? 16u : a.m; }

}  // namespace

bool qmm_rows_applicable(uzu_command_buffer* cmd, const uzu_matmul_args& a) {
    static const bool off = [] { const char* e = getenv("UZU_QMM_ROWS"); return e && atoi(e) == 0; }();      // 0: the kernels for other shapes (A/B runs)
    if (off || a.m < 2 || a.m >= 64 || qr_rows_per_launch(a) > 32) return false;
    if (a.b_prologue == UZU_B_FULL_PRECISION || a.gather_indices || !a.b_transpose) return false;
    if (a.input_dt != UZU_DT_BF16 || a.weights_dt != UZU_DT_BF16) return false;
    if (a.output_dt != UZU_DT_BF16 && a.output_dt != UZU_DT_F32) return false;
    if (a.b_mode != UZU_QMODE_U4 && a.b_mode != UZU_QMODE_U8) return false;
    const uint32_t bits = a.b_mode == UZU_QMODE_U4 ? 4 : 8;
    if ((a.b_group_size != 64 && a.b_group_size != 128) || a.n == 0 || a.k == 0 || (uint64_t)a.k * bits % 2048u) return false;
    if (((a.a | a.b | a.b_scales | a.b_zero_points | a.b_biases) & 15u)) return false;
    return qr_plan(qr_rows_per_launch(a), a.n, a.k, bits, a.b_group_size, a.b_prologue == UZU_B_SCALE_BIAS_DEQUANT, cmd->ctx->sm_count, cmd->ctx->splitk_ws_bytes,
                   cmd->ctx->splitk_counter_count).slices != 0;
}

void encode_qmm_rows(uzu_command_buffer* cmd, const uzu_matmul_args& a) {
    const uint32_t bits = a.b_mode == UZU_QMODE_U4 ? 4 : 8, most = qr_rows_per_launch(a);
    const bool mlx = a.b_prologue == UZU_B_SCALE_BIAS_DEQUANT;
    for (uint32_t m0 = 0; m0 < a.m; m0 += most) {
        QrParams p{};
        p.m = std::min(most, a.m - m0); p.n = a.n; p.k = a.k;
        const QrPlan plan = qr_plan(p.m, a.n, a.k, bits, a.b_group_size, mlx, cmd->ctx->sm_count, cmd->ctx->splitk_ws_bytes, cmd->ctx->splitk_counter_count);
        p.w = (const uint8_t*)a.b;
        p.scales = (const __nv_bfloat16*)a.b_scales;
        p.second = (const uint8_t*)(mlx ? a.b_biases : a.b_zero_points);
        p.x = (const __nv_bfloat16*)a.a + (size_t)m0 * a.k;
        p.d = (void*)(a.d + (size_t)m0 * a.n * (a.output_dt == UZU_DT_F32 ? 4 : 2));
        p.bias = (a.d_transform & UZU_D_BIAS) ? (const __nv_bfloat16*)a.bias : nullptr;
        p.ws = cmd->ctx->splitk_ws; p.counters = cmd->ctx->splitk_counters;
        p.row_bytes = a.k * bits / 8; p.groups = a.k / a.b_group_size;
        p.zp_stride = bits == 4 ? (p.groups + 1) / 2 : p.groups;
        p.xor_mask = a.b_signed_codes ? (bits == 4 ? 0x88888888u : 0x80808080u) : 0u;
        p.steps = a.k / (bits == 4 ? 512u : 256u); p.slice_steps = plan.slice_steps; p.slices = plan.slices; p.whole = plan.whole; p.tiles = (a.n + 15) / 16;
        p.d_is_f32 = a.output_dt == UZU_DT_F32;
        p.accumulate = (a.d_transform & UZU_D_ACCUMULATE) != 0;
        p.has_soft_cap = (a.d_transform & UZU_D_SOFT_CAP) != 0;
        p.ab_scale = ((a.d_transform & UZU_D_SCALE) ? a.ab_scale : 1.0f) / (bits == 4 ? QrShape<4>::DOWN : QrShape<8>::DOWN);
        p.soft_cap = a.soft_cap;
        const uint32_t grid = std::min(p.tiles, (uint32_t)cmd->ctx->sm_count / p.slices) * p.slices;
        if (bits == 4) a.b_group_size == 64 ? qr_method<4, 64>(cmd, p, a.b_prologue, grid, plan.smem) : qr_method<4, 128>(cmd, p, a.b_prologue, grid, plan.smem);
        else a.b_group_size == 64 ? qr_method<8, 64>(cmd, p, a.b_prologue, grid, plan.smem) : qr_method<8, 128>(cmd, p, a.b_prologue, grid, plan.smem);
    }
}

}  // namespace uzu
