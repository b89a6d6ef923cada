// One activation row times a quantised matrix in the decode-stream layout (decode_mega.cu mega_repack: units of 16 rows x 512 nibbles, 4096 bytes of codes in
// the order the lanes read them and 512 bytes of coefficients), with the fusions of uzu_fused_linear_encode. Semantic spec: backends/cpu/kernel/matmul/kernel.rs:164-295.
//
// What bounds it: the bytes of the weights, once nothing else does. A unit is 4608 bytes, 216 SM clocks at 6.2 TB/s over 148 SMs. The kernel before this one
// (matmul.cu's, fed from the same layout) took 610 issue slots a unit, 264 of them on the integer pipe, which takes every other clock: it was bound by that, not
// by memory (asking for its weights ahead of time, into L2, changed nothing).
//   * Codes stay integers: a word of eight nibbles is two registers of bytes (three instructions; bf16 pairs 128 + code took seven), 8-bit codes are taken as they
//     lie, and products run on mma.sync u8 x s8, which has the rate of bf16 per instruction at twice the depth. The row is a 28-bit fixed-point number per element,
//     scaled by the largest exponent of its quantisation group, in four digits of seven bits: one column of the product per digit. A group's two halves of columns
//     keep two groups apart. The integer sums are exact; a pair of digits' sum has up to 24 bits with 4-bit codes, exact in f32 too, and up to 28 with bytes, rounded to
//     24. What a digit cut off at 2^-26 of the group's largest element loses is below the rounding of sums in f32. A row with an infinity or a NaN makes NaN of
//     every output: codes and the zero point, which multiplies the row's sum, are taken apart.
//   * A CTA has 16 warps and whole 16-row tiles; its units lie one behind another in memory and the warps take them in turn, so that each SM reads one
//     contiguous range. A warp copies a unit to registers as soon as it has landed and asks for the next one at once: 74 to 147 KB an SM are on their way. The first
//     half of that is asked for before the kernel waits for its predecessor, the second half behind the row, whose reads would otherwise stand in line for it.
//   * Every unit leaves 16 sums in shared memory; a thread per row adds up its units in order when a batch of tiles is done (one barrier a batch; the bits do not
//     depend on the order of warps).
//   * One CTA an SM. Smaller ones that let the next kernel's in beside them were placed two to an SM here and none there: 362 us a step against 301.
// Llama-3-8B int4 in a decode step, the kernel before / this one, from the end of the launch before: qkv 8.2 / 5.8 us, out 4.3 / 3.7, up 20.3 / 15.5, down 11.7 / 9.2, readout
// (280 MB) 63.7 / 45, of which the step of four layers 362 / 292; Qwen3.5-0.8B's readout (142 MB) 39.7 / 21.6. What is left is the row (up to 3 us in front of the
// first product where a norm is fused) and SMs that finish up to a fifth later than others.
// Every wait is bounded (wait_errors.h).
#include <algorithm>

#include "common.cuh"

namespace uzu {

struct DecodeLinearParams {
    const uint8_t* stream;
    void* d;
    const __nv_bfloat16* bias;
    const __nv_bfloat16 *x, *x2;       // the row; a norm's input and its shortcut, or attention and gate
    __nv_bfloat16* shortcut_out;       // updated residual, written by CTA 0 (null: not)
    const float* norm_scales;
    unsigned int* error;
    uint32_t n, k, C, tiles, pair_tiles, batch;      // batch: tiles (with EPI: of both halves) whose sums are kept until they are added up
    float norm_eps, norm_scale_offset, ab_scale, soft_cap;
    uint32_t norm_residual_add, norm_full_layer, act, d_is_f32, accumulate, has_soft_cap;
};

namespace {

constexpr uint32_t DL_WARPS = 16, DL_THREADS = DL_WARPS * 32, DL_STAGES = 2, DL_UNIT = 4608, DL_SMEM = 226 * 1024;

__device__ __forceinline__ uint32_t dl_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ bool dl_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// false: the copy did not arrive within about a second
__device__ __noinline__ bool dl_wait_long(uint32_t bar, uint32_t parity, unsigned int* error) {
    uint64_t t0, t1;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    for (;;) {
        for (int i = 0; i < 64; ++i)
            if (dl_try(bar, parity)) return true;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
        if (t1 - t0 > 1000000000ull) {
            report_wait_error(error, 0x401u);
            return false;
        }
    }
}
__device__ __forceinline__ bool dl_wait(uint32_t bar, uint32_t parity, unsigned int* error) {
    if (__all_sync(0xffffffffu, dl_try(bar, parity))) return true;
    return __all_sync(0xffffffffu, dl_wait_long(bar, parity, error));
}
__device__ __forceinline__ void dl_copy(uint32_t dst, const void* src, uint32_t bar, uint64_t policy) {
    asm volatile("{ .reg .b64 st; mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1; }" ::"r"(bar), "r"(DL_UNIT) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::"r"(dst), "l"(src), "r"(DL_UNIT), "r"(bar), "l"(policy)
                 : "memory");
}
__device__ __forceinline__ void dl_mma(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float dl_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float dl_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }
__device__ __forceinline__ uint32_t dl_bf2(float a, float b) {
    __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&v);
}

}  // namespace

// PRO: 0 plain row, 1 RMS norm (+ residual add), 3 attention row times sigmoid of its gate; EPI: the rows are [up | gate], D = GatedActMul. Roundings as the
// standalone kernels have them (normalization.rs:50-125, sigmoid_gate.rs:7-22, gated_act_mul/mod.rs:5-12).
template <int NPG, int BITS, bool MLX, int PRO, bool EPI>
__global__ void __launch_bounds__(DL_THREADS, 1) decode_linear_kernel(const DecodeLinearParams p) {
    constexpr uint32_t GPS = 512 / NPG, IPG = NPG / 8;         // groups of a unit; 8-nibble items of a group
    constexpr uint32_t EPT = BITS == 4 ? 8 : 4, NW = EPT / 2;  // elements and words of an item
    constexpr uint32_t XV = BITS == 4 ? 32 : 16;               // vectors of a chunk's digits: [half of the lane's words][t][digit]
    extern __shared__ __align__(128) uint8_t dl_raw[];
    __shared__ __align__(8) uint64_t bars[DL_WARPS * DL_STAGES];
    __shared__ float warp_part[DL_WARPS];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const uint32_t C = p.C, items = C * 64u;
    const uint32_t ring = dl_smem(dl_raw) + warp * (DL_STAGES * DL_UNIT), bar0 = dl_smem(bars) + warp * (DL_STAGES * 8u);
    const uint8_t* ring_p = dl_raw + warp * (DL_STAGES * DL_UNIT);
    uint4* xs = reinterpret_cast<uint4*>(dl_raw + DL_WARPS * DL_STAGES * DL_UNIT);      // digits of the row: [C * 4 chunks][XV] vectors, and two of zeros
    float2* sx = reinterpret_cast<float2*>(xs + C * 4u * XV + 2);                        // [C * GPS]: sum of the row over a group, value of its lowest digit
    float* red = reinterpret_cast<float*>(sx + C * GPS);                                 // [2][batch * C][16]

    // this CTA's tiles (EPI: pairs of tiles; an up tile is followed by its gate tile)
    const uint32_t all = EPI ? p.pair_tiles : p.tiles;
    const uint32_t first = (uint32_t)((uint64_t)blockIdx.x * all / gridDim.x), last = (uint32_t)((uint64_t)(blockIdx.x + 1) * all / gridDim.x);
    const uint32_t vtiles = (last - first) * (EPI ? 2u : 1u), units = vtiles * C;
    uint64_t policy;                                            // weights are read once a token: the small rows stay in L2
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
    if (lane == 0) {
        for (uint32_t s = 0; s < DL_STAGES; ++s) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar0 + 8u * s) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    // the next unit to ask for: its number, tile and place in the tile
    const uint32_t step_t = DL_WARPS / C, step_c = DL_WARPS % C;
    uint32_t iu = warp, ivt = warp / C, ic = warp % C;
    auto ask = [&](uint32_t slot) {
        if (iu < units) {
            const uint32_t tile = EPI ? (ivt & 1u) * p.pair_tiles + first + (ivt >> 1) : first + ivt;
            if (lane == 0) dl_copy(ring + slot * DL_UNIT, p.stream + ((size_t)tile * C + ic) * DL_UNIT, bar0 + 8u * slot, policy);
        }
        iu += DL_WARPS;
        ivt += step_t;
        ic += step_c;
        if (ic >= C) { ic -= C; ++ivt; }
    };
    ask(0);                                                     // the other half when the row has been asked for
    // norm scales are weights too
    constexpr uint32_t PB = 2;                                  // items of a thread whose reads are under way together
    float scales[PRO == 1 ? PB : 1][EPT];
    if constexpr (PRO == 1) {
#pragma unroll
        for (uint32_t u = 0; u < PB; ++u) {
            const uint32_t pos = (tid + u * DL_THREADS) * EPT;
#pragma unroll
            for (uint32_t e = 0; e < EPT; e += 4) {
                float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (pos < p.k) v = __ldg(reinterpret_cast<const float4*>(p.norm_scales + pos + e));
                scales[u][e] = v.x; scales[u][e + 1] = v.y; scales[u][e + 2] = v.z; scales[u][e + 3] = v.w;
            }
        }
    }
    pdl_launch_dependents();
    pdl_wait();

    // ---- the activation row: items of eight nibbles in the order of the products' B operand, and its sums over groups ----
    if (tid < 2) xs[C * 4u * XV + tid] = make_uint4(0, 0, 0, 0);
    auto load = [&](const __nv_bfloat16* src, uint32_t pos, uint32_t (&v)[NW]) {
#pragma unroll
        for (uint32_t i = 0; i < NW; ++i) v[i] = 0;
        if (pos >= p.k) return;
        if constexpr (BITS == 4) {
            const uint4 q = *reinterpret_cast<const uint4*>(src + pos);
            v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
        } else {
            const uint2 q = *reinterpret_cast<const uint2*>(src + pos);
            v[0] = q.x; v[1] = q.y;
        }
    };
    auto put = [&](uint32_t it, const uint32_t (&v)[NW]) {
        float part = 0.0f;
        uint32_t top = 0;
#pragma unroll
        for (uint32_t i = 0; i < NW; ++i) {
            part += dl_lo(v[i]);
            part += dl_hi(v[i]);
            top = max(top, max(v[i] & 0x7fffu, (v[i] >> 16) & 0x7fffu));
        }
#pragma unroll
        for (uint32_t o = 1; o < IPG; o <<= 1) {
            part += __shfl_xor_sync(0xffffffffu, part, o);
            top = max(top, __shfl_xor_sync(0xffffffffu, top, o));
        }
        // |x| < 2^(E + 1) in the group, E its largest exponent: x 2^(25 - E) as an integer, an element 2^18 times smaller than the largest still exact
        const uint32_t e = max(top >> 7, 32u);                  // biased; an infinity or a NaN makes the group's sums NaN, as inf - inf did
        const float up = __uint_as_float((127u + 25u + 127u - min(e, 254u)) << 23), down = e == 255u ? __uint_as_float(0x7fc00000u) : __uint_as_float((e - 25u) << 23);
        if ((it & (IPG - 1)) == 0) sx[it / IPG] = make_float2(part, down);
        uint32_t y[EPT];                                        // digit i is (y >> 7 i & 127) - 64
#pragma unroll
        for (uint32_t i = 0; i < NW; ++i) {
            y[2 * i] = (uint32_t)(__float2int_rn(dl_lo(v[i]) * up) + 0x08102040);
            y[2 * i + 1] = (uint32_t)(__float2int_rn(dl_hi(v[i]) * up) + 0x08102040);
        }
        auto four = [&](uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t digit) {      // digits of four elements
            const uint32_t s = 7u * digit;
            const uint32_t w = (a >> s & 127u) | (b >> s & 127u) << 8 | (c >> s & 127u) << 16 | (d >> s & 127u) << 24;
            return ((w | 0x80808080u) - 0x40404040u) ^ 0x80808080u;
        };
        uint8_t* at = reinterpret_cast<uint8_t*>(xs + (it >> 4) * XV);
        const uint32_t tq = (it >> 2) & 3u, w = it & 3u;
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i) {
            if constexpr (BITS == 4)      // nibbles 0, 2, 4, 6 and 1, 3, 5, 7 of a word are a lane's two registers
                *reinterpret_cast<uint2*>(at + (w >> 1) * 256u + (tq * 4u + i) * 16u + (w & 1u) * 8u) = make_uint2(four(y[0], y[2], y[4], y[6], i), four(y[1], y[3], y[5], y[7], i));
            else
                *reinterpret_cast<uint32_t*>(at + (tq * 4u + i) * 16u + w * 4u) = four(y[0], y[1], y[2], y[3], i);
        }
    };
    auto store = [&](__nv_bfloat16* dst, uint32_t pos, const uint32_t (&v)[NW]) {
        if constexpr (BITS == 4) *reinterpret_cast<uint4*>(dst + pos) = make_uint4(v[0], v[1], v[2], v[3]);
        else *reinterpret_cast<uint2*>(dst + pos) = make_uint2(v[0], v[1]);
    };
    if (tid >= items) ask(1);
    if constexpr (PRO == 1) {
        uint32_t kept[PB][NW];                                  // the first items of a thread; later ones wait in shared memory
        float ssq = 0.0f;
        for (uint32_t it0 = tid; it0 < items; it0 += DL_THREADS * PB) {      // (whole warps: items is a multiple of 64)
            uint32_t a[PB][NW], b[PB][NW];
#pragma unroll
            for (uint32_t u = 0; u < PB; ++u) {
                const uint32_t pos = (it0 + u * DL_THREADS) * EPT;
                load(p.x, pos, a[u]);
                if (p.norm_residual_add) load(p.x2, pos, b[u]);
            }
            if (it0 == tid) ask(1);
#pragma unroll
            for (uint32_t u = 0; u < PB; ++u) {
                const uint32_t it = it0 + u * DL_THREADS;
#pragma unroll
                for (uint32_t i = 0; i < NW; ++i) {
                    if (p.norm_residual_add) a[u][i] = dl_bf2(__fadd_rn(dl_lo(a[u][i]), dl_lo(b[u][i])), __fadd_rn(dl_hi(a[u][i]), dl_hi(b[u][i])));
                    const float lo = dl_lo(a[u][i]), hi = dl_hi(a[u][i]);
                    ssq = __fadd_rn(ssq, __fmul_rn(lo, lo));
                    ssq = __fadd_rn(ssq, __fmul_rn(hi, hi));
                }
                if (it < items && it * EPT < p.k && p.shortcut_out && blockIdx.x == 0) store(p.shortcut_out, it * EPT, a[u]);
                if (it0 == tid) {
#pragma unroll
                    for (uint32_t i = 0; i < NW; ++i) kept[u][i] = a[u][i];
                } else if (it < items) {                        // (the digits of an item take more room than the item, so its own chunk's place holds it)
                    uint4* q = xs + (it >> 4) * XV + (it & 15u);
                    if constexpr (BITS == 4) *q = make_uint4(a[u][0], a[u][1], a[u][2], a[u][3]);
                    else *q = make_uint4(a[u][0], a[u][1], 0, 0);
                }
            }
        }
        ssq = warp_sum(ssq);
        if (lane == 0) warp_part[warp] = ssq;
        __syncthreads();
        float total = 0.0f;
#pragma unroll
        for (uint32_t w = 0; w < DL_WARPS; ++w) total = __fadd_rn(total, warp_part[w]);
        const float rms_inv = __frcp_rn(__fsqrt_rn(__fadd_rn(__fdiv_rn(total, (float)p.k), p.norm_eps)));
        auto norm = [&](uint32_t (&v)[NW], const float* sc) {
#pragma unroll
            for (uint32_t i = 0; i < NW; ++i) {
                float f[2] = {dl_lo(v[i]), dl_hi(v[i])};
#pragma unroll
                for (uint32_t h = 0; h < 2; ++h) {
                    const float normalized = __fmul_rn(f[h], rms_inv), so = __fadd_rn(sc[2 * i + h], p.norm_scale_offset);
                    f[h] = p.norm_full_layer ? __fmul_rn(normalized, so) : __fmul_rn(round_bf16(normalized), round_bf16(so));
                }
                v[i] = dl_bf2(f[0], f[1]);
            }
        };
#pragma unroll
        for (uint32_t u = 0; u < PB; ++u) {
            const uint32_t it = tid + u * DL_THREADS;
            if (it >= items) break;
            if (it * EPT < p.k) norm(kept[u], scales[u]);
            put(it, kept[u]);
        }
        for (uint32_t it = tid + PB * DL_THREADS; it < items; it += DL_THREADS) {
            const uint4 q = xs[(it >> 4) * XV + (it & 15u)];
            __syncwarp();                                       // a chunk's 16 items are one half of a warp's: read before any of them is replaced
            uint32_t v[NW];
            v[0] = q.x; v[1] = q.y;
            if constexpr (BITS == 4) { v[2] = q.z; v[3] = q.w; }
            if (it * EPT < p.k) {
                float sc[EPT];
#pragma unroll
                for (uint32_t e = 0; e < EPT; e += 4) *reinterpret_cast<float4*>(sc + e) = __ldg(reinterpret_cast<const float4*>(p.norm_scales + it * EPT + e));
                norm(v, sc);
            }
            put(it, v);
        }
    } else {
        for (uint32_t it0 = tid; it0 < items; it0 += DL_THREADS * 4) {
            uint32_t a[4][NW], b[PRO == 3 ? 4 : 1][NW];
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u) {
                load(p.x, (it0 + u * DL_THREADS) * EPT, a[u]);
                if constexpr (PRO == 3) load(p.x2, (it0 + u * DL_THREADS) * EPT, b[u]);
            }
            if (it0 == tid) ask(1);
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u) {
                const uint32_t it = it0 + u * DL_THREADS;
                if (it >= items) break;
                if constexpr (PRO == 3) {
                    if (it * EPT < p.k) {
#pragma unroll
                        for (uint32_t i = 0; i < NW; ++i) {
                            const float m0 = __fdiv_rn(1.0f, __fadd_rn(1.0f, expf(-dl_lo(b[u][i])))), m1 = __fdiv_rn(1.0f, __fadd_rn(1.0f, expf(-dl_hi(b[u][i]))));
                            a[u][i] = dl_bf2(__fmul_rn(dl_lo(a[u][i]), m0), __fmul_rn(dl_hi(a[u][i]), m1));
                        }
                    }
                }
                put(it, a[u]);
            }
        }
    }
    __syncthreads();

    // ---- units ----
    const uint32_t digit = g & 3u, h = g >> 2, th = t >> 1;    // the column this lane feeds: a digit of a group; the group of the columns it owns
    const uint4* zero = xs + C * 4u * XV;
    const uint32_t sel = th ? 0x3244u : 0x1044u;               // one of two bf16 as f32 (byte 4: zero)
    const float weight = (t & 1u) ? 16384.0f : 1.0f;           // this lane's columns are digits 0 and 1 or 2 and 3
    bool ok = true;
    uint32_t u = warp, c = warp % C, slot = 0, phase = 0, parity = 0;
    for (uint32_t b0 = 0; b0 < vtiles; b0 += p.batch, parity ^= 1u) {
        const uint32_t b1 = min(vtiles, b0 + p.batch), ub = b0 * C, end = b1 * C;
        float* sums = red + parity * (p.batch * C * 16u);
        for (; u < end; u += DL_WARPS) {
            if (ok && !dl_wait(bar0 + 8u * slot, phase, p.error)) {
                ok = false;                                     // no more copies; the other one may still be on its way to this CTA's shared memory
                if (u + DL_WARPS < units) dl_wait(bar0 + 8u * (slot ^ 1u), phase ^ slot, p.error);
            }
            const uint4* sw = reinterpret_cast<const uint4*>(ring_p + slot * DL_UNIT) + lane;
            const uint4* co = reinterpret_cast<const uint4*>(ring_p + slot * DL_UNIT + 4096) + g;
            uint4 wa[4], wb[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) { wa[j] = sw[j * 32]; wb[j] = sw[(4 + j) * 32]; }
            const uint4 sa = co[0], sb = co[8], za = co[16], zb = co[24];      // scales and zero points / biases of rows g and g + 8, all groups
            __syncwarp();                                       // every lane has read the unit: its place is free
            if (ok) {
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                ask(slot);
            }
            int d[GPS / 2][4];
#pragma unroll
            for (uint32_t i = 0; i < GPS / 2; ++i) d[i][0] = d[i][1] = d[i][2] = d[i][3] = 0;
            const uint4* xc = xs + c * 4u * XV + t * 4u + digit;
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) {
                const bool feeds = NPG == 64 ? th == h : (j & 1u) == h;
                const uint4* xp = feeds ? xc + j * XV : zero;
                const uint32_t av[4] = {wa[j].x, wa[j].y, wa[j].z, wa[j].w}, bv[4] = {wb[j].x, wb[j].y, wb[j].z, wb[j].w};
                int (&dj)[4] = d[NPG == 64 ? j : j >> 1];
                if constexpr (BITS == 4) {
#pragma unroll
                    for (int w = 0; w < 4; w += 2) {
                        const uint4 x = xp[feeds ? w * 8 : 0];
                        dl_mma(dj, av[w] & 0x0f0f0f0fu, bv[w] & 0x0f0f0f0fu, (av[w] >> 4) & 0x0f0f0f0fu, (bv[w] >> 4) & 0x0f0f0f0fu, x.x, x.y);
                        dl_mma(dj, av[w + 1] & 0x0f0f0f0fu, bv[w + 1] & 0x0f0f0f0fu, (av[w + 1] >> 4) & 0x0f0f0f0fu, (bv[w + 1] >> 4) & 0x0f0f0f0fu, x.z, x.w);
                    }
                } else {
                    const uint4 x = xp[0];
                    dl_mma(dj, av[0], bv[0], av[1], bv[1], x.x, x.y);
                    dl_mma(dj, av[2], bv[2], av[3], bv[3], x.z, x.w);
                }
            }
            // this lane's two columns are two digits of group 2 i + th, rows g (0, 1) and g + 8 (2, 3)
            float ra = 0.0f, rb = 0.0f;
#pragma unroll
            for (uint32_t i = 0; i < GPS / 2; ++i) {
                const float2 s2 = sx[c * GPS + 2 * i + th];
                const uint32_t sav[4] = {sa.x, sa.y, sa.z, sa.w}, sbv[4] = {sb.x, sb.y, sb.z, sb.w}, zav[4] = {za.x, za.y, za.z, za.w}, zbv[4] = {zb.x, zb.y, zb.z, zb.w};
                const float unit = s2.y * weight, sum = (t & 1u) ? 0.0f : s2.x;
                const float va = unit * (float)(d[i][0] + d[i][1] * 128), vb = unit * (float)(d[i][2] + d[i][3] * 128);
                const float ca = __uint_as_float(__byte_perm(zav[i], 0, sel)), cb = __uint_as_float(__byte_perm(zbv[i], 0, sel));
                const float fa = __uint_as_float(__byte_perm(sav[i], 0, sel)), fb = __uint_as_float(__byte_perm(sbv[i], 0, sel));
                if constexpr (MLX) {
                    ra += fa * va + ca * sum;
                    rb += fb * vb + cb * sum;
                } else {
                    ra += fa * (va - ca * sum);
                    rb += fb * (vb - cb * sum);
                }
            }
            ra += __shfl_xor_sync(0xffffffffu, ra, 1);
            rb += __shfl_xor_sync(0xffffffffu, rb, 1);
            ra += __shfl_xor_sync(0xffffffffu, ra, 2);
            rb += __shfl_xor_sync(0xffffffffu, rb, 2);
            if (t < 2) sums[(u - ub) * 16u + t * 8u + g] = t ? rb : ra;
            c += step_c;
            if (c >= C) c -= C;
            slot ^= 1u;
            phase ^= slot ^ 1u;                                 // (two stages: the phase turns with every second unit)
        }
        __syncthreads();
        // ---- rows of the batch (its sums are written again only behind the next barrier) ----
        auto row_sum = [&](uint32_t tile, uint32_t r) {
            const float* q = sums + (size_t)tile * C * 16u + r;
            float s = 0.0f;
            for (uint32_t i = 0; i < C; ++i) s += q[i * 16u];
            return s;
        };
        if constexpr (EPI) {
            for (uint32_t idx = tid; idx < (b1 - b0) * 8u; idx += DL_THREADS) {
                const uint32_t pair = idx >> 4, r = idx & 15u, row = (first + (b0 >> 1) + pair) * 16u + r;
                float up = p.ab_scale * row_sum(2 * pair, r), gate = p.ab_scale * row_sum(2 * pair + 1, r);
                if (p.bias) { up += bf2f(p.bias[row]); gate += bf2f(p.bias[row + p.pair_tiles * 16u]); }
                up = round_bf16(up);
                gate = round_bf16(gate);
                reinterpret_cast<__nv_bfloat16*>(p.d)[row] = f2bf(__fmul_rn(up, round_bf16(act_f32_nofma(p.act, gate))));
            }
        } else {
            for (uint32_t idx = tid; idx < (b1 - b0) * 16u; idx += DL_THREADS) {
                const uint32_t r = idx & 15u, row = (first + b0 + (idx >> 4)) * 16u + r;
                if (row >= p.n) continue;
                float value = p.ab_scale * row_sum(idx >> 4, r);
                if (p.accumulate) value += p.d_is_f32 ? reinterpret_cast<const float*>(p.d)[row] : bf2f(reinterpret_cast<const __nv_bfloat16*>(p.d)[row]);
                if (p.bias) value += bf2f(p.bias[row]);
                if (p.has_soft_cap) value = p.soft_cap * tanhf(value / p.soft_cap);
                if (p.d_is_f32) reinterpret_cast<float*>(p.d)[row] = value;
                else reinterpret_cast<__nv_bfloat16*>(p.d)[row] = f2bf(value);
            }
        }
    }
}

// ---------------------------------------------------------------------------------------------------------------------------------
// host
// ---------------------------------------------------------------------------------------------------------------------------------
static size_t decode_linear_smem(uint32_t C, uint32_t bits, uint32_t gps, uint32_t batch) {
    return (size_t)DL_WARPS * DL_STAGES * DL_UNIT + ((size_t)C * 4 * (bits == 4 ? 32 : 16) + 2) * 16 + (size_t)C * gps * 8 + 2ull * batch * C * 64;
}

template <int NPG, int BITS, bool MLX, int PRO, bool EPI>
static void launch_decode_linear(uzu_command_buffer* cmd, const DecodeLinearParams& p, uint32_t grid, size_t smem) {
    static std::atomic<uint64_t> opted{0};
    opt_in_dynamic_smem(cmd, decode_linear_kernel<NPG, BITS, MLX, PRO, EPI>, DL_SMEM, opted);
    launch(cmd, "decode_linear_kernel", decode_linear_kernel<NPG, BITS, MLX, PRO, EPI>, dim3(grid), dim3(DL_THREADS), smem, p);
}
template <int NPG, int BITS, bool MLX>
static void launch_decode_linear_f(uzu_command_buffer* cmd, const DecodeLinearParams& p, uint32_t prologue, bool gated, uint32_t grid, size_t smem) {
    if (prologue == 0 && !gated) launch_decode_linear<NPG, BITS, MLX, 0, false>(cmd, p, grid, smem);
    else if (prologue == 0) launch_decode_linear<NPG, BITS, MLX, 0, true>(cmd, p, grid, smem);
    else if (prologue == 1 && !gated) launch_decode_linear<NPG, BITS, MLX, 1, false>(cmd, p, grid, smem);
    else if (prologue == 1) launch_decode_linear<NPG, BITS, MLX, 1, true>(cmd, p, grid, smem);
    else launch_decode_linear<NPG, BITS, MLX, 3, false>(cmd, p, grid, smem);
}

static uint32_t decode_linear_batch(uint32_t C, bool gated) {
    const uint32_t tiles = std::max(64u / C, 1u);
    return gated ? std::max(tiles & ~1u, 2u) : tiles;
}

// a call that the other conditions of a fused linear hold for: its matrix in a decode stream, the row and the sums in shared memory (4-bit rows of up to 16384)
bool decode_linear_applicable(const uzu_fused_linear_args& f) {
    const uzu_matmul_args& a = f.matmul;
    const uint32_t bits = a.b_mode == UZU_QMODE_U4 ? 4 : 8, npg = a.b_group_size * bits / 4, C = (a.k * bits / 4 + 511) / 512;
    if (!f.decode_stream || a.m != 1 || a.b_mode == UZU_QMODE_I8 || a.b_signed_codes || !(npg == 128 || (npg == 64 && bits == 4)) || a.k % 8) return false;
    return decode_linear_smem(C, bits, 512 / npg, decode_linear_batch(C, f.epilogue == 1)) <= DL_SMEM;
}

void encode_decode_linear(uzu_command_buffer* cmd, const uzu_fused_linear_args& f) {
    const uzu_matmul_args& a = f.matmul;
    const uint32_t bits = a.b_mode == UZU_QMODE_U4 ? 4 : 8, npg = a.b_group_size * bits / 4;
    DecodeLinearParams p{};
    p.stream = (const uint8_t*)f.decode_stream;
    p.d = (void*)a.d;
    p.bias = (a.d_transform & UZU_D_BIAS) ? (const __nv_bfloat16*)a.bias : nullptr;
    p.error = cmd->ctx->wait_errors.device_word;
    p.n = a.n; p.k = a.k;
    p.C = (a.k * bits / 4 + 511) / 512;
    p.tiles = (a.n + 15) / 16;
    p.pair_tiles = a.n / 32;
    p.ab_scale = (a.d_transform & UZU_D_SCALE) ? a.ab_scale : 1.0f;
    p.soft_cap = a.soft_cap;
    p.has_soft_cap = (a.d_transform & UZU_D_SOFT_CAP) != 0;
    p.accumulate = (a.d_transform & UZU_D_ACCUMULATE) != 0;
    p.d_is_f32 = a.output_dt == UZU_DT_F32;
    p.act = f.act_type;
    if (f.prologue == 1) {
        p.x = (const __nv_bfloat16*)f.norm_input;
        p.x2 = (const __nv_bfloat16*)f.norm_shortcut_in;
        p.shortcut_out = (__nv_bfloat16*)f.shortcut_out;
        p.norm_scales = (const float*)f.norm_scales;
        p.norm_eps = f.norm_epsilon; p.norm_scale_offset = f.norm_scale_offset;
        p.norm_residual_add = f.norm_residual_add; p.norm_full_layer = f.norm_full_layer;
    } else if (f.prologue == 3) {
        p.x = (const __nv_bfloat16*)f.sg_attn;
        p.x2 = (const __nv_bfloat16*)f.sg_gate;
    } else {
        p.x = (const __nv_bfloat16*)a.a;
    }
    const bool gated = f.epilogue == 1, mlx = a.b_prologue == UZU_B_SCALE_BIAS_DEQUANT;
    p.batch = decode_linear_batch(p.C, gated);
    const size_t smem = decode_linear_smem(p.C, bits, 512 / npg, p.batch);
    const uint32_t grid = std::min<uint32_t>((uint32_t)cmd->ctx->sm_count, gated ? p.pair_tiles : p.tiles);
#define UZU_DL(NPG_, BITS_)                                                                                             \
    if (npg == NPG_ && bits == BITS_) {                                                                                 \
        if (mlx) launch_decode_linear_f<NPG_, BITS_, true>(cmd, p, f.prologue, gated, grid, smem);                      \
        else launch_decode_linear_f<NPG_, BITS_, false>(cmd, p, f.prologue, gated, grid, smem);                         \
        return;                                                                                                         \
    }
    UZU_DL(64, 4)
    UZU_DL(128, 4)
    UZU_DL(128, 8)
#undef UZU_DL
}

}  // namespace uzu
