// One decoded row a sequence, from the projected row to the attention output: QKVNorm, RoPE, the new key and value into the cache, and attention over it, one launch.
// Specs: backends/cpu/kernel/attention/{qkv_norm.rs:7-35, attention_prepare.rs:7-126, attention_single_pass.rs:49-126}.
//
// What bounds it: the way through it. Its keys and values are 8 MB at 2048 tokens of eight heads, 1.3 us of memory, but the two kernels before this one took
// 18.5 us a layer from the end of the projection (rows of the cache one after another through shuffles and f32 multiply-adds, 2300 instructions a warp; partial results
// through global memory and a ticket).
//   * A warp takes tiles of 16 keys. Scores and the weighted sum are products on mma.sync: the heads of a key head are rows 0..7 of the product, the exact f32
//     probabilities three bf16 planes, two of them in rows g and g + 8 of one product and the third in a second one. Keys go from memory to registers in the
//     order of the product's B operand (channels are permuted alike in the query), values are paired by PRMT; neither passes through shared memory.
//   * The pipe cuts what it adds to an accumulator off at its last bit: a chain is 32 channels of a score or one tile's products, the smallest plane first, and chains
//     are added by rounded additions. As many results are off the correct rounding as on the split-KV kernel, all f32 (1 to 2.5 in 10000); with whole chains up to twice
//     as many, in the same time.
//   * The position and a warp's first tile are read before the kernel waits for its predecessor: what earlier steps wrote is there already, since a step's first
//     kernel is an ordinary launch (uzu_command_buffer::dependent).
//   * A cluster of up to eight CTAs shares a key head's keys, each 128 and more; the parts meet in distributed shared memory, in rank order.
// (Heads of 256 spill 110 to 160 bytes a thread.)
// From the end of the projection, Llama-3-8B at 2048 tokens: 18.5 us a layer before, 8.6 now; Qwen3.5-0.8B at 500 (heads of 256, normed): 22, 10.8. What is left are some
// 2000 instructions of eight warps, one after another, and the trips to the row, to distributed shared memory and back.
#include <algorithm>

#include "common.cuh"

namespace uzu {

struct DecodeAttnParams {
    uint64_t qkv, out, positions;      // positions: device words, one a sequence, or null (then the sequences' own)
    uint64_t cosines, sines;           // [positions][rope_dim] or null
    uint32_t rope_dim, num_heads, num_kv_heads, heads, groups, ranks;      // heads: query heads of a CTA's rows; groups: CTAs of a key head side by side
    uint32_t kv_stride;                // elements between cached tokens
    float scale;
    uzu_qk_norm_config q_norm, k_norm;
};

namespace {

constexpr uint32_t DA_WARPS = 8, DA_THREADS = DA_WARPS * 32, DA_RANK_KEYS = 128;

__device__ __forceinline__ void da_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t da_bf2(float a, float b) {
    __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float da_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float da_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }
__device__ __forceinline__ uint32_t da_word(const uint4& v, uint32_t i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }
__device__ __forceinline__ float da_weight(float m, float top) { return m == -INFINITY ? 0.0f : expf(m - top); }
__device__ __forceinline__ uint32_t da_remote(const void* p, uint32_t rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ void da_store_remote(uint32_t addr, float v) { asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory"); }

// a warp's tiles of one head, key by key in f32: its sums to `out`, the maximum and the sum of the weights returned (not part of the kernel's body: its registers)
template <int D>
__device__ __noinline__ float2 da_key_by_key(const __nv_bfloat16* query, const __nv_bfloat16* fresh, const __nv_bfloat16* keys, const __nv_bfloat16* values, uint32_t stride, uint32_t position,
                                             uint32_t first, uint32_t step, float scale, float* out) {
    const uint32_t lane = threadIdx.x & 31;
    float acc[D / 32], most = -INFINITY, total = 0.0f;
#pragma unroll
    for (uint32_t i = 0; i < D / 32; ++i) acc[i] = 0.0f;
#pragma unroll 1
    for (uint32_t tile = first; tile * 16 <= position; tile += step) {
#pragma unroll 1
        for (uint32_t key = tile * 16; key <= min(tile * 16 + 15, position); ++key) {
            const __nv_bfloat16* k = (key == position ? fresh : keys + (size_t)key * stride) + lane;
            const __nv_bfloat16* v = (key == position ? fresh + D : values + (size_t)key * stride) + lane;
            float score = 0.0f;
            for (uint32_t i = 0; i < D / 32; ++i) score = fmaf(bf2f(query[lane + 32 * i]), bf2f(k[32 * i]), score);
            score = scale * warp_sum(score);
            const float next = fmaxf(most, score), keep = da_weight(most, next), weight = da_weight(score, next);
            total = total * keep + weight;
            most = next;
#pragma unroll
            for (uint32_t i = 0; i < D / 32; ++i) acc[i] = fmaf(weight, bf2f(v[32 * i]), acc[i] * keep);
        }
    }
    __syncwarp();
#pragma unroll
    for (uint32_t i = 0; i < D / 32; ++i) out[lane + 32 * i] = acc[i];
    return make_float2(most, total);
}

}  // namespace

// grid: (ranks, key heads * groups, sequences), a cluster per key head, group and sequence
// FEW: at most four heads. Rows g and g + 4 of the query are then the same head, so that its three planes are rows g, g + 8 and g + 4 of one product.
template <int D, bool FEW>
__global__ void __launch_bounds__(DA_THREADS, 1) decode_attention_kernel(const __grid_constant__ DecodeAttnParams p, const __grid_constant__ AttnSequences seqs) {
    constexpr uint32_t KB = D / 32, VB = D / 64, PER = D / 32;      // 16-byte blocks of a lane: of a key, of a value; elements of a lane of a row
    constexpr bool kRoomy = D <= 128;                                // registers for values beside keys; else values are asked for into L2, and read half by half
    extern __shared__ __align__(16) uint8_t da_raw[];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const uint32_t rank = blockIdx.x, kv_head = blockIdx.y / p.groups, head0 = kv_head * (p.num_heads / p.num_kv_heads) + blockIdx.y % p.groups * p.heads, b = blockIdx.z, G = p.heads;
    __nv_bfloat16* rows = reinterpret_cast<__nv_bfloat16*>(da_raw);                       // [G] queries, the new key, the new value
    float* parts = reinterpret_cast<float*>(rows + (G + 2) * D);                          // [warps][G][D]
    float* part_ml = parts + DA_WARPS * G * D;                                            // [warps][G][2]
    float* weights = part_ml + DA_WARPS * G * 2;                                          // [warps][G]
    float* all_ml = weights + DA_WARPS * G;                                               // [ranks][G][2]: of the cluster
    float* slices = all_ml + ((p.ranks * G * 2 + 3u) & ~3u);                               // [ranks][slice]: this rank's outputs, of every rank

    // (a word that only the last kernel of a step writes: it is there before the second kernel of this step starts, since the first is an ordinary launch)
    // (asm: of a plain load and the parameter the compiler makes one load from either address, and a parameter has none that such a load may take)
    uint32_t position = seqs.prefix[b], rope_row = seqs.position[b];
    if (p.positions) {
        asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(position) : "l"(p.positions + 4ull * b) : "memory");
        rope_row = position;
    }
    const uint32_t length = position + 1;
    const uint32_t used = min(p.ranks, (length + DA_RANK_KEYS - 1) / DA_RANK_KEYS);       // by its own length alone: a sequence's bits do not depend on its neighbours
    const uint32_t slice = ((G * D + used - 1) / used + 3u) & ~3u, tiles = (length + 15) / 16, last_tile = tiles - 1;
    const uint32_t first = rank < used ? rank * DA_WARPS + warp : tiles, step = used * DA_WARPS;
    const bool owner = rank < used && last_tile % step / DA_WARPS == rank;                // its last tile holds the new key
    const __nv_bfloat16* keys = reinterpret_cast<const __nv_bfloat16*>(seqs.keys[b]) + (size_t)kv_head * D;
    const __nv_bfloat16* values = reinterpret_cast<const __nv_bfloat16*>(seqs.values[b]) + (size_t)kv_head * D;

    constexpr uint32_t VR = kRoomy ? VB : VB / 2;                    // blocks of a value that are read at a time
    uint4 kk[2][KB], vv[4][VR];
    // keys g and g + 8 of a tile, channels 32 i + 8 t; values 2t, 2t + 1, 2t + 8 and 2t + 9, channels 64 i + 8 g. The new token's come from shared memory.
    auto read_keys = [&](uint32_t tile) {
#pragma unroll
        for (uint32_t n = 0; n < 2; ++n) {
            const uint32_t key = tile * 16 + n * 8 + g;
            const __nv_bfloat16* src = (key == position ? rows + G * D : keys + (size_t)key * p.kv_stride) + t * 8;
#pragma unroll
            for (uint32_t i = 0; i < KB; ++i) kk[n][i] = key < length ? *reinterpret_cast<const uint4*>(src + i * 32) : make_uint4(0, 0, 0, 0);
        }
    };
    auto read_values = [&](uint32_t tile, uint32_t from, uint32_t count) {
#pragma unroll
        for (uint32_t n = 0; n < 4; ++n) {
            const uint32_t key = tile * 16 + 2 * t + (n & 1u) + (n >> 1) * 8;
            const __nv_bfloat16* src = (key == position ? rows + (G + 1) * D : values + (size_t)key * p.kv_stride) + g * 8;
#pragma unroll
            for (uint32_t i = 0; i < VB; ++i)
                if (i >= from && i < from + count) vv[n][i % VR] = key < length ? *reinterpret_cast<const uint4*>(src + i * 64) : make_uint4(0, 0, 0, 0);
        }
    };
    const bool early = first < last_tile;      // (the last tile may hold the new key)
    if (early) {
        read_keys(first);
        if constexpr (kRoomy) read_values(first, 0, VR);
        else if (lane < 16) {
#pragma unroll
            for (uint32_t i = 0; i < D; i += 64) asm volatile("prefetch.global.L2 [%0];" ::"l"(values + (size_t)(first * 16 + lane) * p.kv_stride + i));
        }
    }
    // the lane's rotation factors: channels lane + 32 i
    float cs[PER], sn[PER];
    const uint32_t half = p.rope_dim / 2;
#pragma unroll
    for (uint32_t i = 0; i < PER; ++i) {
        const uint32_t d = lane + 32 * i;
        cs[i] = d < p.rope_dim ? __ldg(reinterpret_cast<const float*>(p.cosines) + (size_t)rope_row * p.rope_dim + d) : 1.0f;
        sn[i] = d < p.rope_dim ? __ldg(reinterpret_cast<const float*>(p.sines) + (size_t)rope_row * p.rope_dim + d) : 0.0f;
    }
    // and the norms' scales: of queries (a warp's rows are queries but for one), the other row's are read where they are needed
    float qs[PER];
#pragma unroll
    for (uint32_t i = 0; i < PER; ++i) qs[i] = p.q_norm.present && p.q_norm.has_scales ? __ldg(reinterpret_cast<const float*>(p.q_norm.scales) + lane + 32 * i) : 0.0f;
    if (owner && warp == G % DA_WARPS && p.k_norm.present && p.k_norm.has_scales) asm volatile("prefetch.global.L2 [%0];" ::"l"(p.k_norm.scales + 4ull * lane * PER));
    pdl_launch_dependents();
    if (p.ranks > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");      // (every CTA of the cluster runs before another one stores to it)
    pdl_wait();

    // ---- queries, and in the owner the new key and value: a warp a row; roundings as the kernels of single operations have them ----
    const uint32_t total = p.num_heads + 2 * p.num_kv_heads;
    const __nv_bfloat16* qkv = reinterpret_cast<const __nv_bfloat16*>(p.qkv) + (size_t)b * total * D;
    for (uint32_t r = warp; r < (owner ? G + 2 : rank < used ? G : 0u); r += DA_WARPS) {
        const bool is_query = r < G, is_value = r == G + 1;
        const uint32_t head = is_query ? head0 + r : is_value ? p.num_heads + p.num_kv_heads + kv_head : p.num_heads + kv_head;
        const uzu_qk_norm_config& nc = is_query ? p.q_norm : p.k_norm;
        const __nv_bfloat16* src = qkv + (size_t)head * D;
        __nv_bfloat16* dst = rows + r * D;
        __nv_bfloat16 e[PER];
#pragma unroll
        for (uint32_t i = 0; i < PER; ++i) e[i] = src[lane + 32 * i];
        if (!is_value && nc.present) {
            float sum = 0.0f;
#pragma unroll
            for (uint32_t i = 0; i < PER; ++i) sum = __fadd_rn(sum, __fmul_rn(bf2f(e[i]), bf2f(e[i])));
            sum = warp_sum(sum);
            const float inv = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(sum, (float)D), nc.epsilon)));
            const float* scales = reinterpret_cast<const float*>(nc.scales);
#pragma unroll
            for (uint32_t i = 0; i < PER; ++i) {
                const float normalized = __fmul_rn(bf2f(e[i]), inv);
                if (!nc.has_scales) e[i] = f2bf(normalized);
                else {
                    const float so = __fadd_rn(is_query ? qs[i] : scales[lane + 32 * i], nc.scale_offset);
                    e[i] = f2bf(nc.full_layer ? __fmul_rn(normalized, so) : __fmul_rn(round_bf16(normalized), round_bf16(so)));
                }
            }
        }
        if (!is_value && p.rope_dim) {      // the other half's channel is a lane's own where a half is a multiple of 32, else in shared memory
#pragma unroll
            for (uint32_t i = 0; i < PER; ++i) dst[lane + 32 * i] = e[i];
            __syncwarp();
            __nv_bfloat16 other[PER];
#pragma unroll
            for (uint32_t i = 0; i < PER; ++i) {
                const uint32_t d = lane + 32 * i;
                other[i] = d < p.rope_dim ? dst[d < half ? d + half : d - half] : e[i];
            }
            __syncwarp();
#pragma unroll
            for (uint32_t i = 0; i < PER; ++i) {
                const uint32_t d = lane + 32 * i;
                const float pv = bf2f(other[i]);
                if (d < p.rope_dim) e[i] = f2bf(__fadd_rn(__fmul_rn(bf2f(e[i]), cs[i]), __fmul_rn(d < half ? -pv : pv, sn[i])));
            }
        }
#pragma unroll
        for (uint32_t i = 0; i < PER; ++i) dst[lane + 32 * i] = e[i];
        if (!is_query && blockIdx.y % p.groups == 0) {      // into the cache
            __nv_bfloat16* cache = const_cast<__nv_bfloat16*>(is_value ? values : keys) + (size_t)position * p.kv_stride;
#pragma unroll
            for (uint32_t i = 0; i < PER; ++i) cache[lane + 32 * i] = e[i];
        }
    }
    __syncthreads();

    // ---- a warp's tiles ----
    const uint32_t head = FEW ? g & 3u : g;      // of this lane's rows
    auto query = [&](uint32_t i) { return head < G ? *reinterpret_cast<const uint4*>(rows + head * D + i * 32 + t * 8) : make_uint4(0, 0, 0, 0); };
    uint4 q[D == 64 ? KB : 1];
    if constexpr (D == 64) {
#pragma unroll
        for (uint32_t i = 0; i < KB; ++i) q[i] = query(i);
    }
    float m = -INFINITY, l = 0.0f;      // of the lane's head
    float o[VB * 8][4];                 // channels 64 i + 16 t + j and 64 i + 16 t + 8 + j of the lane's planes
#pragma unroll
    for (uint32_t i = 0; i < VB * 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.0f;
    if (!early && first < tiles) {
        read_keys(first);
        if constexpr (kRoomy) read_values(first, 0, VR);
    }
    for (uint32_t tile = first; tile < tiles; tile += step) {
        float s[2][2] = {{0.0f, 0.0f}, {0.0f, 0.0f}};
#pragma unroll
        for (uint32_t i = 0; i < KB; ++i) {
            uint4 qi;
            if constexpr (D == 64) qi = q[i];
            else qi = query(i);
#pragma unroll
            for (uint32_t n = 0; n < 2; ++n) {
                float part[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                da_mma(part, qi.x, 0, qi.y, 0, kk[n][i].x, kk[n][i].y);
                da_mma(part, qi.z, 0, qi.w, 0, kk[n][i].z, kk[n][i].w);
                s[n][0] += part[0];
                s[n][1] += part[1];
            }
        }
        if constexpr (!kRoomy) read_values(tile, 0, VR);
        else if (tile + step < tiles) read_keys(tile + step);
        float pr[4];      // keys 2t, 2t + 1, 2t + 8, 2t + 9
#pragma unroll
        for (uint32_t n = 0; n < 4; ++n) pr[n] = tile * 16 + 2 * t + (n & 1u) + (n >> 1) * 8 < length ? p.scale * s[n >> 1][n & 1u] : -INFINITY;
        float top = fmaxf(fmaxf(pr[0], pr[1]), fmaxf(pr[2], pr[3]));
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
        const float m_new = fmaxf(m, top), factor = da_weight(m, m_new);
        m = m_new;
        l *= factor;
#pragma unroll
        for (uint32_t n = 0; n < 4; ++n) {
            pr[n] = da_weight(pr[n], m);
            l += pr[n];                                     // (this lane's keys; the quad's meet at the end)
        }
        uint32_t plane[3][2];
#pragma unroll
        for (uint32_t i = 0; i < 3; ++i) {
#pragma unroll
            for (uint32_t n = 0; n < 2; ++n) {
                plane[i][n] = da_bf2(pr[2 * n], pr[2 * n + 1]);
                pr[2 * n] -= da_lo(plane[i][n]);
                pr[2 * n + 1] -= da_hi(plane[i][n]);
            }
        }
        uint32_t a[4] = {plane[0][0], plane[1][0], plane[0][1], plane[1][1]};
        if (FEW && g >= 4) { a[0] = plane[2][0]; a[2] = plane[2][1]; a[1] = a[3] = 0; }
#pragma unroll
        for (uint32_t i = 0; i < VB; ++i) {
#pragma unroll
            for (uint32_t j = 0; j < 8; ++j) {
                const uint32_t sel = j & 1u ? 0x7632u : 0x5410u;
                const uint32_t b0 = __byte_perm(da_word(vv[0][i % VR], j / 2), da_word(vv[1][i % VR], j / 2), sel), b1 = __byte_perm(da_word(vv[2][i % VR], j / 2), da_word(vv[3][i % VR], j / 2), sel);
                float part[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                if constexpr (!FEW) da_mma(part, plane[2][0], 0, plane[2][1], 0, b0, b1);
                da_mma(part, a[0], a[1], a[2], a[3], b0, b1);
#pragma unroll
                for (uint32_t c = 0; c < 4; ++c) o[i * 8 + j][c] = fmaf(o[i * 8 + j][c], factor, part[c]);
            }
            if (i + VR < VB) read_values(tile, i + VR, 1);
        }
        if (tile + step < tiles) {
            if constexpr (kRoomy) read_values(tile + step, 0, VR);
            else read_keys(tile + step);
        }
    }
    l += __shfl_xor_sync(0xffffffffu, l, 1);
    l += __shfl_xor_sync(0xffffffffu, l, 2);

    // ---- the warps' parts ----
    if (first < tiles) {
        float* dst = parts + (warp * G + head) * D;
        float probe = 0.0f;      // stays zero while everything is finite
#pragma unroll
        for (uint32_t i = 0; i < VB; ++i) {
#pragma unroll
            for (uint32_t c = 0; c < 2; ++c) {
                float v[8];
#pragma unroll
                for (uint32_t j = 0; j < 8; ++j) {
                    v[j] = o[i * 8 + j][c] + o[i * 8 + j][2 + c];
                    if constexpr (FEW) v[j] += __shfl_xor_sync(0xffffffffu, v[j], 16);
                }
                if (g < G) {
#pragma unroll
                    for (uint32_t j = 0; j < 8; ++j) probe = fmaf(v[j], 0.0f, probe);
                    *reinterpret_cast<float4*>(dst + 64 * i + 16 * t + 8 * c) = make_float4(v[0], v[1], v[2], v[3]);
                    *reinterpret_cast<float4*>(dst + 64 * i + 16 * t + 8 * c + 4) = make_float4(v[4], v[5], v[6], v[7]);
                }
            }
        }
        // A value that is not finite makes NaN of a weight's plane that is zero. Where sums are not finite and weights are, the warp's keys are taken one after another
        // in f32, and what is not finite comes out as the products make it.
        if (!__all_sync(0xffffffffu, probe == 0.0f)) {
            for (uint32_t h = 0; h < G; ++h) {
                if (!(__shfl_sync(0xffffffffu, l, h * 4) < INFINITY)) continue;
                const float2 ml = da_key_by_key<D>(rows + h * D, rows + G * D, keys, values, p.kv_stride, position, first, step, p.scale, parts + (warp * G + h) * D);
                if (g == h) { m = ml.x; l = ml.y; }
            }
        }
    }
    if (g < G && t == 0) {
        part_ml[(warp * G + g) * 2] = m;
        part_ml[(warp * G + g) * 2 + 1] = l;
    }
    __syncthreads();
    if (tid < DA_WARPS * G) {
        const uint32_t h = tid % G;
        float top = -INFINITY;
#pragma unroll
        for (uint32_t w = 0; w < DA_WARPS; ++w) top = fmaxf(top, part_ml[(w * G + h) * 2]);
        weights[tid] = da_weight(part_ml[tid * 2], top);
    }
    __syncthreads();
    if (p.ranks > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(p.out) + ((size_t)b * p.num_heads + head0) * D;
    if (rank < used) {
        auto sum_of = [&](uint32_t h) {
            float sum = 0.0f;
#pragma unroll
            for (uint32_t w = 0; w < DA_WARPS; ++w) sum += weights[w * G + h] * part_ml[(w * G + h) * 2 + 1];
            return sum;
        };
        if (used > 1 && tid < used * G) {
            const uint32_t h = tid % G, at = da_remote(all_ml + (rank * G + h) * 2, tid / G);
            float top = -INFINITY;
#pragma unroll
            for (uint32_t w = 0; w < DA_WARPS; ++w) top = fmaxf(top, part_ml[(w * G + h) * 2]);
            da_store_remote(at, top);
            da_store_remote(at + 4, sum_of(h));
        }
        for (uint32_t idx = tid * 4; idx < G * D; idx += DA_THREADS * 4) {      // (a slice is a multiple of four)
            const uint32_t h = idx / D;
            float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (uint32_t w = 0; w < DA_WARPS; ++w) {
                const float weight = weights[w * G + h];
                const float4 q4 = *reinterpret_cast<const float4*>(parts + w * G * D + idx);
                if (weight != 0.0f) { v[0] += weight * q4.x; v[1] += weight * q4.y; v[2] += weight * q4.z; v[3] += weight * q4.w; }      // (a warp without a tile has written none)
            }
            if (used == 1) {
                const float sum = sum_of(h);
                *reinterpret_cast<uint2*>(out + idx) = make_uint2(da_bf2(v[0] / sum, v[1] / sum), da_bf2(v[2] / sum, v[3] / sum));
            } else {
                const uint32_t at = da_remote(slices + rank * slice + idx % slice, idx / slice);
                asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(at), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]) : "memory");
            }
        }
    }
    if (p.ranks == 1) return;
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (used == 1 || rank >= used) return;
    for (uint32_t i = tid; i < slice && rank * slice + i < G * D; i += DA_THREADS) {
        const uint32_t idx = rank * slice + i, h = idx / D;
        float top = -INFINITY, sum = 0.0f, v = 0.0f;
        for (uint32_t r = 0; r < used; ++r) top = fmaxf(top, all_ml[(r * G + h) * 2]);
        for (uint32_t r = 0; r < used; ++r) {
            const float weight = da_weight(all_ml[(r * G + h) * 2], top);
            sum += weight * all_ml[(r * G + h) * 2 + 1];
            v += weight * slices[r * slice + i];
        }
        out[idx] = f2bf(v / sum);
    }
}

// ---------------------------------------------------------------------------------------------------------------------------------
// host
// ---------------------------------------------------------------------------------------------------------------------------------
// query heads of a CTA: all of a key head's, or the largest divisor of them up to eight
static uint32_t decode_attention_heads(uint32_t gqa) {
    uint32_t h = std::min(gqa, 8u);
    while (gqa % h) --h;
    return h;
}

static size_t decode_attention_smem(uint32_t heads, uint32_t dim, uint32_t ranks) {
    // (a slice is at most all outputs over two ranks, rounded up; every rank has one part of it)
    const size_t outputs = (size_t)heads * dim;
    return (size_t)(heads + 2) * dim * 2 + (DA_WARPS * outputs + DA_WARPS * heads * 3 + (size_t)ranks * heads * 2 + 4 + outputs + 4 * ranks) * 4;
}

template <int D, bool FEW>
static void launch_decode_attention(uzu_command_buffer* cmd, const DecodeAttnParams& p, const AttnSequences& s, size_t smem) {
    static std::atomic<uint64_t> opted{0};
    opt_in_dynamic_smem(cmd, decode_attention_kernel<D, FEW>, 200 * 1024, opted);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(p.ranks, p.num_kv_heads * p.groups, s.count);
    cfg.blockDim = dim3(DA_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = cmd->ctx->stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = p.ranks;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.numAttrs = 1;
    if (cmd->dependent()) {
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.numAttrs = 2;
    }
    cfg.attrs = attr;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, decode_attention_kernel<D, FEW>, p, s);
    if (e != cudaSuccess) cmd->record_error(UZU_ERROR_CUDA, std::string("decode_attention_kernel: ") + cudaGetErrorString(e));
    cmd->launches++;
}

// one plain causal row a sequence, on caches of whole 16-byte pieces
bool decode_attention_applicable(const uzu_attention_prepare_args& p, const uzu_attention_args& a, const AttnSequences& s) {
    if (!s.count || s.count > kMaxAttnSequences || p.batch_dim != s.count || !p.has_kv || !p.num_kv_heads || p.num_q_heads % p.num_kv_heads) return false;
    if (a.head_dim != p.head_dim || (a.head_dim != 64 && a.head_dim != 128 && a.head_dim != 256) || a.num_heads != p.num_q_heads || a.gqa_factor != p.num_q_heads / p.num_kv_heads) return false;
    if (a.suffix_length != 1 || a.is_trie || a.is_kv_cache_ring || a.is_sliding_window || a.has_sinks || a.dynamic_position != p.dynamic_position) return false;
    if (p.has_rope && (!p.cosines || !p.sines || !p.rope_dim || p.rope_dim > p.head_dim || (p.rope_dim & 1))) return false;
    uint64_t caches = 0;
    for (uint32_t b = 0; b < s.count; ++b) {
        if (!s.keys[b] || !s.values[b]) return false;
        caches |= s.keys[b] | s.values[b];
    }
    return p.qkv && a.out && !(caches & 15u) && a.k_head_stride == p.head_dim && a.v_head_stride == p.head_dim && a.k_seq_stride == p.num_kv_heads * p.head_dim &&
           a.v_seq_stride == a.k_seq_stride;
}

void encode_decode_attention(uzu_command_buffer* cmd, const uzu_attention_prepare_args& a, const uzu_qk_norm_config* q_norm, const uzu_qk_norm_config* k_norm, float scale, uint64_t out,
                             const AttnSequences& s, uint32_t longest) {
    if (!encodable(cmd, "decode_attention")) return;
    DecodeAttnParams p{};
    p.qkv = a.qkv;
    p.out = out;
    p.positions = a.dynamic_position;
    if (a.has_rope) { p.cosines = a.cosines; p.sines = a.sines; p.rope_dim = a.rope_dim; }
    p.num_heads = a.num_q_heads;
    p.num_kv_heads = a.num_kv_heads;
    p.heads = decode_attention_heads(a.num_q_heads / a.num_kv_heads);
    p.groups = a.num_q_heads / a.num_kv_heads / p.heads;
    p.kv_stride = a.num_kv_heads * a.head_dim;
    p.scale = scale;
    if (q_norm) p.q_norm = *q_norm;
    if (k_norm) p.k_norm = *k_norm;
    p.ranks = std::min(8u, (longest + DA_RANK_KEYS - 1) / DA_RANK_KEYS);
    const size_t smem = decode_attention_smem(p.heads, a.head_dim, p.ranks);
#define UZU_DA(D_)                                                                          \
    if (a.head_dim == D_) {                                                                 \
        if (p.heads <= 4) launch_decode_attention<D_, true>(cmd, p, s, smem);               \
        else launch_decode_attention<D_, false>(cmd, p, s, smem);                           \
    }
    UZU_DA(64)
    UZU_DA(128)
    UZU_DA(256)
#undef UZU_DA
}

}  // namespace uzu

extern "C" int uzu_debug_decode_attention_encode(uzu_command_buffer* cmd, const uzu_attention_prepare_norm_args* p, const uzu_attention_args* a) {
    if (!cmd || !p || !a || a->sequence_length <= p->prepare.kv_token_offset) return 0;
    uzu::AttnSequences s{};
    s.count = 1;
    s.keys[0] = a->keys; s.values[0] = a->values;
    s.prefix[0] = s.position[0] = p->prepare.kv_token_offset;
    if (!uzu::decode_attention_applicable(p->prepare, *a, s)) return 0;
    uzu::encode_decode_attention(cmd, p->prepare, &p->q_norm, &p->k_norm, a->scale, a->out, s, a->sequence_length);
    return 1;
}
