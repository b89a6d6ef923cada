// Attention of a prompt's rows on the 5th-generation tensor cores. Spec: backends/cpu/kernel/attention/attention_single_pass.rs:49-126 (mask.rs:3-62: causal, trie or none).
//
// What bounded the kernel before it (attention_prefill.cu, still the one for what this does not take): mma.sync has a quarter of this pipe's rate, and its four warps
// reached a third of that. Here a CTA has 128 rows, (token, head) pairs of a key head, two threads of eight softmax warps each, one warp that copies and one that issues:
//   copy    keys and values by TMA, 64 keys a stage, two stages, 64 channels a block of 128-byte swizzled rows (keys past the last are not read: zeros).
//   issue   S = Q K^T into tensor memory, 64 columns for every 64 channels, then a tile's P V with P as operand A there: two or three bf16 planes, as many as the kernel
//           before has, so that the f32 weights are exact to 16 bits or whole. Values are operand B as they lie (N-major).
//   softmax a thread reads 32 of its row's 64 scores, the two tell each other their maxima, and it writes its planes. The tile before is added to O, half of it in each
//           thread's registers; it is rescaled only where a row's maximum has grown by more than 2^8, so that weights reach 256 at most.
// The pipe cuts what it adds to an accumulator off at its last bit. So no chain is longer than 64 channels or the products of a tile, the smallest plane first, and the
// chains are added by rounded additions: with three planes 1.4 to 2.1 results in 10000 are off the correct rounding (split-KV, all f32, 1.8 to 4.7; mma.sync 2.3 to 2.9;
// 33 with whole chains in tensor memory), with two 24 to 25 (mma.sync 23 to 30, whole chains 29 to 31).
// Of 64 channels two CTAs share an SM, one's products run beside the other's softmax (and a thread spills 360 bytes for it); of more, the sums take the registers. Of 256
// channels a CTA sums one half (grid z), so that the prompts of few heads fill the chip. What bounds it now: the softmax warps' way through a tile, 1900 cycles of 128
// channels and 2300 of 256 (exponentials 750, planes 300, the waits for scores, for the tile before and for stores 140 each); products take 860 and 1500 of them. Four
// threads a row instead of two changed nothing.
// 1024 tokens behind 1100 rows, before -> now: 8 heads of 256 in groups of 4 128 -> 52 us, 32 of 128 168 -> 74, 32 of 64 92 -> 53 (with O in tensor memory, two CTAs an
// SM: 53, 48, 43).
// (Accumulators start at multiples of 128 columns, scores at multiples of 64. A form with score tiles 96 columns apart, 256 channels a CTA and clusters that shared the
// keys of a row tile ended in an illegal memory access whose cause was not found; none of the three is built.)
// A value that is not finite makes NaN of a weight of zero, in whole or in one of its planes: a row whose sums are not finite, its weights being so, is computed again
// key by key, each only where it is seen (1024 tokens behind 1024 rows with nothing but infinities: 5 ms of 64 channels, 10 of 128 and 256).
// Every barrier wait is bounded (wait_errors.h).
#include <cuda.h>

#include <algorithm>

#include "common.cuh"

namespace uzu {

namespace {

constexpr uint32_t AU_ROWS = 128, AU_KEYS = 64, AU_SOFT = 256, AU_THREADS = AU_SOFT + 64;      // softmax threads: two a row, 32 keys each

struct AuParams {
    uzu_attention_args a;
    unsigned int* error;
};

template <int D, int PLANES>
struct AuShape {
    static constexpr uint32_t OUT = D < 128 ? D : 128;                       // channels of O that a CTA sums
    static constexpr uint32_t Q_BLOCK = AU_ROWS * 128, KV_BLOCK = AU_KEYS * 128, Q = D / 64 * Q_BLOCK, K = D / 64 * KV_BLOCK, V = OUT / 64 * KV_BLOCK;
    static constexpr uint32_t CTAS = D == 64 ? 2 : 1;      // of an SM
    // tensor memory: scores, 64 columns for every 64 channels; a tile's products; the planes of its weights
    static constexpr uint32_t COLUMNS = 512 / CTAS, O_COL = 256 / CTAS;
    static constexpr __host__ __device__ uint32_t plane(uint32_t i) { return CTAS == 1 ? 384 + 32 * i : i < 2 ? 64 + 32 * i : 192; }
    static constexpr size_t SMEM = Q + 2 * K + 2 * V + 1024;
};

__device__ __forceinline__ uint32_t au_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void au_init(uint32_t bar, uint32_t count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory"); }
// (a whole warp, for all its lanes)
__device__ __forceinline__ void au_arrive(uint32_t bar) {
    __syncwarp();
    if ((threadIdx.x & 31u) == 0) asm volatile("{ .reg .b64 st; mbarrier.arrive.shared::cta.b64 st, [%0]; }" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool au_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3; selp.u32 %0, 1, 0, p; }" : "=r"(ok) : "r"(bar), "r"(parity), "r"(20000u) : "memory");
    return ok != 0;
}
// after a wait that ran out: what is in flight ends before the CTA does
__device__ __forceinline__ void au_settle(uint32_t bar, uint32_t parity) {
    for (uint32_t n = 0; n < 4096 && !au_try(bar, parity); ++n) {}
}
// false: the phase did not complete within about a second, or another role of the CTA has given up
__device__ __noinline__ bool au_wait_long(uint32_t bar, uint32_t parity, volatile uint32_t* gave_up, unsigned int* error, uint32_t code) {
    uint64_t t0, t1;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    for (uint32_t tries = 1;; ++tries) {
        if (au_try(bar, parity)) return true;
        if (tries & 15u) continue;
        if (*gave_up) return false;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
        if (t1 - t0 > 1000000000ull) {
            *gave_up = 1;
            report_wait_error(error, code);
            return false;
        }
    }
}
__device__ __forceinline__ bool au_wait(uint32_t bar, uint32_t parity, volatile uint32_t* gave_up, unsigned int* error, uint32_t code) {      // by whole warps
    if (__all_sync(0xffffffffu, au_try(bar, parity))) return true;
    return __all_sync(0xffffffffu, au_wait_long(bar, parity, gave_up, error, code));
}
__device__ __forceinline__ bool au_elect() {
    uint32_t p = 0;
    asm volatile("{ .reg .pred q; .reg .b32 r; elect.sync r|q, 0xffffffff; @q mov.u32 %0, 1; }" : "+r"(p));
    return p != 0;
}
__device__ __forceinline__ void au_expect(uint32_t bar, uint32_t bytes) {
    asm volatile("{ .reg .b64 st; mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1; }" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void au_tma(uint32_t dst, const CUtensorMap* map, uint32_t x, uint32_t y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
__device__ __forceinline__ void au_commit(uint32_t bar) { asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void au_mma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{ .reg .pred p; setp.ne.b32 p, %4, 0; tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p; }" ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void au_mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{ .reg .pred p; setp.ne.b32 p, %4, 0; tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p; }" ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void au_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void au_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void au_ld32(uint32_t taddr, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
          "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]),
          "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void au_st16(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]),
                 "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
                 : "memory");
}
// nothing that uses what was asked for is done before the wait
__device__ __forceinline__ void au_wait_ld(uint32_t (&v)[32]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]), "+r"(v[8]), "+r"(v[9]), "+r"(v[10]),
                   "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15]), "+r"(v[16]), "+r"(v[17]), "+r"(v[18]), "+r"(v[19]), "+r"(v[20]), "+r"(v[21]),
                   "+r"(v[22]), "+r"(v[23]), "+r"(v[24]), "+r"(v[25]), "+r"(v[26]), "+r"(v[27]), "+r"(v[28]), "+r"(v[29]), "+r"(v[30]), "+r"(v[31])
                 :
                 : "memory");
}
__device__ __forceinline__ void au_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t au_pack(float a, float b) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
}
// pairs of f32 in one instruction
__device__ __forceinline__ float2 au_fma2(float2 a, float2 b, float2 c) {
    float2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(reinterpret_cast<uint64_t&>(d)) : "l"(reinterpret_cast<uint64_t&>(a)), "l"(reinterpret_cast<uint64_t&>(b)), "l"(reinterpret_cast<uint64_t&>(c)));
    return d;
}
__device__ __forceinline__ float2 au_add2(float2 a, float2 b) {
    float2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(reinterpret_cast<uint64_t&>(d)) : "l"(reinterpret_cast<uint64_t&>(a)), "l"(reinterpret_cast<uint64_t&>(b)));
    return d;
}
__device__ __forceinline__ float au_exp2(float x) {      // 2 ulp, as exp2f; weights below 2^-126 are zero
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float au_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float au_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }
struct AuRow {
    const __nv_bfloat16 *query, *keys, *values;
    __nv_bfloat16* out;
    const uzu_trie_node* nodes;      // null: no trie
    uint64_t k_stride, v_stride;
    uint32_t token, lim, prefix, kend;
    float scale2;
};
// some channels of a row key by key, each key only where it is seen: for sums of values that are not finite (a warp's rows share their keys, so that its lanes read alike)
template <int D, uint32_t CHANNELS>
__device__ __noinline__ void au_row_by_key(const AuRow r) {
    float o[CHANNELS], most = -INFINITY, total = 0.0f;
#pragma unroll
    for (uint32_t j = 0; j < CHANNELS; ++j) o[j] = 0.0f;
#pragma unroll 1
    for (uint32_t key = 0; key < r.kend; ++key) {
        if (key >= r.lim && !(r.nodes && key >= r.prefix && r.token >= r.nodes[key - r.prefix].trie_start && r.token <= r.nodes[key - r.prefix].trie_end)) continue;
        const uint4 *q = reinterpret_cast<const uint4*>(r.query), *k = reinterpret_cast<const uint4*>(r.keys + key * r.k_stride), *v = reinterpret_cast<const uint4*>(r.values + key * r.v_stride);
        float s = 0.0f;
#pragma unroll 4
        for (uint32_t d = 0; d < D / 8; ++d) {
            const uint4 x = q[d], y = k[d];
            const uint32_t xs[4] = {x.x, x.y, x.z, x.w}, ys[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
            for (uint32_t i = 0; i < 4; ++i) s = fmaf(au_hi(xs[i]), au_hi(ys[i]), fmaf(au_lo(xs[i]), au_lo(ys[i]), s));
        }
        s *= r.scale2;
        const float next = fmaxf(most, s), from = next == -INFINITY ? 0.0f : next, keep = exp2f(most - from), w = exp2f(s - from);
        total = total * keep + w;
        most = next;
#pragma unroll
        for (uint32_t j = 0; j < CHANNELS; j += 8) {
            const uint4 y = v[j / 8];
            const uint32_t ys[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
            for (uint32_t i = 0; i < 4; ++i) {
                o[j + 2 * i] = fmaf(w, au_lo(ys[i]), o[j + 2 * i] * keep);
                o[j + 2 * i + 1] = fmaf(w, au_hi(ys[i]), o[j + 2 * i + 1] * keep);
            }
        }
    }
    const float inv = total > 0.0f ? 1.0f / total : 0.0f;
#pragma unroll
    for (uint32_t j = 0; j < CHANNELS; j += 8)
        *reinterpret_cast<uint4*>(r.out + j) = make_uint4(au_pack(o[j] * inv, o[j + 1] * inv), au_pack(o[j + 2] * inv, o[j + 3] * inv), au_pack(o[j + 4] * inv, o[j + 5] * inv),
                                                          au_pack(o[j + 6] * inv, o[j + 7] * inv));
}
}  // namespace

template <int D, int PLANES>
__global__ void __launch_bounds__(AU_THREADS, AuShape<D, PLANES>::CTAS) attn_umma_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v, const AuParams p) {
    using S = AuShape<D, PLANES>;
    extern __shared__ uint8_t au_raw[];
    __shared__ __align__(8) uint64_t bars[14];
    __shared__ uint32_t tmem_slot;
    __shared__ volatile uint32_t gave_up;
    __shared__ float row_max[2][2][AU_ROWS], row_sum[2][AU_ROWS];      // [tile][side][row]: what the two threads of a row tell each other
    const uzu_attention_args& a = p.a;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const uint32_t base = (au_smem(au_raw) + 1023u) & ~1023u, q0 = base, k0 = q0 + S::Q, v0 = k0 + 2 * S::K, bar0 = au_smem(bars);
    uint8_t* const base_p = au_raw + (base - au_smem(au_raw));
    const uint32_t q_full = bar0;
    auto k_full = [&](uint32_t s) { return bar0 + 8u * (1 + s); };
    auto k_empty = [&](uint32_t s) { return bar0 + 8u * (3 + s); };
    auto v_full = [&](uint32_t s) { return bar0 + 8u * (5 + s); };
    auto v_empty = [&](uint32_t s) { return bar0 + 8u * (7 + s); };
    const uint32_t s_full = bar0 + 8u * 9, s_empty = bar0 + 8u * 10, p_full = bar0 + 8u * 11, o_done = bar0 + 8u * 12, last_products = bar0 + 8u * 13;

    const uint32_t G = a.gqa_factor, m = a.suffix_length, seq = a.sequence_length, prefix = seq - m, rows = m * G, half = blockIdx.z * S::OUT;      // half: the first of this CTA's channels
    const uint32_t row0 = (gridDim.x - 1u - blockIdx.x) * AU_ROWS, kvh = blockIdx.y;      // the rows with the most keys first
    const bool causal = a.is_causal != 0, trie = causal && a.is_trie;
    const uint32_t last_row = min(row0 + AU_ROWS, rows) - 1u, kend = causal && !trie ? prefix + last_row / G + 1u : seq;
    const uint32_t whole = !causal ? seq : trie ? prefix : prefix + row0 / G + 1u;      // every row sees keys below it
    const uint32_t tiles = (kend + AU_KEYS - 1) / AU_KEYS;

    if (warp == 0) {
        if (lane == 0) {
            au_init(q_full, AU_SOFT / 32);
            for (uint32_t s = 0; s < 2; ++s) {
                au_init(k_full(s), 1); au_init(k_empty(s), 1); au_init(v_full(s), 1); au_init(v_empty(s), 1);
            }
            au_init(s_full, 1); au_init(s_empty, AU_SOFT / 32); au_init(p_full, AU_SOFT / 32); au_init(o_done, 1); au_init(last_products, 1);
            gave_up = 0;
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(au_smem(&tmem_slot)), "r"(S::COLUMNS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    au_fence_before();
    __syncthreads();
    au_fence_after();
    const uint32_t tmem = tmem_slot;
    pdl_launch_dependents();      // (not before this CTA has its tensor memory: a dependent's CTA that took it would wait for this one)
    pdl_wait();

    // a row's visible keys
    const uint32_t lr = tid & (AU_ROWS - 1), side = tid / AU_ROWS, row = row0 + lr, token = row / G, lim = row < rows ? (!causal ? seq : trie ? prefix : prefix + token + 1u) : 0u;
    const uzu_trie_node* nodes = reinterpret_cast<const uzu_trie_node*>(a.trie);
    auto sees = [&](uint32_t key) {
        if (key < lim) return true;
        if (!trie || row >= rows || key < prefix || key >= seq) return false;
        const uzu_trie_node& n = nodes[key - prefix];
        return token >= n.trie_start && token <= n.trie_end;
    };
    const float scale2 = a.scale * 1.4426950408889634f;
    float top = -INFINITY, sum = 0.0f;                                   // of the row: what its weights are relative to (in units of ln 2), their sum
    constexpr uint32_t MINE = S::OUT / 2;                                // columns of this thread
    float acc[MINE];
#pragma unroll
    for (uint32_t j = 0; j < MINE; ++j) acc[j] = 0.0f;
    bool ok = true;
    // a tile's products to the sums, by rounded additions (its weights are relative to the row's maximum at that time)
    auto add_tile = [&]() {
#pragma unroll
        for (uint32_t c = 0; c < MINE; c += 32) {
            uint32_t v[32];
            au_ld32(tmem + ((warp & 3u) << 21) + S::O_COL + side * MINE + c, v);
            au_wait_ld(v);
#pragma unroll
            for (uint32_t j = 0; j < 32; ++j) acc[c + j] += __uint_as_float(v[j]);
        }
    };

    if (warp < 8) {
        // ================================ softmax ================================
        {   // the row to shared memory, 128-byte swizzled blocks of 64 channels
            const __nv_bfloat16* src = reinterpret_cast<const __nv_bfloat16*>(a.queries) + ((size_t)(kvh * G + (row < rows ? row % G : 0u)) * m + (row < rows ? token : 0u)) * D;
#pragma unroll 8
            for (uint32_t c = side * (D / 16); c < (side + 1) * (D / 16); ++c) {
                const uint4 v = row < rows ? *reinterpret_cast<const uint4*>(src + c * 8) : make_uint4(0, 0, 0, 0);
                *reinterpret_cast<uint4*>(base_p + (c >> 3) * S::Q_BLOCK + lr * 128u + (((c & 7u) ^ (lr & 7u)) << 4)) = v;
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            au_arrive(q_full);
        }
        const uint32_t lanes = (warp & 3u) << 21, pair = 1u + (warp & 3u);      // pair: the barrier of the two warps of 32 rows
        auto leave = [&]() { asm volatile("bar.arrive %0, 64;" ::"r"(pair) : "memory"); };      // a wait ran out: the other warp is not left waiting
        for (uint32_t i = 0; i < tiles; ++i) {
            if (ok) ok = au_wait(s_full, i & 1u, &gave_up, p.error, 0x501u);
            if (!ok) { leave(); break; }
            au_fence_after();
            float2 s[16];
#pragma unroll
            for (uint32_t c = 0; c < D / 64; ++c) {                          // the sums over 64 channels each
                uint32_t raw[32];
                au_ld32(tmem + lanes + c * 64u + side * 32u, raw);
                au_wait_ld(raw);
#pragma unroll
                for (uint32_t j = 0; j < 16; ++j) {
                    const float2 x = make_float2(__uint_as_float(raw[2 * j]), __uint_as_float(raw[2 * j + 1]));
                    s[j] = c ? au_add2(s[j], x) : x;
                }
            }
            au_fence_before();
            au_arrive(s_empty);
            const bool part = (i + 1) * AU_KEYS > whole;                     // (rows past the last one sum what nobody reads)
            const uint32_t key0 = i * AU_KEYS + side * 32u;
            if (part) {
#pragma unroll
                for (uint32_t j = 0; j < 16; ++j) {
                    if (!sees(key0 + 2 * j)) s[j].x = -INFINITY;
                    if (!sees(key0 + 2 * j + 1)) s[j].y = -INFINITY;
                }
            }
            float mosts[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (uint32_t j = 0; j < 16; ++j) mosts[j & 3u] = fmaxf(mosts[j & 3u], fmaxf(s[j].x, s[j].y));
            float most = fmaxf(fmaxf(mosts[0], mosts[1]), fmaxf(mosts[2], mosts[3]));
            row_max[i & 1u][side][lr] = most;
            asm volatile("bar.sync %0, 64;" ::"r"(pair) : "memory");
            if (gave_up) { ok = false; leave(); break; }
            most = scale2 * fmaxf(most, row_max[i & 1u][side ^ 1u][lr]);     // (the scale is positive)
            // the maximum moves when it has grown by 2^8; from -inf (nothing seen yet) always
            const bool moves = most > top + 8.0f || (top == -INFINITY && most != -INFINITY);
            const float factor = moves ? exp2f(top - most) : 1.0f;          // (exp2(-inf - most) = 0)
            if (moves) top = most;
            const float from = top == -INFINITY ? 0.0f : top;
            const float2 scale_2 = make_float2(scale2, scale2), from_2 = make_float2(-from, -from), minus = make_float2(-1.0f, -1.0f);
            float2 sums[2] = {make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f)};
#pragma unroll
            for (uint32_t j = 0; j < 16; ++j) {
                const float2 x = au_fma2(s[j], scale_2, from_2);
                s[j] = make_float2(au_exp2(x.x), au_exp2(x.y));
                sums[j & 1u] = au_add2(sums[j & 1u], s[j]);
            }
            sum = sum * factor + ((sums[0].x + sums[0].y) + (sums[1].x + sums[1].y));
            if (i) {                                                         // the tile before is done, its weights' place free
                ok = au_wait(o_done, (i - 1) & 1u, &gave_up, p.error, 0x502u);
                if (!ok) { leave(); break; }
                au_fence_after();
                add_tile();
                if (__any_sync(0xffffffffu, moves)) {
#pragma unroll
                    for (uint32_t j = 0; j < MINE; ++j) acc[j] *= factor;
                }
            }
#pragma unroll
            for (uint32_t pl = 0; pl < (uint32_t)PLANES; ++pl) {
                uint32_t w[16];
#pragma unroll
                for (uint32_t j = 0; j < 16; ++j) {
                    w[j] = au_pack(s[j].x, s[j].y);
                    if (pl + 1 < (uint32_t)PLANES) s[j] = au_fma2(make_float2(au_lo(w[j]), au_hi(w[j])), minus, s[j]);
                }
                au_st16(tmem + lanes + S::plane(pl) + 16u * side, w);
            }
            au_wait_st();
            au_fence_before();
            au_arrive(p_full);
        }
        if (ok) {
            ok = au_wait(o_done, (tiles - 1) & 1u, &gave_up, p.error, 0x502u);
            au_fence_after();
            if (ok) add_tile();
        }
        row_sum[side][lr] = sum;
    } else if (warp == 8) {
        // ================================ keys and values by TMA ================================
        const uint32_t xk = kvh * (uint32_t)a.k_head_stride, xv = kvh * (uint32_t)a.v_head_stride + half;
        // keys one tile ahead of values: the next scores do not wait for a value stage
        auto copy = [&](uint32_t i, bool key) {
            const uint32_t s = i & 1u, full = key ? k_full(s) : v_full(s), at = key ? k0 + s * S::K : v0 + s * S::V, x = key ? xk : xv;
            ok = au_wait(key ? k_empty(s) : v_empty(s), (i >> 1 & 1u) ^ 1u, &gave_up, p.error, key ? 0x504u : 0x505u);
            if (ok && au_elect()) {
                au_expect(full, key ? S::K : S::V);
                for (uint32_t c = 0; c < (key ? (uint32_t)D : S::OUT) / 64; ++c) au_tma(at + c * S::KV_BLOCK, key ? &map_k : &map_v, x + c * 64u, i * AU_KEYS, full);
            }
            __syncwarp();
        };
        uint32_t asked_k = 0, asked_v = 0;
        copy(0, true);
        asked_k += ok;
        for (uint32_t i = 0; i < tiles && ok; ++i) {
            if (i + 1 < tiles) { copy(i + 1, true); asked_k += ok; }
            if (ok) { copy(i, false); asked_v += ok; }
        }
        if (!ok) {      // copies that are on their way end before the CTA does
            for (uint32_t n = 1; n <= 2; ++n) {
                if (asked_k >= n) au_settle(k_full((asked_k - n) & 1u), (asked_k - n) >> 1 & 1u);
                if (asked_v >= n) au_settle(v_full((asked_v - n) & 1u), (asked_v - n) >> 1 & 1u);
            }
        }
    } else {
        // ================================ products ================================
        // shared-memory descriptors: 128-byte swizzle, 1024 bytes between groups of 8 rows; values N-major, KV_BLOCK between blocks of 64 channels
        constexpr uint64_t desc_hi = (uint64_t)((1024u >> 4) | (1u << 14) | (2u << 29)) << 32;
        constexpr uint32_t idesc_s = (1u << 4) | (1u << 7) | (1u << 10) | ((AU_KEYS >> 3) << 17) | ((AU_ROWS >> 4) << 24);
        constexpr uint32_t idesc_o = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((S::OUT >> 3) << 17) | ((AU_ROWS >> 4) << 24);
        auto scores = [&](uint32_t i) {
            const uint32_t s = i & 1u;
            ok = au_wait(k_full(s), i >> 1 & 1u, &gave_up, p.error, 0x507u);
            if (ok && i) ok = au_wait(s_empty, (i - 1) & 1u, &gave_up, p.error, 0x506u);
            if (!ok) return;
            au_fence_after();
            if (au_elect()) {
#pragma unroll
                for (uint32_t kk = 0; kk < D / 16; ++kk) {                   // 64 channels a sum
                    const uint32_t qa = q0 + (kk >> 2) * S::Q_BLOCK + (kk & 3u) * 32u, ka = k0 + s * S::K + (kk >> 2) * S::KV_BLOCK + (kk & 3u) * 32u;
                    au_mma_ss(tmem + (kk >> 2) * 64u, desc_hi | (1u << 16) | (qa >> 4), desc_hi | (1u << 16) | (ka >> 4), idesc_s, (kk & 3u) != 0);
                }
                au_commit(s_full);
                au_commit(k_empty(s));
            }
            __syncwarp();
        };
        ok = au_wait(q_full, 0, &gave_up, p.error, 0x508u);
        au_fence_after();
        if (ok) scores(0);
        for (uint32_t i = 0; i < tiles && ok; ++i) {
            const uint32_t s = i & 1u;
            if (i + 1 < tiles) scores(i + 1);
            if (ok) ok = au_wait(p_full, i & 1u, &gave_up, p.error, 0x509u);
            if (ok) ok = au_wait(v_full(s), i >> 1 & 1u, &gave_up, p.error, 0x50au);
            if (!ok) break;
            au_fence_after();
            if (au_elect()) {
#pragma unroll
                for (uint32_t n = 0; n < (uint32_t)PLANES * (AU_KEYS / 16); ++n) {      // the smallest plane first
                    const uint32_t pl = PLANES - 1 - n / (AU_KEYS / 16), kk = n % (AU_KEYS / 16), va = v0 + s * S::V + kk * 2048u;
                    au_mma_ts(tmem + S::O_COL, tmem + S::plane(pl) + kk * 8u, desc_hi | ((uint64_t)(S::KV_BLOCK >> 4) << 16) | (va >> 4), idesc_o, n != 0);
                }
                au_commit(v_empty(s));
                au_commit(o_done);
            }
            __syncwarp();
        }
        if (!ok) {
            if (au_elect()) au_commit(last_products);
            __syncwarp();
            au_settle(last_products, 0);                                 // none in flight when tensor memory is given back
        }
    }

    // ---- the rows: out[token, head, d] = O / sum, rounded once ----
    __syncthreads();      // (gave_up and the sums; no copy or product is under way)
    ok = !gave_up;
    if (warp < 8 && ok) {
        const uint32_t head = kvh * G + (row < rows ? row % G : 0u), at = row < rows ? token : 0u;
        __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(a.out) + ((size_t)at * a.num_heads + head) * D + half + side * MINE;
        const float both = row_sum[0][lr] + row_sum[1][lr], inv = both > 0.0f ? 1.0f / both : 0.0f;
        bool finite = true;
#pragma unroll
        for (uint32_t j = 0; j < MINE; ++j) finite &= fabsf(acc[j]) < INFINITY;
        if (row < rows && (finite || !(both < INFINITY))) {
#pragma unroll
            for (uint32_t j = 0; j < MINE; j += 8)
                *reinterpret_cast<uint4*>(out + j) = make_uint4(au_pack(acc[j] * inv, acc[j + 1] * inv), au_pack(acc[j + 2] * inv, acc[j + 3] * inv),
                                                                au_pack(acc[j + 4] * inv, acc[j + 5] * inv), au_pack(acc[j + 6] * inv, acc[j + 7] * inv));
        } else if (row < rows) {
            AuRow r;
            r.query = reinterpret_cast<const __nv_bfloat16*>(a.queries) + ((size_t)head * m + token) * D;
            r.keys = reinterpret_cast<const __nv_bfloat16*>(a.keys) + (size_t)kvh * a.k_head_stride;
            r.values = reinterpret_cast<const __nv_bfloat16*>(a.values) + (size_t)kvh * a.v_head_stride + half + side * MINE;
            r.out = out;
            r.nodes = trie ? nodes : nullptr;
            r.k_stride = a.k_seq_stride; r.v_stride = a.v_seq_stride;
            r.token = token; r.lim = lim; r.prefix = prefix; r.kend = kend;
            r.scale2 = scale2;
            au_row_by_key<D, MINE>(r);
        }
    }
    au_fence_before();
    __syncthreads();
    if (warp == 0) {
        au_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(S::COLUMNS) : "memory");
    }
}

// ---------------------------------------------------------------------------------------------------------------------------------
// host
// ---------------------------------------------------------------------------------------------------------------------------------
static decltype(&cuTensorMapEncodeTiled) au_encoder() {
    static decltype(&cuTensorMapEncodeTiled) fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) f = nullptr;
        cudaGetLastError();
        return (decltype(&cuTensorMapEncodeTiled))f;
    }();
    return fn;
}
// cached rows, every head's channels side by side in one
static bool au_map(CUtensorMap* map, uint64_t addr, uint64_t row, uint64_t rows, uint64_t pitch) {
    const cuuint64_t dims[2] = {row, rows}, strides[1] = {pitch * 2};
    const cuuint32_t box[2] = {64, AU_KEYS}, steps[2] = {1, 1};
    return au_encoder()(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (void*)addr, dims, strides, box, steps, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int D, int PLANES>
static void launch_attn_umma(uzu_command_buffer* cmd, const AuParams& p, const CUtensorMap& mk, const CUtensorMap& mv) {
    static std::atomic<uint64_t> opted{0};
    opt_in_dynamic_smem(cmd, attn_umma_kernel<D, PLANES>, (int)AuShape<D, PLANES>::SMEM, opted);
    const uint32_t row_tiles = (p.a.suffix_length * p.a.gqa_factor + AU_ROWS - 1) / AU_ROWS;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(row_tiles, p.a.num_heads / p.a.gqa_factor, D / AuShape<D, PLANES>::OUT);
    cfg.blockDim = dim3(AU_THREADS);
    cfg.dynamicSmemBytes = AuShape<D, PLANES>::SMEM;
    cfg.stream = cmd->ctx->stream;
    cudaLaunchAttribute attr[1];
    cfg.attrs = attr;
    if (cmd->dependent()) {
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.numAttrs = 1;
    }
    const cudaError_t e = cudaLaunchKernelEx(&cfg, attn_umma_kernel<D, PLANES>, mk, mv, p);
    if (e != cudaSuccess) cmd->record_error(UZU_ERROR_CUDA, std::string("attn_umma_kernel: ") + cudaGetErrorString(e));
    cmd->launches++;
}

// of calls that the prompt kernel takes (encode_attention_prefill's conditions): every head's channels of a cached row in one run of memory
bool attn_umma_applicable(const uzu_attention_args& a) {
    const uint64_t heads = a.num_heads / a.gqa_factor;
    return a.scale > 0.0f && (heads - 1) * a.k_head_stride + a.head_dim <= a.k_seq_stride && (heads - 1) * a.v_head_stride + a.head_dim <= a.v_seq_stride && a.k_seq_stride < (1ull << 31) && a.v_seq_stride < (1ull << 31) &&
           au_encoder() != nullptr;
}

// planes: bf16 planes of a weight, 2 or 3
bool encode_attn_umma(uzu_command_buffer* cmd, const uzu_attention_args& a, uint32_t planes) {
    const uint32_t heads = a.num_heads / a.gqa_factor, D = a.head_dim;
    CUtensorMap mk, mv;
    if (!au_map(&mk, a.keys, (uint64_t)(heads - 1) * a.k_head_stride + D, a.sequence_length, a.k_seq_stride) ||
        !au_map(&mv, a.values, (uint64_t)(heads - 1) * a.v_head_stride + D, a.sequence_length, a.v_seq_stride)) return false;
    AuParams p{};
    p.a = a;
    p.error = cmd->ctx->wait_errors.device_word;
    if (D == 64) planes == 2 ? launch_attn_umma<64, 2>(cmd, p, mk, mv) : launch_attn_umma<64, 3>(cmd, p, mk, mv);
    else if (D == 128) planes == 2 ? launch_attn_umma<128, 2>(cmd, p, mk, mv) : launch_attn_umma<128, 3>(cmd, p, mk, mv);
    else launch_attn_umma<256, 3>(cmd, p, mk, mv);
    return true;
}

}  // namespace uzu
