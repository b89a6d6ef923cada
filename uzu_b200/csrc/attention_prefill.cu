// Attention of several query tokens on the tensor cores: prompt chunks, short portions and speculation passes over the token-major KV cache.
//
// Semantic spec: backends/cpu/kernel/attention/attention_single_pass.rs:49-126 (online softmax per query over the visible keys, q scaled by
// `scale`, GQA kv_head = h / gqa, output [suffix, heads, D] cast after the division by the sum), mask.rs:3-62 restricted to the plain causal /
// non-causal case and the trie (no ring, sliding window, sinks: those keep the split-KV kernel of attention.cu).
//
// One CTA = 64 rows of one KV head, a row being one (query token, query head) pair: the heads that share a KV head read its keys and values
// once, and a speculation pass of 16 nodes x 4 heads is one tile. Four warps of 16 rows:
//   * S = Q K^T with mma.sync.m16n8k16 (bf16 x bf16 products are exact, f32 accumulate), Q, K and V fragments by ldmatrix from shared memory
//     (64 keys x D, rows padded to D + 8: conflict-free);
//   * online softmax in f32 registers, row statistics over the 4 lanes of a quad; O is rescaled only when some row's maximum moved;
//   * O += P V with P as bf16 planes (bf16(p), then bf16 of what is left): three hold a probability to its last bit. A prompt's passes of 64 and 128
//     channels have two (16 bits of it); a single plane would put 2^-9 on every probability. V fragments come from ldmatrix.trans. The pipe cuts what it
//     adds to an accumulator off at its last bit, so with three planes no chain is longer than four products of either sum, and the chains are added by
//     rounded additions: as many results differ from the correctly rounded ones as on the split-KV kernel (2 in 10000), with two planes and whole chains
//     it was 20 in 10000.
// A weight of zero does not hide a value that is not finite (0 x NaN): value tiles that some row sees in part are looked over first, and one with infinities
// or NaN is summed key by key for the rows that see them, so that no token reaches an earlier one or another branch of a trie (with three planes: the
// passes that the split-KV kernel served before, which never multiplied what a token does not see).
// The next key tile is requested when S is done (it arrives during P V), the next value tile when P V is done: one buffer each, so that two or
// three CTAs share an SM and fill one another's waits. Causal tiles past the CTA's last query are never loaded, and tiles every row of a
// warp sees whole are not masked. CTAs with the most keys start first.
// Where rows x KV heads do not fill the chip a cluster of up to 8 CTAs shares the keys of a tile and merges its partial results over
// distributed shared memory in rank order.
// Bound: shared-memory reads and mma.sync issue. 8 heads of 256 channels (2 KV heads), 1024 rows behind 1024: 0.13 ms against 1.11 ms one query
// token at a time on the split-KV kernel.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <type_traits>

#include "common.cuh"

namespace uzu {

constexpr int PA_BM = 64;   // rows per CTA
constexpr int PA_BN = 64;   // keys per K / V tile

__device__ __forceinline__ void pa_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void pa_ldmatrix_x4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void pa_ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void pa_cp16(uint32_t dst_smem, const void* src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst_smem), "l"(src), "r"(valid ? 16u : 0u) : "memory");
}
__device__ __forceinline__ uint32_t pa_pack(float lo_elem, float hi_elem) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo_elem, hi_elem);
    return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ void pa_cluster_sync() { asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ float pa_remote(uint32_t addr, uint32_t rank) {
    uint32_t remote;
    float x;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(x) : "r"(remote) : "memory");
    return x;
}

template <int D, int PLANES>
__global__ void __launch_bounds__(128, D == 256 ? 2 : 3) attn_prefill_kernel(const uzu_attention_args a, const uint32_t splits) {
    pdl_launch_dependents();
    pdl_wait();
    constexpr uint32_t LD = D + 8;                  // padded tile row (elements): 16-byte aligned rows, conflict-free ldmatrix
    constexpr uint32_t TILE = PA_BN * LD * 2;       // bytes
    constexpr uint32_t CH = D / 8;                  // 16-byte chunks per row
    constexpr float kLog2e = 1.4426950408889634f;
    constexpr bool kRounded = PLANES == 3;          // sums of more than four products by rounded additions
    extern __shared__ __align__(16) uint8_t pa_smem[];
    const uint32_t sq = (uint32_t)__cvta_generic_to_shared(pa_smem), sk = sq + TILE, sv = sk + TILE;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, quad = lane >> 2, tq = lane & 3;
    const uint32_t G = a.gqa_factor, m = a.suffix_length, seq = a.sequence_length, prefix = seq - m, rows = m * G;
    const uint32_t rank = splits > 1 ? blockIdx.x % splits : 0u;
    const uint32_t tile = gridDim.x / splits - 1u - blockIdx.x / splits;      // the rows with the most keys first
    const uint32_t row0 = tile * PA_BM, kvh = blockIdx.y;
    const bool causal = a.is_causal != 0;
    const uint32_t q_last = min(row0 + (uint32_t)PA_BM, rows) - 1u;           // last row of the CTA
    // keys [0, kend) can be visible to some row of this CTA (a trie node may be seen by any later node: all suffix keys)
    const uint32_t kend = causal && !a.is_trie ? prefix + q_last / G + 1u : seq;
    const uint32_t all_tiles = (kend + PA_BN - 1) / PA_BN, per = (all_tiles + splits - 1) / splits;
    const uint32_t t_begin = min(rank * per, all_tiles), t_end = min(t_begin + per, all_tiles);
    const __nv_bfloat16* kbase = reinterpret_cast<const __nv_bfloat16*>(a.keys) + (size_t)kvh * a.k_head_stride;
    const __nv_bfloat16* vbase = reinterpret_cast<const __nv_bfloat16*>(a.values) + (size_t)kvh * a.v_head_stride;

    auto load_tile = [&](uint32_t dst, const __nv_bfloat16* src, size_t stride, uint32_t t) {
#pragma unroll 4
        for (uint32_t c = tid; c < PA_BN * CH; c += 128) {
            const uint32_t key = c / CH, ch = c % CH, kg = t * PA_BN + key;
            const bool ok = kg < kend;                               // rows past the visible range may be unmapped cache pages: never read
            pa_cp16(dst + (key * LD + ch * 8) * 2, src + (size_t)(ok ? kg : 0u) * stride + ch * 8, ok);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (uint32_t c = tid; c < PA_BM * CH; c += 128) {               // row r of the tile: token r / G, head r % G of the group
        const uint32_t r = c / CH, ch = c % CH, row = row0 + r;
        const bool ok = row < rows;
        const uint32_t token = ok ? row / G : 0u, head = kvh * G + (ok ? row % G : 0u);
        pa_cp16(sq + (r * LD + ch * 8) * 2, reinterpret_cast<const __nv_bfloat16*>(a.queries) + ((size_t)head * m + token) * D + ch * 8, ok);
    }
    if (t_begin < t_end) load_tile(sk, kbase, a.k_seq_stride, t_begin);      // (one group with the queries)
    else asm volatile("cp.async.commit_group;" ::: "memory");
    if (t_begin < t_end) load_tile(sv, vbase, a.v_seq_stride, t_begin);

    float o[D / 8][4];
#pragma unroll
    for (int nd = 0; nd < D / 8; ++nd) o[nd][0] = o[nd][1] = o[nd][2] = o[nd][3] = 0.0f;
    float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.0f, l1 = 0.0f;     // running max (in units of ln 2) / sum of rows r0 and r0 + 8
    const uint32_t r0 = row0 + warp * 16 + quad, r1 = r0 + 8;
    // exclusive key bound per row: causal -> keys up to and including the query's own position; trie: the prefix, suffix keys by their node's range
    const uint32_t n0 = r0 / G, n1 = r1 / G;
    const uint32_t lim0 = r0 < rows ? (!causal ? seq : a.is_trie ? prefix : prefix + n0 + 1) : 0u;
    const uint32_t lim1 = r1 < rows ? (!causal ? seq : a.is_trie ? prefix : prefix + n1 + 1) : 0u;
    const uint32_t w_first = row0 + warp * 16, w_last = w_first + 15;        // every row of the warp sees keys below `whole`
    const uint32_t whole = w_last >= rows ? 0u : (!causal ? seq : a.is_trie ? prefix : prefix + w_first / G + 1);
    const uint32_t cta_whole = !causal ? seq : a.is_trie ? prefix : prefix + row0 / G + 1;      // every row of the CTA sees keys below it
    const bool trie = causal && a.is_trie;
    const uzu_trie_node* nodes = reinterpret_cast<const uzu_trie_node*>(a.trie);
    auto sees = [&](uint32_t key, uint32_t lim, uint32_t node, bool row_ok) {
        if (key < lim) return true;
        if (!trie || !row_ok || key < prefix || key >= seq) return false;
        const uzu_trie_node& n = nodes[key - prefix];
        return node >= n.trie_start && node <= n.trie_end;
    };
    const float scale2 = a.scale * kLog2e;
    // ldmatrix rows of this lane: Q (16 rows x 16 d): row lane & 15, d half lane >> 4; K (two 8-key tiles): key (lane >> 4) * 8 + (lane & 7), d half
    // (lane >> 3) & 1; V (16 keys x two 8-d tiles): key lane & 15, d half lane >> 4
    const uint32_t q_addr = sq + ((warp * 16 + (lane & 15)) * LD + (lane >> 4) * 8) * 2;
    const uint32_t k_addr = sk + (((lane >> 4) * 8 + (lane & 7)) * LD + ((lane >> 3) & 1) * 8) * 2;
    const uint32_t v_addr = sv + ((lane & 15) * LD + (lane >> 4) * 8) * 2;

    auto tile_step = [&](const uint32_t t, auto part_c) {           // part: not every row of the CTA sees the whole tile
        asm volatile("cp.async.wait_group 1;" ::: "memory");        // this tile's keys (and the queries) have landed
        __syncthreads();
        // ---- S = Q K^T ----
        float s[PA_BN / 8][4];
#pragma unroll
        for (int nt = 0; nt < PA_BN / 8; ++nt) s[nt][0] = s[nt][1] = s[nt][2] = s[nt][3] = 0.0f;
        if constexpr (!kRounded) {
#pragma unroll
            for (int ks = 0; ks < D / 16; ++ks) {
                uint32_t qf[4];
                pa_ldmatrix_x4(qf, q_addr + ks * 32);
#pragma unroll
                for (int nt = 0; nt < PA_BN / 8; nt += 2) {
                    uint32_t kf[4];
                    pa_ldmatrix_x4(kf, k_addr + nt * 8 * LD * 2 + ks * 32);
                    pa_mma(s[nt], qf, kf[0], kf[1]);
                    pa_mma(s[nt + 1], qf, kf[2], kf[3]);
                }
            }
        } else {
#pragma unroll
            for (int k0 = 0; k0 < D / 16; k0 += 4) {
                uint32_t qf[4][4];
#pragma unroll
                for (int ks = 0; ks < 4; ++ks) pa_ldmatrix_x4(qf[ks], q_addr + (k0 + ks) * 32);
#pragma unroll
                for (int nt = 0; nt < PA_BN / 8; nt += 2) {
                    float part[2][4] = {};
#pragma unroll
                    for (int ks = 0; ks < 4; ++ks) {
                        uint32_t kf[4];
                        pa_ldmatrix_x4(kf, k_addr + nt * 8 * LD * 2 + (k0 + ks) * 32);
                        pa_mma(part[0], qf[ks], kf[0], kf[1]);
                        pa_mma(part[1], qf[ks], kf[2], kf[3]);
                    }
#pragma unroll
                    for (int i = 0; i < 8; ++i) s[nt + (i >> 2)][i & 3] += part[i >> 2][i & 3];
                }
            }
        }
        __syncthreads();                                            // every warp is done with the key tile
        if (t + 1 < t_end) load_tile(sk, kbase, a.k_seq_stride, t + 1);
        else asm volatile("cp.async.commit_group;" ::: "memory");
        // ---- scale, mask, online softmax (c0,c1: row r0, keys 2t, 2t+1; c2,c3: row r0 + 8) ----
        const uint32_t key0 = t * PA_BN + 2 * tq;
        float mx0 = -INFINITY, mx1 = -INFINITY;
        if ((t + 1) * PA_BN <= whole) {
#pragma unroll
            for (int nt = 0; nt < PA_BN / 8; ++nt) {
#pragma unroll
                for (int c = 0; c < 4; ++c) s[nt][c] *= scale2;
                mx0 = fmaxf(mx0, fmaxf(s[nt][0], s[nt][1]));
                mx1 = fmaxf(mx1, fmaxf(s[nt][2], s[nt][3]));
            }
        } else {
#pragma unroll
            for (int nt = 0; nt < PA_BN / 8; ++nt) {
                const uint32_t kg = key0 + nt * 8;
                s[nt][0] = sees(kg, lim0, n0, r0 < rows) ? s[nt][0] * scale2 : -INFINITY;
                s[nt][1] = sees(kg + 1, lim0, n0, r0 < rows) ? s[nt][1] * scale2 : -INFINITY;
                s[nt][2] = sees(kg, lim1, n1, r1 < rows) ? s[nt][2] * scale2 : -INFINITY;
                s[nt][3] = sees(kg + 1, lim1, n1, r1 < rows) ? s[nt][3] * scale2 : -INFINITY;
                mx0 = fmaxf(mx0, fmaxf(s[nt][0], s[nt][1]));
                mx1 = fmaxf(mx1, fmaxf(s[nt][2], s[nt][3]));
            }
        }
        mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 1)); mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 2));
        mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 1)); mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 2));
        const float top0 = fmaxf(m0, mx0), top1 = fmaxf(m1, mx1);
        const float base0 = top0 == -INFINITY ? 0.0f : top0, base1 = top1 == -INFINITY ? 0.0f : top1;      // (exp2(-inf - 0) = 0)
        const float c0 = exp2f(m0 - base0), c1 = exp2f(m1 - base1);
        const bool moved = __any_sync(0xffffffffu, top0 != m0 || top1 != m1);
        float rs0 = 0.0f, rs1 = 0.0f;
#pragma unroll
        for (int nt = 0; nt < PA_BN / 8; ++nt) {
            s[nt][0] = exp2f(s[nt][0] - base0);
            s[nt][1] = exp2f(s[nt][1] - base0);
            s[nt][2] = exp2f(s[nt][2] - base1);
            s[nt][3] = exp2f(s[nt][3] - base1);
            rs0 += s[nt][0] + s[nt][1];
            rs1 += s[nt][2] + s[nt][3];
        }
        if (moved) {
            l0 *= c0;
            l1 *= c1;
#pragma unroll
            for (int nd = 0; nd < D / 8; ++nd) {
                o[nd][0] *= c0; o[nd][1] *= c0;
                o[nd][2] *= c1; o[nd][3] *= c1;
            }
        }
        l0 += rs0;                                                  // (a lane's share of the row sum; the quad meets at the end)
        l1 += rs1;
        m0 = top0;
        m1 = top1;
        asm volatile("cp.async.wait_group 1;" ::: "memory");        // this tile's values have landed
        bool key_by_key = false;
        if constexpr (decltype(part_c)::value) {
            uint32_t bad = 0;
#pragma unroll 4
            for (uint32_t c = tid; c < PA_BN * CH; c += 128) {       // (what this thread copied)
                uint32_t x[4];
                asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(x[0]), "=r"(x[1]), "=r"(x[2]), "=r"(x[3]) : "r"(sv + (c / CH * LD + c % CH * 8) * 2));
#pragma unroll
                for (int j = 0; j < 4; ++j) bad |= (uint32_t)((x[j] & 0x7F80u) == 0x7F80u) | (uint32_t)((x[j] & 0x7F800000u) == 0x7F800000u);
            }
            key_by_key = __syncthreads_or((int)bad) != 0;
        } else {
            __syncthreads();
        }
        if (decltype(part_c)::value && key_by_key) {
#pragma unroll
            for (int nt = 0; nt < PA_BN / 8; ++nt)
#pragma unroll 1
            for (uint32_t j = 0; j < 8; ++j) {
                const uint32_t k = nt * 8u + j, kg = t * PA_BN + k, holder = (lane & ~3u) | (j >> 1);
                const float w0 = __shfl_sync(0xffffffffu, (j & 1u) ? s[nt][1] : s[nt][0], holder), w1 = __shfl_sync(0xffffffffu, (j & 1u) ? s[nt][3] : s[nt][2], holder);
                const bool sees0 = sees(kg, lim0, n0, r0 < rows), sees1 = sees(kg, lim1, n1, r1 < rows);
#pragma unroll
                for (int nd = 0; nd < D / 8; ++nd) {
                    uint32_t v;
                    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(sv + (k * LD + nd * 8 + 2 * tq) * 2));
                    const float v0 = __uint_as_float(v << 16), v1 = __uint_as_float(v & 0xffff0000u);
                    if (sees0) { o[nd][0] = fmaf(w0, v0, o[nd][0]); o[nd][1] = fmaf(w0, v1, o[nd][1]); }
                    if (sees1) { o[nd][2] = fmaf(w1, v0, o[nd][2]); o[nd][3] = fmaf(w1, v1, o[nd][3]); }
                }
            }
        } else {
            // ---- O += P V: the S accumulator layout IS the A fragment layout of the next MMA (k = key) ----
            auto planes = [&](uint32_t (&p)[PLANES][4], int kt) {   // a0 = (row, k 2t..): s[2 kt][0..1]; a1 = (row + 8): [2..3]; a2 = (row, k + 8): s[2 kt + 1][0..1]; a3: [2..3]
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    float x = s[2 * kt + (r >> 1)][2 * (r & 1)], y = s[2 * kt + (r >> 1)][2 * (r & 1) + 1];
#pragma unroll
                    for (int i = 0; i < PLANES; ++i) {
                        p[i][r] = pa_pack(x, y);
                        x -= __uint_as_float(p[i][r] << 16);
                        y -= __uint_as_float(p[i][r] & 0xffff0000u);
                    }
                }
            };
            if constexpr (!kRounded) {
#pragma unroll
                for (int kt = 0; kt < PA_BN / 16; ++kt) {
                    uint32_t p[PLANES][4];
                    planes(p, kt);
#pragma unroll
                    for (int nd = 0; nd < D / 8; nd += 2) {
                        uint32_t vf[4];
                        pa_ldmatrix_x4_trans(vf, v_addr + kt * 16 * LD * 2 + nd * 16);
#pragma unroll
                        for (int i = 0; i < PLANES; ++i) {
                            pa_mma(o[nd], p[i], vf[0], vf[1]);
                            pa_mma(o[nd + 1], p[i], vf[2], vf[3]);
                        }
                    }
                }
            } else {
                uint32_t p[PA_BN / 16][PLANES][4];
#pragma unroll
                for (int kt = 0; kt < PA_BN / 16; ++kt) planes(p[kt], kt);
#pragma unroll
                for (int nd = 0; nd < D / 8; nd += 2) {
                    float part[2][4] = {};
#pragma unroll
                    for (int kt = 0; kt < PA_BN / 16; ++kt) {
                        uint32_t vf[4];
                        pa_ldmatrix_x4_trans(vf, v_addr + kt * 16 * LD * 2 + nd * 16);
#pragma unroll
                        for (int i = PLANES - 1; i >= 0; --i) {
                            pa_mma(part[0], p[kt][i], vf[0], vf[1]);
                            pa_mma(part[1], p[kt][i], vf[2], vf[3]);
                        }
                    }
#pragma unroll
                    for (int i = 0; i < 8; ++i) o[nd + (i >> 2)][i & 3] += part[i >> 2][i & 3];
                }
            }
        }
        __syncthreads();                                            // every warp is done with the value tile
        if (t + 1 < t_end) load_tile(sv, vbase, a.v_seq_stride, t + 1);
        else asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (uint32_t t = t_begin; t < t_end; ++t) {
        if (kRounded && (t + 1) * PA_BN > cta_whole) tile_step(t, std::true_type{});
        else tile_step(t, std::false_type{});
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    l0 += __shfl_xor_sync(0xffffffffu, l0, 1); l0 += __shfl_xor_sync(0xffffffffu, l0, 2);
    l1 += __shfl_xor_sync(0xffffffffu, l1, 1); l1 += __shfl_xor_sync(0xffffffffu, l1, 2);

    // ---- out[token, head, d] = O / l, cast after the division ----
    __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(a.out);
    auto out_row = [&](uint32_t row) { return out + ((size_t)(row / G) * a.num_heads + kvh * G + row % G) * D; };
    if (splits == 1) {
        const float i0 = l0 > 0.0f ? 1.0f / l0 : 0.0f, i1 = l1 > 0.0f ? 1.0f / l1 : 0.0f;
#pragma unroll
        for (int nd = 0; nd < D / 8; ++nd) {
            const int d = nd * 8 + 2 * tq;
            if (r0 < rows) *reinterpret_cast<uint32_t*>(out_row(r0) + d) = pa_pack(o[nd][0] * i0, o[nd][1] * i0);
            if (r1 < rows) *reinterpret_cast<uint32_t*>(out_row(r1) + d) = pa_pack(o[nd][2] * i1, o[nd][3] * i1);
        }
        return;
    }
    // partial rows to shared memory (over the key and value tiles), then rank r merges rows r, r + splits, ..
    static_assert((size_t)PA_BM * D * 4 <= 2 * (size_t)TILE, "the partial rows take the place of the key and value tiles");
    __syncthreads();
    float* so = reinterpret_cast<float*>(pa_smem + TILE);            // [64][D]
    float* sml = reinterpret_cast<float*>(pa_smem);                  // [64] max, [64] sum (over the queries)
    const uint32_t lr = warp * 16 + quad;
#pragma unroll
    for (int nd = 0; nd < D / 8; ++nd) {
        *reinterpret_cast<float2*>(so + lr * D + nd * 8 + 2 * tq) = make_float2(o[nd][0], o[nd][1]);
        *reinterpret_cast<float2*>(so + (lr + 8) * D + nd * 8 + 2 * tq) = make_float2(o[nd][2], o[nd][3]);
    }
    if (tq == 0) {
        sml[lr] = m0; sml[lr + 8] = m1;
        sml[64 + lr] = l0; sml[64 + lr + 8] = l1;
    }
    pa_cluster_sync();
    const uint32_t so_addr = sk, ml_addr = sq;
    for (uint32_t r = rank + splits * warp; r < (uint32_t)PA_BM && row0 + r < rows; r += splits * 4) {
        float top = -INFINITY;
        for (uint32_t c = 0; c < splits; ++c) top = fmaxf(top, pa_remote(ml_addr + r * 4, c));
        const float base = top == -INFINITY ? 0.0f : top;
        float l = 0.0f, acc[D / 32];
#pragma unroll
        for (int i = 0; i < D / 32; ++i) acc[i] = 0.0f;
        for (uint32_t c = 0; c < splits; ++c) {
            const float w = exp2f(pa_remote(ml_addr + r * 4, c) - base);
            l += w * pa_remote(ml_addr + (64 + r) * 4, c);
#pragma unroll
            for (int i = 0; i < D / 32; ++i) acc[i] += w * pa_remote(so_addr + (r * D + i * 32 + lane) * 4, c);
        }
        const float inv = l > 0.0f ? 1.0f / l : 0.0f;
        __nv_bfloat16* dst = out_row(row0 + r);
#pragma unroll
        for (int i = 0; i < D / 32; ++i) dst[i * 32 + lane] = f2bf(acc[i] * inv);
    }
    pa_cluster_sync();                                              // no CTA leaves while another may still read its rows
}

// CTAs that share a tile's keys: more while the chip has room for them and each keeps two tiles or more
static uint32_t pa_splits(const uzu_attention_args& a, uint32_t sms) {
    const uint32_t row_tiles = (a.suffix_length * a.gqa_factor + PA_BM - 1) / PA_BM, kv_heads = a.num_heads / a.gqa_factor;
    const uint32_t key_tiles = (a.sequence_length + PA_BN - 1) / PA_BN, room = sms * (a.head_dim == 256 ? 2u : 3u);
    uint32_t splits = 1;
    while (splits < 8 && row_tiles * kv_heads * splits * 2 <= room && key_tiles >= splits * 4) splits *= 2;
    return splits;
}

static bool pa_two_planes(const uzu_attention_args& a) { return a.suffix_length >= 16 && !a.is_trie && a.head_dim != 256; }

// Which kernel takes a call. Estimates in us of this one and the split-KV kernel, fitted to 1480 sizes (8 to 256 tokens, 0 to 8000 cached rows, 4 to 64 heads in groups
// of 1 to 8; the choice costs 0.7 % on average). The split-KV kernel pays for every (token, head) and key, this one for whole tiles of 64 x 64. 32 heads of 128 in
// groups of 4, split-KV / this one: 8 tokens behind 16 rows 6.7 / 13.7, behind 450 23 / 19, behind 2048 48 / 31; 16 tokens behind 16 6.6 / 11.5, behind 1000
// 41 / 15. 8 heads of 256, 64 tokens alone 10.7 / 27, behind 1000 73 / 28. Fewer than 8 tokens stay with the split-KV kernel: 4 behind 200 take 12.4 / 14.5,
// behind 1000 19 / 14.5, behind 4096 45 / 37.
// The tcgen05 kernel (attention_umma.cu) walks the keys in CTAs of 128 rows that share nothing: the chip has to be filled by the rows. Fitted to 720 sizes (16 to 1024
// tokens, 0 to 6000 cached rows), within 10 % for nine in ten, so that it is taken where it is the faster by a sixth (none of the 720 is then slower). This one / that
// one: 32 heads of 128 in groups of 4, 64 tokens behind 100 16.2 / 12.3, behind 1100 20.3 / 27.2 (its keys are split, that one's not), 256 behind 1100 44.1 / 30.7, 1024
// behind 1100 168 / 74; of 64, 1024 behind 1100 92 / 53; 8 heads of 256 in groups of 4, 256 behind 1100 38.4 / 38.2, 400 58 / 41, 1024 128 / 52. In place of the
// split-KV kernel, whose weights are f32, it has to have three planes: 8 heads of 256, 100 tokens behind 100 21.6 / 16.4.
enum class PaKernel { Split, Mma, Umma };
static PaKernel pa_choose(const uzu_attention_args& a, uint32_t sms) {
    const uint32_t D = a.head_dim, rows = a.suffix_length, keys = a.sequence_length, gq = a.gqa_factor, g = gq % 8 == 0 ? 8 : gq % 4 == 0 ? 4 : gq % 2 == 0 ? 2 : 1;
    if (rows < 8) return PaKernel::Split;
    const uint32_t kv_heads = a.num_heads / gq, ctas = a.num_heads / g * rows;      // as encode_attn_rows (attention.cu) cuts it
    const uint32_t nsplits = rows <= 16 ? std::max(1u, std::min(std::min((2 * sms + ctas - 1) / ctas, (keys + 63) / 64), 32u)) : 1u;
    const float fill = (float)ctas * nsplits / (sms * (D == 128 ? 1.0f : 2.0f));
    const float waves = D == 128 ? 0.5f * (std::ceil(fill) + std::max(1.0f, fill)) : std::ceil(fill);
    const float per_key = D == 64 ? 0.0118f + 0.00064f * g * g : D == 128 ? 0.0103f + 0.00081f * g * g : 0.035f + 0.0019f * g * g;
    const float split = (D == 64 ? 1.0f : D == 128 ? 1.15f : 1.1f) *
                        ((D == 64 ? 5.5f : 6.2f) + waves * per_key * keys / nsplits + (nsplits == 1 ? 0.0f : D == 64 ? 2.8f : D == 128 ? 4.5f : 6.1f));
    const bool two = pa_two_planes(a);
    const uint32_t shares = pa_splits(a, sms), row_tiles = (rows * gq + PA_BM - 1) / PA_BM, key_tiles = (keys + PA_BN - 1) / PA_BN, room = sms * (D == 256 ? 2u : 3u);
    const uint32_t all = row_tiles * kv_heads * shares, turns = std::max(1u, (all + room - 1) / room), per = (key_tiles + shares - 1) / shares;
    const float start = D == 64 ? 5.0f : D == 128 ? 8.6f : 14.5f, tile = D == 64 ? (two ? 1.8f : 3.0f) : D == 128 ? (two ? 2.8f : 4.65f) : 7.0f;
    const float merge = shares == 1 ? 0.0f : D == 64 ? (two ? 4.4f : 2.3f) : D == 128 ? (two ? 1.9f : 0.6f) : -0.7f;
    const float mma = start * (0.5f + 0.5f * turns) + tile * per * turns + merge;
    const bool split_is_faster = mma >= split;
    if (!attn_umma_applicable(a) || (split_is_faster && (two || rows <= 16))) return split_is_faster ? PaKernel::Split : PaKernel::Mma;
    const uint32_t u_ctas = (rows * gq + 127) / 128 * kv_heads * (D == 256 ? 2u : 1u), u_room = sms * (D == 64 ? 2u : 1u), u_turns = std::max(1u, (u_ctas + u_room - 1) / u_room);
    const float u_start = D == 64 ? 19.7f - 12.3f * u_turns : D == 128 ? 11.4f - 2.4f * u_turns : 16.3f - 5.5f * u_turns;
    const float u_tile = (D == 64 ? 1.03f : D == 128 ? 0.97f : 1.2f) * u_turns + (D == 64 && u_ctas > sms ? 0.26f : 0.0f);
    const float umma = u_start + u_tile * key_tiles * (D != 256 && !two ? 1.1f : 1.0f);
    if (1.2f * umma < std::min(mma, split)) return PaKernel::Umma;
    return split_is_faster ? PaKernel::Split : PaKernel::Mma;
}

template <int D, int PLANES>
static void launch_attn_prefill(uzu_command_buffer* cmd, const uzu_attention_args& a) {
    constexpr size_t smem = (size_t)3 * PA_BN * (D + 8) * sizeof(__nv_bfloat16);
    static std::atomic<uint64_t> smem_opt_in{0};
    opt_in_dynamic_smem(cmd, attn_prefill_kernel<D, PLANES>, (int)smem, smem_opt_in);
    const uint32_t row_tiles = (a.suffix_length * a.gqa_factor + PA_BM - 1) / PA_BM, kv_heads = a.num_heads / a.gqa_factor, splits = pa_splits(a, (uint32_t)cmd->ctx->sm_count);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(row_tiles * splits, kv_heads);
    cfg.blockDim = dim3(128);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = cmd->ctx->stream;
    cudaLaunchAttribute attr[1];
    cfg.attrs = attr;
    if (splits > 1) {
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = splits;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.numAttrs = 1;
    }
    else if (cmd->dependent()) {      // (not clusters: started beside the last CTAs of the kernel before, they share SMs that others leave idle, 31 us -> 44 for 16 rows and 2048 keys)
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.numAttrs = 1;
    }
    const cudaError_t e = cudaLaunchKernelEx(&cfg, attn_prefill_kernel<D, PLANES>, a, splits);
    if (e != cudaSuccess) cmd->record_error(UZU_ERROR_CUDA, std::string("attn_prefill_kernel: ") + cudaGetErrorString(e));
    cmd->launches++;
}

// true = handled: where it is the faster kernel, for a dense prefix, a plain mask or a causal trie
static int g_prefill_attn = -1;   // -1: follow UZU_PREFILL_ATTN and the rule, 0: never, 1: wherever it can, 2: the tcgen05 kernel wherever that can (uzu_debug_set_prefill_attention)

bool encode_attention_prefill(uzu_command_buffer* cmd, const uzu_attention_args& a) {
    static const bool env_enabled = [] { const char* e = getenv("UZU_PREFILL_ATTN"); return !e || atoi(e) != 0; }();   // =0 keeps the split-KV kernel
    if (!(g_prefill_attn < 0 ? env_enabled : g_prefill_attn != 0)) return false;
    if (a.suffix_length < 2 || a.dynamic_position || a.has_sinks || a.is_kv_cache_ring || a.is_sliding_window) return false;
    if (a.is_trie && (!a.is_causal || !a.trie)) return false;
    if (a.head_dim != 64 && a.head_dim != 128 && a.head_dim != 256) return false;
    if (a.gqa_factor == 0 || a.num_heads % a.gqa_factor || (uint64_t)a.suffix_length * a.gqa_factor > 0x7fffffffull) return false;
    if ((a.k_head_stride % 8) || (a.v_head_stride % 8) || (a.k_seq_stride % 8) || (a.v_seq_stride % 8)) return false;   // 16-byte cp.async rows
    if ((a.queries | a.keys | a.values | a.out) & 15u) return false;
    if (a.sequence_length < a.suffix_length) return false;
    const bool two = pa_two_planes(a);
    PaKernel kernel = g_prefill_attn == 1 ? PaKernel::Mma : g_prefill_attn == 2 ? PaKernel::Umma : pa_choose(a, (uint32_t)cmd->ctx->sm_count);
    if (kernel == PaKernel::Umma) {
        if (attn_umma_applicable(a) && encode_attn_umma(cmd, a, two ? 2u : 3u)) return true;
        kernel = g_prefill_attn == 2 ? PaKernel::Split : PaKernel::Mma;
    }
    if (kernel == PaKernel::Split) return false;
    if (a.head_dim == 64) two ? launch_attn_prefill<64, 2>(cmd, a) : launch_attn_prefill<64, 3>(cmd, a);
    else if (a.head_dim == 128) two ? launch_attn_prefill<128, 2>(cmd, a) : launch_attn_prefill<128, 3>(cmd, a);
    else launch_attn_prefill<256, 3>(cmd, a);
    return true;
}

}  // namespace uzu

extern "C" void uzu_debug_set_prefill_attention(int mode) { uzu::g_prefill_attn = mode; }
