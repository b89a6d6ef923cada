// Quantised MatmulKernel for more than 32 activation rows (qmm_rows.cu; other groups: from 3 rows) on the 5th-generation tensor cores: D[m, n] = epilogue(A[m, k] * dequant(B[n, k])^T).
// Semantic spec: backends/cpu/kernel/matmul/kernel.rs:164-295 (caller encodable_block/linear/matmul.rs:122-148).
//
// Weights are turned in the kernel into TWO bf16 planes, hi = bf16(w) and lo = w - hi. For ZeroPoint / Symmetric weights w = scale * (code - zp) has
// at most 16 significant bits, so hi + lo is w exactly; for MLX weights (scale * code + bias in f32) the remainder is below 2^-17 |w|. A single
// rounded plane would put 2^-9 on every weight. The products are exact, the sums f32 in tensor memory.
//
// CTA = 128 output features x NT activation rows (the products' M and N), K in blocks of 64; warps:
//   dequant    three or four groups of four, each takes every third or fourth block: a thread owns a feature row, turns its 64 codes and stores both
//              planes to TENSOR MEMORY (tcgen05.st). The weights are the products' A operand there, so that shared memory feeds the activations
//              only: a product that reads both operands from shared memory is capped at half of the tensor rate, and that was the bound of the
//              kernel before this one (128 x 128 tiles; 1024 rows x 28672 x 4096 in 579 us).
//   one warp each: TMA of the codes (128 rows x 128 bytes, 128B swizzle), TMA of the activations (NT rows x 128 k a stage), and the products
//              (tcgen05.mma, 8 a block). What one lane issues stands behind elect.sync: there an instruction takes about 10 clocks to issue, behind
//              `lane == 0` about 300, and the product warp was the bound.
//   epilogue   four: finished tiles from tensor memory (a feature per lane, a row per column) to D; next to the following tile's products for NT <= 64
//              (two accumulators).
// CTAs stay for several tiles; where the tiles do not fill the chip (few rows, few features) a cluster of up to 8 CTAs shares a tile's k and adds
// its partial tiles over distributed shared memory in rank order (the same bits every time).
// (Tried instead: integer codes as one plane, group scales applied to the partial sums as they leave tensor memory. Half the products, but reading
// 128 x NT partial sums per 64 k costs more than that: 815 us at the size above. With eight warps for the sums, chains of 128 k and 4-bit codes it pays: qmm_wide.cu.)
// Tiles of up to 64 rows of ZeroPoint / Symmetric weights in groups of 64 and more take ONE plane, the integers code - zp (exact in bf16): half the products,
// half the stores to tensor memory and no scale in the dequant warps. A chain of at most 128 k inside a group is summed unscaled; the epilogue warps (eight
// for 64 rows) bring each chain to their sums with one rounded multiply-add by its scale. For wider tiles reading 128 x NT sums per 64 k costs more than the
// second plane (128 rows: 180 us with two planes, 187 with one). A layer of an 8B model, two planes / integers: 40 rows 153 / 140 us, in groups of 128
// 160 / 131, 8-bit 201 / 176; 60 rows 170 / 155; groups of 32 187 / 225, so they keep the planes.
//
// Bounds, per block and CTA: the tensor pipe 4 NT cycles; the dequant warps about 230 instructions each, four warps a block. Prompts are bound by the
// tensor pipe (half of its rate is the most two planes can give), few rows by the way of a
// block through its roles (28672 x 4096 at 40 rows: 1000 cycles per 64 k with fill and drain, issue slots 56 % used, tensor pipe 10 %); more dequant groups
// and a product role of one lane changed nothing.
// Every barrier wait is bounded (about a second): a wait that runs out is reported (wait_errors.h: the call then fails on the host) and the CTA ends its work.
#include <cstdlib>
#include <type_traits>

#include "qmm_scaled.cuh"

namespace uzu {

namespace {

template <int NT, int PL>
struct QsShape {
    // PL = 1: the codes as integers; a group's sum is scaled as it leaves tensor memory
    static constexpr int EW = PL == 1 && NT == 64 ? 8 : 4, EC = NT * 4 / EW;      // epilogue warps and the columns of one
    // dequant groups: a block takes one about 2000 cycles, hardly a third of them issuing
    static constexpr int DG = PL == 1 && NT < 64 ? 4 : NT > 128 || NT == 64 || PL == 3 ? 3 : 4;
    static constexpr int ND = PL == 1 ? 4 : NT > 64 ? 1 : 2;    // accumulators in tensor memory
    static constexpr int CHAIN = NT > 64 ? 0 : 2;                            // blocks whose products share an accumulator (0: all)
    static constexpr int AS = PL == 1 ? 8 : NT > 192 || PL == 3 ? 4 : NT > 128 ? 5 : 6;    // weight blocks in tensor memory: 32 columns a plane
    static constexpr int BS = NT > 192 ? 2 : NT > 64 ? 3 : 4;                // activation stages of 128 k
    static constexpr int CS = NT > 64 ? 4 : 8;                               // code tiles
    static constexpr int THREADS = (EW + 4 * DG + 3) * 32;
    static constexpr uint32_t ACT = NT * 256, COLS = 32 * PL, A_COL = 512 - COLS * AS;
    static constexpr size_t SMEM = (size_t)BS * ACT + (size_t)CS * QS_CODE_TILE + 1024;
    static_assert(ND * NT <= (int)A_COL && DG < AS, "tensor memory columns; a group never waits for its own block");
    static_assert(PL == 1 || (CHAIN % 2 == 0 && (CHAIN == 0 || ND == 2)), "a chain is whole activation stages; the next one runs while its sums are taken");
    static_assert((size_t)NT * 512 <= (size_t)BS * ACT + (size_t)CS * QS_CODE_TILE, "the split-k exchange reuses the rings");
};

// MLX: the reference's scale * code + bias in f32, then its planes: bf16 of what is left, three hold all of it
template <int PL>
__device__ __forceinline__ void qs_planes_f32(float w0, float w1, uint32_t (&plane)[PL][16], uint32_t at) {
#pragma unroll
    for (int i = 0; i < PL; ++i) {
        const uint32_t h = qs_u(__floats2bfloat162_rn(w0, w1));
        plane[i][at] = h;
        w0 -= __uint_as_float(h << 16);
        w1 -= __uint_as_float(h & 0xFFFF0000u);
    }
}

__device__ __forceinline__ void qs_finish(const QsParams& p, float sum, uint32_t token, uint32_t row) {
    if (token >= p.m || row >= p.n) return;
    const size_t at = (size_t)token * p.n + row;
    float val = __fmul_rn(p.ab_scale, sum);                                  // separate roundings, like the reference
    if (p.accumulate) val = __fadd_rn(val, p.d_is_f32 ? reinterpret_cast<const float*>(p.d)[at] : bf2f(reinterpret_cast<const __nv_bfloat16*>(p.d)[at]));
    if (p.bias) val = __fadd_rn(val, bf2f(p.bias[row]));
    if (p.has_soft_cap) val = __fmul_rn(p.soft_cap, tanhf(__fdiv_rn(val, p.soft_cap)));
    if (p.d_is_f32) reinterpret_cast<float*>(p.d)[at] = val;
    else reinterpret_cast<__nv_bfloat16*>(p.d)[at] = f2bf(val);
}
// Columns `first`, `first` + step, .. of a tile whose partial sums lie in the shared memory of a cluster's CTAs, at `own` in each (this thread's feature, 512 bytes a
// column), added in rank order. (Not part of the kernel's body: there it cost the tiles that share nothing a tenth of their time.)
__device__ __noinline__ void qs_exchange(const QsParams& params, uint32_t own, uint32_t first, uint32_t step, uint32_t columns, uint32_t t0, uint32_t row) {
    const QsParams p = params;                                               // (in registers: read again for each column, 7 us at 256 columns)
    uint32_t remote[8];
#pragma unroll
    for (uint32_t q = 0; q < 8; ++q) asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote[q]) : "r"(own), "r"(min(q, p.splits - 1u)));
    for (uint32_t j0 = first; j0 < columns; j0 += 4 * step) {
        float part[4][8];
#pragma unroll
        for (uint32_t u = 0; u < 4; ++u) {
            const uint32_t at = min(j0 + u * step, columns - 1u) * 512u;
#pragma unroll
            for (uint32_t q = 0; q < 8; ++q) {
                part[u][q] = 0.0f;
                if (q < p.splits) asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(part[u][q]) : "r"(remote[q] + at) : "memory");
            }
        }
#pragma unroll
        for (uint32_t u = 0; u < 4; ++u) {
            if (j0 + u * step >= columns) continue;
            float sum = part[u][0];
#pragma unroll
            for (int q = 1; q < 8; ++q) sum += part[u][q];
            qs_finish(p, sum, t0 + j0 + u * step, row);
        }
    }
}

}  // namespace

template <int BITS, int NT, int PL>
__global__ void __launch_bounds__(QsShape<NT, PL>::THREADS, 1) qmm_scaled_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const __grid_constant__ QsParams p) {
    using S = QsShape<NT, PL>;
    constexpr int DG = S::DG, ND = S::ND, AS = S::AS, BS = S::BS, CS = S::CS, DQ_WARPS = 4 * DG, EW = S::EW, EC = S::EC;
    constexpr uint32_t kpt = BITS == 4 ? 4u : 2u;                            // k blocks per code tile
    extern __shared__ uint8_t qs_raw[];
    __shared__ __align__(8) uint64_t bars[2 * CS + 2 * BS + 2 * AS + 2 * ND + 1];
    __shared__ uint32_t tmem_slot;
    __shared__ volatile uint32_t gave_up;
    const uint32_t tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;     // (warp: the same in every lane)
    const uint32_t base = (qs_smem(qs_raw) + 1023u) & ~1023u;            // swizzle atoms sit on 1024-byte boundaries
    const uint32_t act0 = base, code0 = base + BS * S::ACT, bar0 = qs_smem(bars);
    auto code_full = [&](uint32_t i) { return bar0 + 8u * i; };
    auto code_empty = [&](uint32_t i) { return bar0 + 8u * (CS + i); };
    auto act_full = [&](uint32_t i) { return bar0 + 8u * (2 * CS + i); };
    auto act_empty = [&](uint32_t i) { return bar0 + 8u * (2 * CS + BS + i); };
    auto a_full = [&](uint32_t i) { return bar0 + 8u * (2 * CS + 2 * BS + i); };
    auto a_empty = [&](uint32_t i) { return bar0 + 8u * (2 * CS + 2 * BS + AS + i); };
    auto d_full = [&](uint32_t i) { return bar0 + 8u * (2 * CS + 2 * BS + 2 * AS + i); };
    auto d_empty = [&](uint32_t i) { return bar0 + 8u * (2 * CS + 2 * BS + 2 * AS + ND + i); };
    const uint32_t last_products = bar0 + 8u * (2 * CS + 2 * BS + 2 * AS + 2 * ND);

    if (warp == 0) {
        if (lane == 0) {
            for (int i = 0; i < CS; ++i) { qs_init(code_full(i), 1); qs_init(code_empty(i), DQ_WARPS); }
            for (int i = 0; i < BS; ++i) { qs_init(act_full(i), 1); qs_init(act_empty(i), 1); }
            for (int i = 0; i < AS; ++i) { qs_init(a_full(i), 4); qs_init(a_empty(i), 1); }
            for (int i = 0; i < ND; ++i) { qs_init(d_full(i), 1); qs_init(d_empty(i), EW); }
            qs_init(last_products, 1);
            gave_up = 0;
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(qs_smem(&tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    qs_fence_before();
    __syncthreads();
    qs_fence_after();
    const uint32_t tmem = tmem_slot;
    pdl_launch_dependents();      // (not before this CTA has its tensor memory: a dependent's CTA that took it would wait for this one)

    // this CTA's work: items blockIdx.x / splits, then in steps of the grid; the k blocks of its rank
    const uint32_t rank = p.splits > 1 ? blockIdx.x % p.splits : 0u, item0 = blockIdx.x / p.splits, item_step = gridDim.x / p.splits;
    const uint32_t kb0 = rank * p.split_kb, nk = min(p.split_kb, p.nkb - kb0);       // (every rank has some)
    const uint32_t tiles = (nk + kpt - 1) / kpt;                                     // code tiles per item
    // neighbouring items share their weights: the row tiles of a feature tile are in flight together
    auto item_n = [&](uint32_t item) { return item / p.m_tiles * 128u; };
    auto item_m = [&](uint32_t item) { return item % p.m_tiles * (uint32_t)NT; };

    if (warp < (uint32_t)EW) {
        // ================================ finished tiles ================================
        uint32_t buf = 0, ph = 0;
        pdl_wait();                                                      // D may be read (accumulate) and is written below
        for (uint32_t item = item0; item < p.items; item += item_step) {
            const uint32_t lanes = (warp & 3u) * 32u, cb = (warp >> 2) * EC, f = lanes + lane, row = item_n(item) + f, t0 = item_m(item);      // cb: this warp's first column
            const uint32_t columns = min((uint32_t)NT, p.m - t0);
            bool ok = true;
            constexpr bool kSums = PL == 1 || S::CHAIN != 0;
            float acc[kSums ? EC : 1];                                   // sums of the chains (else they stay in tensor memory until they are stored)
            if constexpr (kSums) {
#pragma unroll
                for (int c = 0; c < EC; ++c) acc[c] = 0.0f;
            }
            auto next = [&]() {
                qs_fence_before();
                __syncwarp();
                if (lane == 0) qs_arrive(d_empty(buf));
                if (++buf == (uint32_t)ND) { buf = 0; ph ^= 1u; }
            };
            if constexpr (PL == 1) {
                // a chain is a group or a part of one: its exact integer products were summed unscaled; one rounded multiply-add brings it to the sums
                const uint32_t chains = (nk * 64u + p.chain_k - 1) / p.chain_k, last = p.groups - 1u;
                const uint16_t* srow = reinterpret_cast<const uint16_t*>(p.scales) + (size_t)min(row, p.n - 1u) * p.groups;
                auto scale_of = [&](uint32_t i) { return (uint32_t)__ldg(srow + min((kb0 * 64u + i * p.chain_k) >> p.gshift, last)); };
                uint32_t ahead[4];                                       // scales of the next four chains
#pragma unroll
                for (int u = 0; u < 4; ++u) ahead[u] = scale_of(u);
                for (uint32_t i0 = 0; i0 < chains && ok; i0 += 4) {
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        if (i0 + u >= chains || !ok) continue;
                        ok = qs_wait(d_full(buf), ph, &gave_up, p.error, 0x101u);
                        qs_fence_after();
                        const float scale = __uint_as_float(ahead[u] << 16);
                        ahead[u] = scale_of(i0 + u + 4);
#pragma unroll
                        for (uint32_t c0 = 0; c0 < (uint32_t)EC; c0 += 16) {
                            if (cb + c0 >= columns || !ok) continue;
                            uint32_t v[16];
                            qs_tmem_ld16(tmem + (lanes << 16) + buf * NT + cb + c0, v);
#pragma unroll
                            for (int j = 0; j < 16; ++j) acc[c0 + j] = fmaf(scale, __uint_as_float(v[j]), acc[c0 + j]);
                        }
                        if (ok) next();
                    }
                }
#pragma unroll
                for (int c = 0; c < EC; ++c) acc[c] *= qs_unit<BITS>;
            } else
            for (uint32_t i = 0; i < (S::CHAIN ? nk : 1u) && ok; i += S::CHAIN ? S::CHAIN : 1) {
                ok = qs_wait(d_full(buf), ph, &gave_up, p.error, 0x101u);
                qs_fence_after();
                if constexpr (S::CHAIN != 0) {
#pragma unroll
                    for (uint32_t c0 = 0; c0 < (uint32_t)NT; c0 += 16) {
                        if (c0 >= columns || !ok) continue;
                        uint32_t v[16];
                        qs_tmem_ld16(tmem + ((warp * 32u) << 16) + buf * NT + c0, v);
#pragma unroll
                        for (int j = 0; j < 16; ++j) acc[c0 + j] += __uint_as_float(v[j]);
                    }
                    if (ok) next();
                }
            }
            // f(c0, the sums of columns c0 .. c0 + 15) for the tile's columns
            auto each16 = [&](auto f) {
                if constexpr (kSums) {
#pragma unroll
                    for (uint32_t c0 = 0; c0 < (uint32_t)EC; c0 += 16)
                        if (cb + c0 < columns && ok) f(cb + c0, acc + c0);
                } else {
                    for (uint32_t c0 = 0; c0 < columns && ok; c0 += 16) {
                        uint32_t v[16];
                        qs_tmem_ld16(tmem + ((warp * 32u) << 16) + buf * NT + c0, v);
                        f(c0, reinterpret_cast<const float*>(v));
                    }
                }
            };
            if (p.splits == 1 && p.plain && item_n(item) + 128u <= p.n) {
                // D is the rounded sum: a store per column (64 neighbouring bytes a warp), no more than an address step between them
                __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(p.d) + (size_t)(t0 + cb) * p.n + row;
                each16([&](uint32_t c0, const float* v) {
                    if (c0 + 16 <= columns) {
#pragma unroll
                        for (int j = 0; j < 16; ++j, out += p.n) *out = f2bf(v[j]);
                    } else {
#pragma unroll
                        for (int j = 0; j < 16; ++j, out += p.n)
                            if (c0 + j < columns) *out = f2bf(v[j]);
                    }
                });
            } else if (p.splits == 1) {
                each16([&](uint32_t c0, const float* v) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) qs_finish(p, v[j], t0 + c0 + j, row);
                });
            } else {
                // this CTA's tile to shared memory (the rings are idle: every block has been consumed); below, column shares over the cluster
                each16([&](uint32_t c0, const float* v) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) asm volatile("st.shared.f32 [%0], %1;" ::"r"(base + ((c0 + j) * 128u + f) * 4u), "f"(v[j]) : "memory");
                });
                break;                                                   // (one item per cluster)
            }
            if (!ok) break;
            if constexpr (!kSums) next();
        }
    } else if (warp < (uint32_t)(EW + DQ_WARPS)) {
        // ================================ codes -> two bf16 planes in tensor memory ================================
        const uint32_t dg = (warp - EW) >> 2, lw = warp & 3u, r = lw * 32u + lane;
        const bool mlx = PL == 3 || p.method == UZU_QMETHOD_SCALE_BIAS, has_zp = p.method == UZU_QMETHOD_SCALE_ZERO_POINT, halves = p.gshift == 5u;
        uint32_t turn = 0, stage = dg, a_ph = 1, slot = 0, c_ph = 0;     // whose block it is; this group's next weight block; code tile
        bool ok = true;
        for (uint32_t item = item0; item < p.items && ok; item += item_step) {
            const uint32_t brow = min(item_n(item) + r, p.n - 1u);
            const uint16_t* srow = reinterpret_cast<const uint16_t*>(p.scales) + (size_t)brow * p.groups;
            const uint16_t* crow = reinterpret_cast<const uint16_t*>(p.biases) + (size_t)brow * p.groups;
            const uint8_t* zrow = p.zero_points + (size_t)brow * p.zp_stride;
            // scale | (zero point or bias) << 16 of a half block, requested a turn ahead
            auto factor = [&](uint32_t k) -> uint32_t {
                const uint32_t g = min(k >> p.gshift, p.groups - 1u);
                uint32_t c = BITS == 4 ? 8u : 128u;
                if (mlx) c = crow[g];
                else if (has_zp) c = BITS == 4 ? (uint32_t)(zrow[g >> 1] >> (4u * (g & 1u))) & 15u : (uint32_t)zrow[g];
                return (PL == 1 ? 0u : (uint32_t)srow[g]) | c << 16;
            };
            auto first_block = [&]() -> uint32_t { return (dg + DG - turn) % DG; };      // blocks until this group's turn
            uint32_t f_next[2];
            {
                const uint32_t k0 = (kb0 + first_block()) * 64u;
                f_next[0] = factor(k0);
                f_next[1] = halves ? factor(k0 + 32u) : f_next[0];
            }
            for (uint32_t tile = 0, kb = 0; tile < tiles; ++tile) {
                ok = qs_wait(code_full(slot), c_ph, &gave_up, p.error, 0x102u);
                if (!ok) break;
                const uint32_t line = code0 + slot * QS_CODE_TILE + r * 128u, blocks = min(kpt, nk - kb);
#pragma unroll 1
                for (uint32_t j = 0; j < blocks; ++j, ++kb) {
                    const bool mine = turn == dg;
                    if (++turn == (uint32_t)DG) turn = 0;
                    if (!mine) continue;
                    const uint32_t f_cur[2] = {f_next[0], f_next[1]};
                    {
                        const uint32_t k0 = (kb0 + kb + DG) * 64u;
                        f_next[0] = factor(k0);
                        f_next[1] = halves ? factor(k0 + 32u) : f_next[0];
                    }
                    const uint32_t t_col = tmem + ((lw * 32u) << 16) + S::A_COL + stage * S::COLS;
#pragma unroll
                    for (uint32_t h = 0; h < 2; ++h) {                   // 32 k at a time
                        uint32_t plane[PL][16], (&hi)[16] = plane[0], (&lo)[16] = plane[PL > 1 ? 1 : 0];
                        const uint32_t s1 = f_cur[h] & 0xFFFFu, z = f_cur[h] >> 16, s2 = s1 * 0x00010001u;
                        if constexpr (BITS == 4) {
                            uint32_t q[4];
                            asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(q[0]), "=r"(q[1]), "=r"(q[2]), "=r"(q[3]) : "r"(line + (((j * 2 + h) ^ (r & 7u)) << 4)));
                            const uint32_t z2 = ((PL == 1 ? qs_base<4> : 0x4300u) | z) * 0x00010001u;      // bf16 128 + zp
                            if constexpr (PL == 1) {
#pragma unroll
                                for (int i = 0; i < 4; ++i) qs_integers4(q[i] ^ p.xor_mask, z2, hi + 4 * i);
                            } else if (!mlx) {
#pragma unroll
                                for (int i = 0; i < 4; ++i) qs_dequant4(q[i] ^ p.xor_mask, z2, s2, hi + 4 * i, lo + 4 * i);
                            } else {
                                const float s = __uint_as_float(s1 << 16), c = __uint_as_float(z << 16);
#pragma unroll
                                for (int i = 0; i < 16; ++i) {           // pair i: nibbles 2 (i & 3), + 1 of word i / 4
                                    const uint32_t w = (q[i >> 2] ^ p.xor_mask) >> (8 * (i & 3));
                                    qs_planes_f32<PL>(fmaf(s, (float)(w & 15u), c), fmaf(s, (float)((w >> 4) & 15u), c), plane, i);
                                }
                            }
                        } else {
#pragma unroll
                            for (uint32_t i2 = 0; i2 < 2; ++i2) {
                                uint32_t q[4];
                                asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(q[0]), "=r"(q[1]), "=r"(q[2]), "=r"(q[3]) : "r"(line + (((j * 4 + h * 2 + i2) ^ (r & 7u)) << 4)));
                                constexpr uint32_t base = PL == 1 ? qs_base<8> : 0x4300u;
                                const uint32_t zh2 = (base | (z >> 4)) * 0x00010001u, zl2 = (base | (z & 15u)) * 0x00010001u;
                                if constexpr (PL == 1) {
#pragma unroll
                                    for (int i = 0; i < 4; ++i) qs_integers8(q[i] ^ p.xor_mask, zh2, zl2, hi + 8 * i2 + 2 * i);
                                } else if (!mlx) {
#pragma unroll
                                    for (int i = 0; i < 4; ++i) qs_dequant8(q[i] ^ p.xor_mask, zh2, zl2, s2, hi + 8 * i2 + 2 * i, lo + 8 * i2 + 2 * i);
                                } else {
                                    const float s = __uint_as_float(s1 << 16), c = __uint_as_float(z << 16);
#pragma unroll
                                    for (int i = 0; i < 8; ++i) {
                                        const uint32_t w = (q[i >> 1] ^ p.xor_mask) >> (16 * (i & 1));
                                        qs_planes_f32<PL>(fmaf(s, (float)(w & 255u), c), fmaf(s, (float)((w >> 8) & 255u), c), plane, 8 * i2 + i);
                                    }
                                }
                            }
                        }
                        if (h == 0) {
                            ok = qs_wait(a_empty(stage), a_ph, &gave_up, p.error, 0x103u);
                            if (!ok) break;
                            qs_fence_after();
                        }
#pragma unroll
                        for (int i = 0; i < PL; ++i) qs_tmem_st16(t_col + 32u * i + h * 16u, plane[i]);
                    }
                    if (!ok) break;
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    qs_fence_before();
                    __syncwarp();
                    if (lane == 0) qs_arrive(a_full(stage));
                    stage += DG;
                    if (stage >= (uint32_t)AS) { stage -= AS; a_ph ^= 1u; }
                }
                if (!ok) break;
                __syncwarp();
                if (lane == 0) qs_arrive(code_empty(slot));
                if (++slot == (uint32_t)CS) { slot = 0; c_ph ^= 1u; }
            }
        }
    } else {
        const uint32_t role = warp - (EW + DQ_WARPS);
        bool ok = true;
        if (role == 0) {
            // ================================ codes by TMA (they depend on no kernel) ================================
            uint32_t slot = 0, ph = 1, asked = 0;
            for (uint32_t item = item0; item < p.items && ok; item += item_step) {
                const uint32_t y = item_n(item), x0 = kb0 / kpt * 128u;
                for (uint32_t tile = 0; tile < tiles; ++tile) {
                    ok = qs_wait(code_empty(slot), ph, &gave_up, p.error, 0x104u);
                    if (!ok) break;
                    if (qs_elect()) {
                        qs_expect(code_full(slot), QS_CODE_TILE);
                        qs_tma_2d(code0 + slot * QS_CODE_TILE, &map_w, x0 + tile * 128u, y, code_full(slot));
                    }
                    __syncwarp();
                    ++asked;
                    if (++slot == (uint32_t)CS) { slot = 0; ph ^= 1u; }
                }
            }
            if (!ok)
                for (uint32_t n = asked > (uint32_t)CS ? asked - CS : 0; n < asked; ++n) qs_settle(code_full(n % CS), n / CS & 1u);
        } else if (role == 1) {
            // ================================ activations by TMA, 128 k a stage ================================
            uint32_t slot = 0, ph = 1, asked = 0;
            pdl_wait();
            for (uint32_t item = item0; item < p.items && ok; item += item_step) {
                const uint32_t y = item_m(item);
                for (uint32_t i = 0; i < nk; i += 2) {
                    ok = qs_wait(act_empty(slot), ph, &gave_up, p.error, 0x105u);
                    if (!ok) break;
                    if (qs_elect()) {                                    // (a half stage behind the last k reads zeros)
                        qs_expect(act_full(slot), S::ACT);
                        qs_tma_2d(act0 + slot * S::ACT, &map_x, (kb0 + i) * 64u, y, act_full(slot));
                        qs_tma_2d(act0 + slot * S::ACT + S::ACT / 2, &map_x, (kb0 + i + 1) * 64u, y, act_full(slot));
                    }
                    __syncwarp();
                    ++asked;
                    if (++slot == (uint32_t)BS) { slot = 0; ph ^= 1u; }
                }
            }
            if (!ok)
                for (uint32_t n = asked > (uint32_t)BS ? asked - BS : 0; n < asked; ++n) qs_settle(act_full(n % BS), n / BS & 1u);
        } else {
            // ================================ products ================================
            // shared-memory descriptor: K-major SWIZZLE_128B, 1024 bytes between 8-row groups, +32 bytes per 16 k
            constexpr uint64_t desc_hi = (uint64_t)((1024u >> 4) | (1u << 14) | (2u << 29)) << 32;
            constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(NT >> 3) << 17) | ((128u >> 4) << 24);
            const uint32_t desc_lo = (act0 >> 4) | (1u << 16);
            uint32_t bs = 0, bs_ph = 0, as = 0, as_ph = 0, buf = 0, d_ph = 1;
            for (uint32_t item = item0; item < p.items && ok; item += item_step) {
                if constexpr (PL == 1) {
                    const bool pairs = p.chain_k == 128u;                // a chain is two blocks or one
                    for (uint32_t i = 0; i < nk && ok; i += 2) {
                        ok = qs_wait(act_full(bs), bs_ph, &gave_up, p.error, 0x106u);
#pragma unroll
                        for (uint32_t half = 0; half < 2; ++half) {
                            if (i + half >= nk || !ok) continue;
                            const bool begins = !pairs || half == 0, ends = !pairs || half == 1 || i + half + 1 >= nk;
                            ok = qs_wait(a_full(as), as_ph, &gave_up, p.error, 0x107u);
                            if (begins && ok) ok = qs_wait(d_empty(buf), d_ph, &gave_up, p.error, 0x108u);
                            if (!ok) break;
                            qs_fence_after();
                            if (qs_elect()) {
                                const uint32_t d = tmem + buf * NT, a_col = tmem + S::A_COL + as * S::COLS, lo = desc_lo + (bs * S::ACT + half * (S::ACT / 2) >> 4);
#pragma unroll
                                for (uint32_t kk = 0; kk < 4; ++kk) qs_mma(d, a_col + kk * 8u, desc_hi | (lo + kk * 2u), idesc, !begins || kk != 0 ? 1u : 0u);
                                qs_commit(a_empty(as));
                                if (ends) qs_commit(d_full(buf));
                            }
                            __syncwarp();
                            if (++as == (uint32_t)AS) { as = 0; as_ph ^= 1u; }
                            if (ends && ++buf == (uint32_t)ND) { buf = 0; d_ph ^= 1u; }
                        }
                        if (!ok) break;
                        if (qs_elect()) qs_commit(act_empty(bs));
                        __syncwarp();
                        if (++bs == (uint32_t)BS) { bs = 0; bs_ph ^= 1u; }
                    }
                } else
                for (uint32_t i = 0; i < nk && ok; i += 2) {
                    const bool begins = S::CHAIN ? i % (S::CHAIN ? S::CHAIN : 1) == 0 : i == 0, ends = i + 2 >= nk || (S::CHAIN && (i + 2) % (S::CHAIN ? S::CHAIN : 1) == 0);
                    const uint32_t d = tmem + buf * NT;
                    if (begins) ok = qs_wait(d_empty(buf), d_ph, &gave_up, p.error, 0x108u);
                    if (!ok) break;
                    ok = qs_wait(act_full(bs), bs_ph, &gave_up, p.error, 0x106u);
                    if (!ok) break;
#pragma unroll
                    for (uint32_t half = 0; half < 2; ++half) {
                        if (i + half >= nk) continue;
                        ok = qs_wait(a_full(as), as_ph, &gave_up, p.error, 0x107u);
                        if (!ok) break;
                        qs_fence_after();
                        if (qs_elect()) {
                            const uint32_t a_col = tmem + S::A_COL + as * S::COLS, lo = desc_lo + (bs * S::ACT + half * (S::ACT / 2) >> 4);
#pragma unroll
                            for (uint32_t kk = 0; kk < 4; ++kk) {
#pragma unroll
                                for (uint32_t pl = 0; pl < (uint32_t)PL; ++pl) qs_mma(d, a_col + 32u * pl + kk * 8u, desc_hi | (lo + kk * 2u), idesc, !begins || (half | kk | pl) != 0 ? 1u : 0u);
                            }
                            qs_commit(a_empty(as));
                        }
                        __syncwarp();
                        if (++as == (uint32_t)AS) { as = 0; as_ph ^= 1u; }
                    }
                    if (!ok) break;
                    if (qs_elect()) qs_commit(act_empty(bs));
                    __syncwarp();
                    if (++bs == (uint32_t)BS) { bs = 0; bs_ph ^= 1u; }
                    if (!ends) continue;
                    if (qs_elect()) qs_commit(d_full(buf));
                    __syncwarp();
                    if (++buf == (uint32_t)ND) { buf = 0; d_ph ^= 1u; }
                }
            }
            if (!ok) {
                if (qs_elect()) qs_commit(last_products);
                __syncwarp();
                qs_settle(last_products, 0);                             // none in flight when tensor memory is given back
            }
        }
        __syncwarp();
    }
    if (p.splits > 1) {
        // A rank's columns of the tile: the partial sums of all ranks in rank order. The warps that turned codes help, and loads of four columns are in flight (the
        // epilogue warps alone, a column at a time, took 25 us for 256 columns of two ranks).
        qs_cluster_sync();
        if (warp < (uint32_t)(EW + DQ_WARPS)) {
            if (warp >= (uint32_t)EW) pdl_wait();                        // (the epilogue's have waited: D may be read)
            const uint32_t f = (warp & 3u) * 32u + lane, t0 = item_m(item0);
            qs_exchange(p, base + f * 4u, rank + p.splits * (warp >> 2), p.splits * ((EW + DQ_WARPS) / 4), min((uint32_t)NT, p.m - t0), t0, item_n(item0) + f);
        }
        qs_cluster_sync();      // no CTA of a cluster leaves while another may still read its tile
    }
    qs_fence_before();
    __syncthreads();
    if (warp == 0) {
        qs_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

// ---- host side -------------------------------------------------------------------------------------------------------------------------
bool qmm_scaled_applicable(const uzu_matmul_args& a) {
    static const bool off = [] { const char* e = getenv("UZU_QMM_SCALED"); return e && atoi(e) == 0; }();      // 0: the kernels for other shapes (A/B runs)
    static const int min_rows = [] { const char* e = getenv("UZU_PREFILL_GEMM_MIN_M"); return e ? atoi(e) : 2; }();      // fewer rows take the other kernels; 0: all do
    if (off || min_rows <= 0 || a.m < 2 || a.m < (uint32_t)min_rows) return false;
    if (a.b_prologue == UZU_B_FULL_PRECISION || a.gather_indices || !a.b_transpose) return false;
    if (a.input_dt != UZU_DT_BF16 || a.weights_dt != UZU_DT_BF16) return false;
    if (a.output_dt != UZU_DT_BF16 && a.output_dt != UZU_DT_F32) return false;
    if (a.b_mode != UZU_QMODE_U4 && a.b_mode != UZU_QMODE_U8) return false;
    const uint32_t gs = a.b_group_size;
    if (a.k == 0 || a.k > (1u << 18) || a.n == 0 || a.k % 64u != 0 || gs < 32 || (gs & (gs - 1)) != 0 || a.k % gs != 0) return false;
    if ((a.a & 15u) || (a.b & 15u)) return false;            // TMA operands (their pitches are multiples of 32 bytes with k a multiple of 64)
    // two rows with groups of 32 or 256 (64 and 128: qmm_rows.cu): the streaming kernel of matmul.cu, which reads whole 512-nibble steps. A layer of an
    // 8B model, MLX groups of 32: 2 rows 150 us there, 176 here; 4 rows 199 and 155
    const uint32_t bits = a.b_mode == UZU_QMODE_U4 ? 4 : 8;
    if (a.m <= 2 && a.k * bits % 2048u == 0) return false;
    // MLX with groups of 256: three planes cost more than the streaming kernel up to 8 rows. A layer of an 8B model: 3 rows 130 us there, 168 here; 8 rows
    // 166 and 169; 9 rows 216 and 170
    if (a.m <= 8 && bits == 4 && gs == 256 && a.b_prologue == UZU_B_SCALE_BIAS_DEQUANT && a.k * bits % 2048u == 0) return false;
    // 17 .. 63 rows over a matrix of at most 2^21 weights with groups of 64 or 128: launches of 16 rows (qmm_rows.cu, with the times)
    if (a.m > 16 && a.m < 64 && (uint64_t)a.n * a.k <= (1u << 21) && (gs == 64 || gs == 128)) return false;
    return tensor_map_encoder() != nullptr;
}

namespace {

struct QsPlan { int nt = 0; uint32_t splits = 1; float cost = 1e30f; };

// The plan's estimate in us: 5 for a launch; for each turn of the chip, what filling the pipeline and storing a tile of that many rows take, and 64 k as often as a CTA
// has them; where CTAs share a tile's k, their exchange. Fitted to 3500 times of 13 matrices (512 x 1024 to 28672 x 4096) with 5 to 1024 rows, within 4 % for half of
// them and 12 % for nine in ten; its choices cost 1 % over the best tile and split of each. (The estimate before it, in cycles, took splits for cheap and turns for
// all alike: 21 % over the best, 38.8 us for 13.6 at 256 rows x 7168 x 1024.)
struct QsCost { float fill, integers4, integers8, planes4, planes8, mlx4, mlx8, three4, three8; };
constexpr int QS_TILES[6] = {16, 32, 64, 128, 192, 256};
constexpr QsCost QS_COST[6] = {{0.5f, 0.342f, 0.448f, 0.472f, 0.624f, 0.516f, 0.522f, 0.603f, 0.574f}, {0.5f, 0.361f, 0.479f, 0.483f, 0.636f, 0.543f, 0.535f, 0.617f, 0.587f},
                               {0.9f, 0.376f, 0.487f, 0.491f, 0.646f, 0.539f, 0.561f, 0.659f, 0.629f}, {2.0f, 0.0f, 0.0f, 0.395f, 0.558f, 0.502f, 0.520f, 0.0f, 0.0f},
                               {1.7f, 0.0f, 0.0f, 0.494f, 0.591f, 0.511f, 0.536f, 0.0f, 0.0f}, {3.2f, 0.0f, 0.0f, 0.558f, 0.588f, 0.584f, 0.569f, 0.0f, 0.0f}};

// Rows per tile and CTAs per tile: the shortest estimated time over the chip. A wider tile turns its codes once for more rows; a narrower one or a
// split k fills the chip where tiles are few. (Clusters leave SMs idle whose neighbours are taken: of 148, 144 work in pairs, 132 in fours and 112 in eights.)
QsPlan qs_plan(uint32_t m, uint32_t n, uint32_t nkb, uint32_t bits, bool mlx, bool three, bool integers, bool halves, uint32_t sms) {
    QsPlan best;
    const uint32_t n_tiles = (n + 127u) / 128u;
    for (int i = 0; i < 6; ++i) {
        const int nt = QS_TILES[i];
        const QsCost& c = QS_COST[i];
        if (nt > 16 && m <= (uint32_t)nt / 2) break;
        if (nt < 128 && m > 2u * nt) continue;                              // (up to 64 rows sum in another order: the widest of them up to twice its rows)
        if (nt >= 128 && three) break;                                       // (three planes: fewer than 64 rows)
        const float block = integers && nt < 128 ? (bits == 4 ? c.integers4 : c.integers8) : three ? (bits == 4 ? c.three4 : c.three8) : mlx ? (bits == 4 ? c.mlx4 : c.mlx8) : bits == 4 ? c.planes4 : c.planes8;
        const float two_factors = mlx && halves ? (nt == 256 ? 0.015f : 0.055f) : 0.0f;      // groups of 32
        const uint32_t tiles = n_tiles * ((m + nt - 1) / nt);
        for (uint32_t splits = 1; splits <= 8; splits *= 2) {
            const uint32_t per = ((nkb + splits - 1) / splits + 3u) & ~3u;           // whole code tiles per rank
            const uint32_t room = splits == 1 ? sms : splits == 2 ? sms * 36 / 37 : splits == 4 ? sms * 33 / 37 : sms * 28 / 37;
            if (splits > 1 && (per * (splits - 1) >= nkb || tiles * splits > room)) break;
            const uint32_t turns = (tiles * splits + room - 1) / room;
            const float exchange = splits == 1 ? 0.0f : (splits == 2 ? 2.3f : splits == 4 ? 1.7f : 4.5f) + 0.01f * nt;
            const float cost = 5.2f + turns * (c.fill + (block + two_factors) * std::min(per, nkb)) + exchange;
            if (cost < best.cost) best = {nt, splits, cost};
        }
    }
    return best;
}

int g_tile_rows = 0, g_tile_splits = 0, g_wide = 0;      // uzu_debug_set_qmm_tile; 0: the plan's own

template <int BITS, int NT, int PL>
void qs_launch(uzu_command_buffer* cmd, const CUtensorMap& w, const CUtensorMap& x, const QsParams& p, uint32_t grid) {
    static std::atomic<uint64_t> smem_opt_in{0};
    opt_in_dynamic_smem(cmd, qmm_scaled_kernel<BITS, NT, PL>, (int)QsShape<NT, PL>::SMEM, smem_opt_in);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(QsShape<NT, PL>::THREADS);
    cfg.dynamicSmemBytes = QsShape<NT, PL>::SMEM;
    cfg.stream = cmd->ctx->stream;
    cudaLaunchAttribute attr[2];
    if (cmd->dependent()) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (p.splits > 1) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
        attr[cfg.numAttrs].val.clusterDim.x = p.splits;
        attr[cfg.numAttrs].val.clusterDim.y = 1;
        attr[cfg.numAttrs++].val.clusterDim.z = 1;
    }
    cfg.attrs = attr;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, qmm_scaled_kernel<BITS, NT, PL>, w, x, p);
    if (e != cudaSuccess) cmd->record_error(UZU_ERROR_CUDA, std::string("matmul qmm_scaled_kernel: ") + cudaGetErrorString(e));
    cmd->launches++;
}

}  // namespace

void encode_qmm_scaled(uzu_command_buffer* cmd, const uzu_matmul_args& a) {
    QsParams p{};
    const uint32_t bits = a.b_mode == UZU_QMODE_U4 ? 4 : 8;
    p.scales = (const __nv_bfloat16*)a.b_scales;
    p.method = a.b_prologue == UZU_B_SCALE_BIAS_DEQUANT ? UZU_QMETHOD_SCALE_BIAS
               : a.b_prologue == UZU_B_SCALE_ZERO_POINT_DEQUANT ? UZU_QMETHOD_SCALE_ZERO_POINT : UZU_QMETHOD_SCALE_SYMMETRIC;
    p.zero_points = (const uint8_t*)a.b_zero_points;
    p.biases = p.method == UZU_QMETHOD_SCALE_BIAS ? (const __nv_bfloat16*)a.b_biases : nullptr;
    p.bias = ((a.d_transform & UZU_D_BIAS) && a.bias) ? (const __nv_bfloat16*)a.bias : nullptr;
    p.n = a.n; p.k = a.k;
    p.groups = a.k / a.b_group_size;
    p.zp_stride = bits == 4 ? (p.groups + 1) / 2 : p.groups;
    while ((1u << p.gshift) < a.b_group_size) ++p.gshift;
    p.xor_mask = a.b_signed_codes ? (bits == 4 ? 0x88888888u : 0x80808080u) : 0u;
    p.nkb = a.k / 64u;
    p.d_is_f32 = a.output_dt == UZU_DT_F32;
    p.accumulate = (a.d_transform & UZU_D_ACCUMULATE) != 0;
    p.has_soft_cap = (a.d_transform & UZU_D_SOFT_CAP) != 0;
    p.ab_scale = (a.d_transform & UZU_D_SCALE) ? a.ab_scale : 1.0f;
    p.soft_cap = a.soft_cap;
    p.plain = !p.d_is_f32 && !p.accumulate && !p.has_soft_cap && !p.bias && p.ab_scale == 1.0f;
    p.error = cmd->ctx->wait_errors.device_word;
    p.m = a.m;
    p.d = (void*)a.d;
    uzu_context* ctx = cmd->ctx;
    // MLX weights of passes that the kernels before this one summed with the codes as integers keep all their bits; longer ones had two planes always
    const bool three = p.biases && p.m < 64, integers = !p.biases && a.b_group_size >= 64;      // (integers: tiles of up to 64 rows)
    p.chain_k = std::min(a.b_group_size, 128u);
    QsPlan plan = qs_plan(p.m, a.n, p.nkb, bits, p.biases != nullptr, three, integers, a.b_group_size == 32, (uint32_t)ctx->sm_count);
    const bool wide_can = integers && bits == 4 && p.chain_k == 128u && !p.has_soft_cap;
    if (g_wide && !wide_can) {
        cmd->record_error(UZU_ERROR_UNSUPPORTED, "matmul: the kernel asked for (qmm_wide.cu) does not take this call");
        return;
    }
    // one plane of integers for wide tiles: 4-bit codes in groups of 128 and more (qmm_wide.cu, with the times of both kernels)
    if (wide_can && (g_wide || (p.m > 64 && !g_tile_rows && !g_tile_splits))) {
        const QwPlan wide = qw_plan(p.m, a.n, p.nkb, (uint32_t)ctx->sm_count);
        if (g_wide || wide.cost < plan.cost) return encode_qmm_wide(cmd, a, p, g_wide ? (uint32_t)g_wide : wide.width);
    }
    if (g_tile_rows) plan.nt = g_tile_rows;
    if (g_tile_splits) {
        plan.splits = (uint32_t)g_tile_splits;
        while (plan.splits > 1 && (((p.nkb + plan.splits - 1) / plan.splits + 3u) & ~3u) * (plan.splits - 1) >= p.nkb) plan.splits /= 2;      // every rank has some
    }
    p.splits = plan.splits;
    p.split_kb = p.splits == 1 ? p.nkb : ((p.nkb + p.splits - 1) / p.splits + 3u) & ~3u;
    p.m_tiles = (p.m + plan.nt - 1) / plan.nt;
    p.items = p.m_tiles * ((a.n + 127u) / 128u);
    CUtensorMap mw, mx;
    if (!tensor_map(&mw, CU_TENSOR_MAP_DATA_TYPE_UINT8, a.b, (uint64_t)a.k * bits / 8, a.n, (uint64_t)a.k * bits / 8, 128, 128) ||
        !tensor_map(&mx, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, a.a, a.k, p.m, (uint64_t)a.k * 2, 64, (uint32_t)plan.nt)) {
        cmd->record_error(UZU_ERROR_CUDA, "matmul: cuTensorMapEncodeTiled failed");
        return;
    }
    const uint32_t grid = p.splits > 1 ? p.items * p.splits : std::min(p.items, (uint32_t)ctx->sm_count);
    auto go = [&](auto bits_c) {
        constexpr int BITS = decltype(bits_c)::value;
        switch (plan.nt) {
            case 16: integers ? qs_launch<BITS, 16, 1>(cmd, mw, mx, p, grid) : three ? qs_launch<BITS, 16, 3>(cmd, mw, mx, p, grid) : qs_launch<BITS, 16, 2>(cmd, mw, mx, p, grid); break;
            case 32: integers ? qs_launch<BITS, 32, 1>(cmd, mw, mx, p, grid) : three ? qs_launch<BITS, 32, 3>(cmd, mw, mx, p, grid) : qs_launch<BITS, 32, 2>(cmd, mw, mx, p, grid); break;
            case 64: integers ? qs_launch<BITS, 64, 1>(cmd, mw, mx, p, grid) : three ? qs_launch<BITS, 64, 3>(cmd, mw, mx, p, grid) : qs_launch<BITS, 64, 2>(cmd, mw, mx, p, grid); break;
            case 128: qs_launch<BITS, 128, 2>(cmd, mw, mx, p, grid); break;
            case 192: qs_launch<BITS, 192, 2>(cmd, mw, mx, p, grid); break;
            default: qs_launch<BITS, 256, 2>(cmd, mw, mx, p, grid); break;
        }
    };
    if (bits == 4) go(std::integral_constant<int, 4>{});
    else go(std::integral_constant<int, 8>{});
}

}  // namespace uzu

// mt: 1, 2: tiles of 128, 256 rows; 0: the plan's own. (The others described operands of an earlier kernel.)
extern "C" void uzu_debug_set_umma(int, uint32_t, uint32_t, uint32_t, uint32_t, int mt) { uzu::g_tile_rows = mt == 1 ? 128 : mt == 2 ? 256 : 0; }

// splits -1: the kernel of qmm_wide.cu, where it can run, with tiles of that many rows, a multiple of 16 up to 256
extern "C" int uzu_debug_set_qmm_tile(int rows, int splits) {
    uzu::g_wide = 0;
    if (splits == -1) {
        if (rows < 16 || rows > 256 || rows % 16) return 0;
        uzu::g_wide = rows;
        uzu::g_tile_rows = uzu::g_tile_splits = 0;
        return 1;
    }
    const bool known = rows == 0 || rows == 16 || rows == 32 || rows == 64 || rows == 128 || rows == 192 || rows == 256;
    if (!known || (splits != 0 && splits != 1 && splits != 2 && splits != 4 && splits != 8)) return 0;
    uzu::g_tile_rows = rows;
    uzu::g_tile_splits = splits;
    return 1;
}
