// Quantised MatmulKernel for more than 64 activation rows, 4-bit ZeroPoint / Symmetric weights in groups of 128 and more: D[m, n] = epilogue(A[m, k] * dequant(B[n, k])^T).
// Semantic spec: backends/cpu/kernel/matmul/kernel.rs:164-295 (caller encodable_block/linear/matmul.rs:122-148).
//
// The kernel before it (qmm_scaled.cu, still the one for all else) multiplies two bf16 planes of a weight, which are its scale times its code: half of the tensor pipe's
// rate is the most that two planes can give, and wide tiles run at nine tenths of that. Here the operand is ONE plane, the integers code - zero point, exact in bf16. A
// chain of 128 k (a group or a part of one) is summed unscaled in tensor memory and brought to f32 sums in registers by one rounded multiply-add with the group's
// scale.
//
// CTA = 128 output features x up to 256 rows (any multiple of 16), K in blocks of 64. A tile's rows are two halves of up to 128, each with a sum of its own, in one of
// three buffers of 128 columns: one is summed into, one is read, one is between.
//   sums      eight warps: a thread owns a feature, half of each half's columns, 128 sums in 208 registers.
//   dequant   four warps: a thread owns a feature row, turns its 64 codes and stores them to tensor memory (four blocks of 32 columns, operand A).
//   one warp each: TMA of the codes (128 rows x 128 bytes), of the activations (64 k a stage), and the products of each half (tcgen05.mma, 4 a block).
// Registers: 512 threads x 128 = 65536 = 256 x 208 + 128 x 64 + 128 x 32.
//
// What bounds it: per block of 256 rows the products take 512 cycles, the multiply-adds 256 a chain of each scheduler's issue slots, the codes about 200; a wait that
// need not wait costs a warp 150 cycles, so each role asks about its next barriers before its work (28672 x 4096, 1024 rows, groups of 128: 233 -> 215 us; one product
// warp for both halves and 64 sums read at a time in two goes: 345 in groups of 64, now 280). With chains of 64 the multiply-adds are twice as many and the two planes
// are as fast (280 / 275), and so are they with bytes for codes (groups of 128: 275 / 278), whose dequant is twice as long. 4-bit groups of 128, two planes / this:
// 28672 x 4096: 1024 rows 275 / 215 us, 509 rows 160 / 125, 256 rows 84 / 67; 4096 x 14336, 1024 rows 133 / 110.
// Errors against 64 bits are smaller, since tensor memory adds up 128 k instead of all: 1.0e-7 of the outputs' root mean square at k = 4096 (two planes 7.5e-6), 1.9e-7
// at 14336 (2.8e-5).
// Every barrier wait is bounded (about a second): a wait that runs out is reported (wait_errors.h: the call then fails on the host), copies and products in flight are
// waited for, and the CTA ends its work.
#include <algorithm>
#include <cstdlib>
#include <type_traits>

#include "qmm_scaled.cuh"

namespace uzu {

namespace {

constexpr uint32_t QW_WIDTH = 256, QW_D = 3, QW_A = 4, QW_ACTS = 4, QW_CODES = 5, QW_A_COL = 384;
constexpr uint32_t QW_ACT = QW_WIDTH * 128, QW_THREADS = 512;
constexpr size_t QW_SMEM = (size_t)QW_ACTS * QW_ACT + (size_t)QW_CODES * QS_CODE_TILE + 1024;

struct QwParams {
    QsParams s;
    uint32_t width, first;      // rows of a tile, of its first half
};

// whether a phase has completed, without a wait
__device__ __forceinline__ uint32_t qw_test(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{ .reg .pred p; mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok;
}
// as qs_wait, without a call: the registers are split between the warps
__device__ __forceinline__ bool qw_wait_long(uint32_t bar, uint32_t parity, volatile uint32_t* gave_up, unsigned int* error, uint32_t code) {
    uint64_t t0 = 0, t1 = 0;
    for (uint32_t tries = 1;; ++tries) {
        if (__all_sync(0xffffffffu, qs_try(bar, parity))) return true;
        if (tries & 255u) continue;
        if (__any_sync(0xffffffffu, *gave_up)) return false;
        if (!t0) pdl_wait();                                                 // the time of a kernel that this one depends on does not count
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
        t1 = __shfl_sync(0xffffffffu, t1, 0);
        if (!t0) t0 = t1;
        if (t1 - t0 > 1000000000ull) {
            *gave_up = 1;
            report_wait_error(error, code);
            return false;
        }
    }
}
// ready: what a test of the same phase said some instructions before (a wait that need not wait costs a warp 150 cycles, a test beside other work a few)
__device__ __forceinline__ bool qw_wait(uint32_t ready, uint32_t bar, uint32_t parity, volatile uint32_t* gave_up, unsigned int* error, uint32_t code) {
    return __all_sync(0xffffffffu, ready) || qw_wait_long(bar, parity, gave_up, error, code);
}
__device__ __forceinline__ void qw_ld32(uint32_t taddr, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
          "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]),
          "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr)
        : "memory");
}
// nothing that uses v is done before this point (the wait for the loads)
__device__ __forceinline__ void qw_from_here(uint32_t (&v)[32]) {
    asm volatile(""
                 : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]), "+r"(v[8]), "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15]),
                   "+r"(v[16]), "+r"(v[17]), "+r"(v[18]), "+r"(v[19]), "+r"(v[20]), "+r"(v[21]), "+r"(v[22]), "+r"(v[23]), "+r"(v[24]), "+r"(v[25]), "+r"(v[26]), "+r"(v[27]), "+r"(v[28]), "+r"(v[29]), "+r"(v[30]), "+r"(v[31])
                 :
                 : "memory");
}
__device__ __forceinline__ float2 qw_fma2(float2 a, float2 b, float2 c) {
    float2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(reinterpret_cast<uint64_t&>(d)) : "l"(reinterpret_cast<uint64_t&>(a)), "l"(reinterpret_cast<uint64_t&>(b)), "l"(reinterpret_cast<uint64_t&>(c)));
    return d;
}
__device__ __forceinline__ void qw_lds4(uint32_t addr, uint32_t* q) {
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(q[0]), "=r"(q[1]), "=r"(q[2]), "=r"(q[3]) : "r"(addr) : "memory");
}

}  // namespace

__global__ void __launch_bounds__(QW_THREADS, 1) qmm_wide_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const QwParams w) {
    constexpr uint32_t kpt = 4;                                              // k blocks per code tile
    const QsParams& p = w.s;
    extern __shared__ uint8_t qw_raw[];
    __shared__ __align__(8) uint64_t bars[2 * QW_CODES + 2 * QW_ACTS + 2 * QW_A + 2 * QW_D + 1];
    __shared__ uint32_t tmem_slot;
    __shared__ volatile uint32_t gave_up;
    const uint32_t tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const uint32_t base = (qs_smem(qw_raw) + 1023u) & ~1023u;                // swizzle atoms sit on 1024-byte boundaries
    const uint32_t act0 = base, code0 = base + QW_ACTS * QW_ACT, bar0 = qs_smem(bars);
    auto code_full = [&](uint32_t i) { return bar0 + 8u * i; };
    auto code_empty = [&](uint32_t i) { return bar0 + 8u * (QW_CODES + i); };
    auto act_full = [&](uint32_t i) { return bar0 + 8u * (2 * QW_CODES + i); };
    auto act_empty = [&](uint32_t i) { return bar0 + 8u * (2 * QW_CODES + QW_ACTS + i); };
    auto a_full = [&](uint32_t i) { return bar0 + 8u * (2 * QW_CODES + 2 * QW_ACTS + i); };
    auto a_empty = [&](uint32_t i) { return bar0 + 8u * (2 * QW_CODES + 2 * QW_ACTS + QW_A + i); };
    auto d_full = [&](uint32_t i) { return bar0 + 8u * (2 * QW_CODES + 2 * QW_ACTS + 2 * QW_A + i); };
    auto d_empty = [&](uint32_t i) { return bar0 + 8u * (2 * QW_CODES + 2 * QW_ACTS + 2 * QW_A + QW_D + i); };
    const uint32_t last_products = bar0 + 8u * (2 * QW_CODES + 2 * QW_ACTS + 2 * QW_A + 2 * QW_D);

    const uint32_t nk = p.nkb, halves = w.width > w.first ? 2u : 1u, second = w.width - w.first, chains = nk / 2;
    if (warp == 0) {
        if (lane == 0) {
            for (uint32_t i = 0; i < QW_CODES; ++i) { qs_init(code_full(i), 1); qs_init(code_empty(i), 4); }
            for (uint32_t i = 0; i < QW_ACTS; ++i) { qs_init(act_full(i), 1); qs_init(act_empty(i), halves); }
            for (uint32_t i = 0; i < QW_A; ++i) { qs_init(a_full(i), 4); qs_init(a_empty(i), halves); }
            for (uint32_t i = 0; i < QW_D; ++i) { qs_init(d_full(i), 1); qs_init(d_empty(i), 8); }
            qs_init(last_products, halves);
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
    // neighbouring items share their weights: the row tiles of a feature tile are in flight together
    auto item_n = [&](uint32_t item) { return item / p.m_tiles * 128u; };
    auto item_m = [&](uint32_t item) { return item % p.m_tiles * w.width; };

    if (warp < 8) {
        // ================================ sums ================================
        asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");
        const uint32_t quarter = ((warp & 3u) * 32u) << 16, side = warp >> 2;
        const uint32_t mine0 = w.first / 2, mine1 = second / 2, at0 = side * mine0, at1 = side * mine1;      // this warp's columns of a half and where they begin
        uint32_t buf = 0, ph = 0, ready = 0;
        pdl_wait();                                                      // D may be read (accumulate) and is written below
        for (uint32_t item = blockIdx.x; item < p.items; item += gridDim.x) {
            const uint32_t row = item_n(item) + (warp & 3u) * 32u + lane, t0 = item_m(item);
            float2 acc[2][32];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
#pragma unroll
                for (int c = 0; c < 32; ++c) acc[h][c] = make_float2(0.0f, 0.0f);
            }
            const uint16_t* srow = reinterpret_cast<const uint16_t*>(p.scales) + (size_t)min(row, p.n - 1u) * p.groups;
            auto scale_of = [&](uint32_t i) { return (uint32_t)__ldg(srow + ((min(i, chains - 1u) * 128u) >> p.gshift)); };
            uint32_t ahead[2] = {scale_of(0), scale_of(1)};              // scales of the next two chains
            bool ok = true;
            for (uint32_t i = 0; i < chains; ++i) {
                const float scale = __uint_as_float(ahead[0] << 16);
                const float2 scale2 = make_float2(scale, scale);
                ahead[0] = ahead[1];
                ahead[1] = scale_of(i + 2);
#pragma unroll
                for (uint32_t h = 0; h < 2; ++h) {
                    if (h >= halves) continue;
                    ok = qw_wait(ready, d_full(buf), ph, &gave_up, p.error, 0x601u);
                    if (!ok) break;
                    qs_fence_after();
                    const uint32_t from = tmem + quarter + buf * 128u + (h ? at1 : at0), mine = h ? mine1 : mine0;
                    // (columns behind the last one, in the buffer all the same, are summed for nobody)
                    uint32_t v[2][32];
                    qw_ld32(from, v[0]);
                    if (mine > 32) qw_ld32(from + 32, v[1]);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    qw_from_here(v[0]);
                    qw_from_here(v[1]);
                    qs_fence_before();
                    __syncwarp();
                    if (lane == 0) qs_arrive(d_empty(buf));
                    if (++buf == QW_D) { buf = 0; ph ^= 1u; }
                    ready = qw_test(d_full(buf), ph);
#pragma unroll
                    for (uint32_t j = 0; j < 16; ++j) acc[h][j] = qw_fma2(make_float2(__uint_as_float(v[0][2 * j]), __uint_as_float(v[0][2 * j + 1])), scale2, acc[h][j]);
                    if (mine > 32) {
#pragma unroll
                        for (uint32_t j = 0; j < 16; ++j) acc[h][16 + j] = qw_fma2(make_float2(__uint_as_float(v[1][2 * j]), __uint_as_float(v[1][2 * j + 1])), scale2, acc[h][16 + j]);
                    }
                }
                if (!ok) break;
            }
            if (!ok) break;
#pragma unroll
            for (uint32_t h = 0; h < 2; ++h) {
                if (h >= halves) continue;
                const uint32_t token0 = t0 + (h ? w.first + at1 : at0), mine = h ? mine1 : mine0;
                const uint32_t columns = row < p.n && token0 < p.m ? min(mine, p.m - token0) : 0u;
                const size_t at = (size_t)token0 * p.n + row;
                if (p.plain) {                                           // D is the rounded sum: a store per column (64 neighbouring bytes a warp)
                    __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(p.d) + at;
#pragma unroll
                    for (uint32_t c = 0; c < 64; ++c, out += p.n)
                        if (c < columns) *out = f2bf((c & 1u ? acc[h][c / 2].y : acc[h][c / 2].x) * qs_unit<4>);
                } else {
                    const float bias = p.bias && row < p.n ? bf2f(p.bias[row]) : 0.0f;
                    float* out32 = reinterpret_cast<float*>(p.d) + at;
                    __nv_bfloat16* out16 = reinterpret_cast<__nv_bfloat16*>(p.d) + at;
#pragma unroll
                    for (uint32_t c = 0; c < 64; ++c, out32 += p.n, out16 += p.n) {
                        if (c >= columns) continue;
                        float val = __fmul_rn(p.ab_scale, (c & 1u ? acc[h][c / 2].y : acc[h][c / 2].x) * qs_unit<4>);      // separate roundings, like the reference
                        if (p.accumulate) val = __fadd_rn(val, p.d_is_f32 ? *out32 : bf2f(*out16));
                        if (p.bias) val = __fadd_rn(val, bias);
                        if (p.d_is_f32) *out32 = val;
                        else *out16 = f2bf(val);
                    }
                }
            }
        }
    } else if (warp < 12) {
        // ================================ codes -> integers in tensor memory ================================
        asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
        const uint32_t lw = warp & 3u, r = lw * 32u + lane;
        const bool has_zp = p.method == UZU_QMETHOD_SCALE_ZERO_POINT;
        // the bits above a code's; a signed code's top bit is turned over
        const uint32_t above = qs_base<4> * 0x00010001u ^ (p.xor_mask & 0x00080008u);
        uint32_t stage = 0, a_ph = 1, slot = 0, c_ph = 0;
        bool ok = true;
        for (uint32_t item = blockIdx.x; item < p.items && ok; item += gridDim.x) {
            const uint8_t* zrow = p.zero_points + (size_t)min(item_n(item) + r, p.n - 1u) * p.zp_stride;
            auto zero_of = [&](uint32_t kb) -> uint32_t {
                const uint32_t g = min(kb * 64u >> p.gshift, p.groups - 1u);
                return has_zp ? (uint32_t)(zrow[g >> 1] >> (4u * (g & 1u))) & 15u : 8u;
            };
            uint32_t q[8], z[2] = {zero_of(0), zero_of(1)};
            // a block's codes; the tile's place is free with its last block
            auto fetch = [&](uint32_t kb) {
                const uint32_t j = kb % kpt;
                if (j == 0) ok = qw_wait(qw_test(code_full(slot), c_ph), code_full(slot), c_ph, &gave_up, p.error, 0x602u);
                if (!ok) return;
                const uint32_t line = code0 + slot * QS_CODE_TILE + r * 128u;
#pragma unroll
                for (uint32_t i = 0; i < 2; ++i) qw_lds4(line + (((j * 2 + i) ^ (r & 7u)) << 4), q + 4 * i);
                if (j == kpt - 1 || kb + 1 == nk) {
                    __syncwarp();
                    if (lane == 0) qs_arrive(code_empty(slot));
                    if (++slot == QW_CODES) { slot = 0; c_ph ^= 1u; }
                }
            };
            fetch(0);
            for (uint32_t kb = 0; kb < nk && ok; ++kb) {
                const uint32_t ready = qw_test(a_empty(stage), a_ph);
                uint32_t v[32];
                const uint32_t zero = z[0];
                z[0] = z[1];
                z[1] = zero_of(kb + 2);
                const uint32_t z2 = (qs_base<4> | zero) * 0x00010001u;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    uint32_t d[4];
#pragma unroll
                    for (int n = 0; n < 4; ++n) d[n] = qs_u(__hsub2(qs_b2(((q[i] >> (4 * n)) & 0x000F000Fu) ^ above), qs_b2(z2)));
                    v[4 * i] = __byte_perm(d[0], d[1], 0x5410); v[4 * i + 1] = __byte_perm(d[2], d[3], 0x5410);
                    v[4 * i + 2] = __byte_perm(d[0], d[1], 0x7632); v[4 * i + 3] = __byte_perm(d[2], d[3], 0x7632);
                }
                if (kb + 1 < nk) fetch(kb + 1);
                if (ok) ok = qw_wait(ready, a_empty(stage), a_ph, &gave_up, p.error, 0x603u);
                if (!ok) break;
                qs_fence_after();
                const uint32_t t_col = tmem + ((lw * 32u) << 16) + QW_A_COL + stage * 32u;
#pragma unroll
                for (uint32_t h = 0; h < 2; ++h) {
                    uint32_t part[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) part[i] = v[16 * h + i];
                    qs_tmem_st16(t_col + h * 16u, part);
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                qs_fence_before();
                __syncwarp();
                if (lane == 0) qs_arrive(a_full(stage));
                if (++stage == QW_A) { stage = 0; a_ph ^= 1u; }
            }
        }
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 32;");
        const uint32_t role = warp - 12;
        bool ok = true;
        if (role == 0) {
            // ================================ codes by TMA (they depend on no kernel) ================================
            uint32_t slot = 0, ph = 1, asked = 0;
            const uint32_t tiles = (nk + kpt - 1) / kpt;
            for (uint32_t item = blockIdx.x; item < p.items && ok; item += gridDim.x) {
                const uint32_t y = item_n(item);
                for (uint32_t tile = 0; tile < tiles; ++tile) {
                    ok = qw_wait(0, code_empty(slot), ph, &gave_up, p.error, 0x604u);
                    if (!ok) break;
                    if (qs_elect()) {
                        qs_expect(code_full(slot), QS_CODE_TILE);
                        qs_tma_2d(code0 + slot * QS_CODE_TILE, &map_w, tile * 128u, y, code_full(slot));
                    }
                    __syncwarp();
                    ++asked;
                    if (++slot == QW_CODES) { slot = 0; ph ^= 1u; }
                }
            }
            if (!ok)
                for (uint32_t n = asked > QW_CODES ? asked - QW_CODES : 0; n < asked; ++n) qs_settle(code_full(n % QW_CODES), n / QW_CODES & 1u);
        } else if (role == 1) {
            // ================================ activations by TMA, 64 k a stage ================================
            uint32_t slot = 0, ph = 1, asked = 0;
            pdl_wait();
            for (uint32_t item = blockIdx.x; item < p.items && ok; item += gridDim.x) {
                const uint32_t y = item_m(item);
                for (uint32_t i = 0; i < nk; ++i) {
                    ok = qw_wait(0, act_empty(slot), ph, &gave_up, p.error, 0x605u);
                    if (!ok) break;
                    if (qs_elect()) {
                        qs_expect(act_full(slot), w.width * 128u);
                        qs_tma_2d(act0 + slot * QW_ACT, &map_x, i * 64u, y, act_full(slot));
                    }
                    __syncwarp();
                    ++asked;
                    if (++slot == QW_ACTS) { slot = 0; ph ^= 1u; }
                }
            }
            if (!ok)
                for (uint32_t n = asked > QW_ACTS ? asked - QW_ACTS : 0; n < asked; ++n) qs_settle(act_full(n % QW_ACTS), n / QW_ACTS & 1u);
        } else if (role - 2 < halves) {
            // ================================ products: a warp for each half ================================
            // shared-memory descriptor: K-major SWIZZLE_128B, 1024 bytes between 8-row groups, +32 bytes per 16 k
            constexpr uint64_t desc_hi = (uint64_t)((1024u >> 4) | (1u << 14) | (2u << 29)) << 32;
            const uint32_t half = role - 2, shape = (1u << 4) | (1u << 7) | (1u << 10) | ((half ? second : w.first) >> 3) << 17 | (128u >> 4) << 24;
            const uint32_t desc_lo = ((act0 + (half ? w.first * 128u : 0u)) >> 4) | (1u << 16);
            uint32_t bs = 0, bs_ph = 0, as = 0, as_ph = 0, buf = half, d_ph = 1, left = 2, ready[3] = {};      // left: blocks of the chain
            for (uint32_t item = blockIdx.x; item < p.items && ok; item += gridDim.x) {
                for (uint32_t i = 0; i < nk; ++i) {
                    const bool begins = left == 2, ends = left == 1;
                    if (begins) ok = qw_wait(ready[2], d_empty(buf), d_ph, &gave_up, p.error, 0x608u);
                    if (ok) ok = qw_wait(ready[0], act_full(bs), bs_ph, &gave_up, p.error, 0x606u);
                    if (ok) ok = qw_wait(ready[1], a_full(as), as_ph, &gave_up, p.error, 0x607u);
                    if (!ok) break;
                    qs_fence_after();
                    if (qs_elect()) {
                        const uint32_t d = tmem + buf * 128u, a_col = tmem + QW_A_COL + as * 32u, lo = desc_lo + (bs * QW_ACT >> 4);
#pragma unroll
                        for (uint32_t kk = 0; kk < 4; ++kk) qs_mma(d, a_col + kk * 8u, desc_hi | (lo + kk * 2u), shape, !begins || kk != 0 ? 1u : 0u);
                        if (ends) qs_commit(d_full(buf));
                        qs_commit(a_empty(as));
                        qs_commit(act_empty(bs));
                    }
                    __syncwarp();
                    if (++as == QW_A) { as = 0; as_ph ^= 1u; }
                    if (++bs == QW_ACTS) { bs = 0; bs_ph ^= 1u; }
                    if (ends) {
                        buf += halves;
                        if (buf >= QW_D) { buf -= QW_D; d_ph ^= 1u; }
                        left = 2;
                    } else --left;
                    ready[0] = qw_test(act_full(bs), bs_ph);
                    ready[1] = qw_test(a_full(as), as_ph);
                    ready[2] = qw_test(d_empty(buf), d_ph);
                }
            }
            if (qs_elect()) qs_commit(last_products);
            __syncwarp();
            qs_settle(last_products, 0);                                 // none in flight when tensor memory is given back
        }
        __syncwarp();
    }
    qs_fence_before();
    __syncthreads();
    if (warp == 0) {
        qs_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

// ---- host side -------------------------------------------------------------------------------------------------------------------------
// The width whose tiles take the chip the shortest time, and that time in us: 5 for a launch, filling the pipeline and storing a tile, 64 k as often as there are.
// Fitted to the times of 13 matrices with 66 to 1024 rows (half of them within 3 %, nine in ten within 7 %).
QwPlan qw_plan(uint32_t m, uint32_t n, uint32_t nkb, uint32_t sms) {
    QwPlan best;
    const uint32_t n_tiles = (n + 127u) / 128u;
    for (uint32_t width : {96u, 128u, 160u, 176u, 208u, 256u}) {
        const uint32_t tiles = n_tiles * ((m + width - 1) / width), turns = (tiles + sms - 1) / sms;
        const float cost = 5.2f + turns * (width <= 128 ? 0.9f + 0.391f * nkb : 3.6f + 0.424f * nkb);
        if (cost < best.cost) best = {width, cost};
    }
    return best;
}

static void qw_launch(uzu_command_buffer* cmd, const CUtensorMap& mw, const CUtensorMap& mx, const QwParams& w, uint32_t grid) {
    static std::atomic<uint64_t> smem_opt_in{0};
    opt_in_dynamic_smem(cmd, qmm_wide_kernel, (int)QW_SMEM, smem_opt_in);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(QW_THREADS);
    cfg.dynamicSmemBytes = QW_SMEM;
    cfg.stream = cmd->ctx->stream;
    cudaLaunchAttribute attr[1];
    if (cmd->dependent()) {
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    }
    const cudaError_t e = cudaLaunchKernelEx(&cfg, qmm_wide_kernel, mw, mx, w);
    if (e != cudaSuccess) cmd->record_error(UZU_ERROR_CUDA, std::string("matmul qmm_wide_kernel: ") + cudaGetErrorString(e));
    cmd->launches++;
}

void encode_qmm_wide(uzu_command_buffer* cmd, const uzu_matmul_args& a, QsParams p, uint32_t width) {
    QwParams w{};
    w.width = width;
    w.first = width <= 128 ? width : (width / 2 + 15u) / 16u * 16u;
    p.m_tiles = (p.m + width - 1) / width;
    p.items = p.m_tiles * ((a.n + 127u) / 128u);
    w.s = p;
    CUtensorMap mw, mx;
    if (!tensor_map(&mw, CU_TENSOR_MAP_DATA_TYPE_UINT8, a.b, (uint64_t)a.k / 2, a.n, (uint64_t)a.k / 2, 128, 128) ||
        !tensor_map(&mx, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, a.a, a.k, p.m, (uint64_t)a.k * 2, 64, width)) {
        cmd->record_error(UZU_ERROR_CUDA, "matmul: cuTensorMapEncodeTiled failed");
        return;
    }
    const uint32_t grid = std::min(p.items, (uint32_t)cmd->ctx->sm_count);
    qw_launch(cmd, mw, mx, w, grid);
}

}  // namespace uzu
