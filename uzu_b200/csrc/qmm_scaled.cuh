// What the two kernels for quantised products on tcgen05 share (qmm_scaled.cu, qmm_wide.cu): instructions, bounded waits, codes as bf16, tensor maps.
#pragma once
#include <cuda.h>

#include "common.cuh"

namespace uzu {

struct QsParams {
    const __nv_bfloat16* scales;
    const uint8_t* zero_points;      // ScaleZeroPoint
    const __nv_bfloat16* biases;     // ScaleBias
    void* d;
    const __nv_bfloat16* bias;
    unsigned int* error;
    uint32_t m, n, k, groups, zp_stride, gshift, xor_mask, method;
    uint32_t nkb, split_kb, splits, items, m_tiles;
    uint32_t chain_k;                // PL = 1: k of a chain, 64 or 128: a group or a part of one
    uint32_t d_is_f32, accumulate, has_soft_cap, plain;
    float ab_scale, soft_cap;
};

namespace {

constexpr uint32_t QS_CODE_TILE = 128 * 128;

__device__ __forceinline__ uint32_t qs_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void qs_init(uint32_t bar, uint32_t count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory"); }
__device__ __forceinline__ void qs_arrive(uint32_t bar) { asm volatile("{ .reg .b64 st; mbarrier.arrive.shared::cta.b64 st, [%0]; }" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void qs_expect(uint32_t bar, uint32_t bytes) {
    asm volatile("{ .reg .b64 st; mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1; }" ::"r"(bar), "r"(bytes) : "memory");
}
// (the thread sleeps in the barrier for up to 20 us a try: spinning warps would take the issue slots of the working ones)
__device__ __forceinline__ bool qs_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3; selp.u32 %0, 1, 0, p; }" : "=r"(ok) : "r"(bar), "r"(parity), "r"(20000u) : "memory");
    return ok != 0;
}
// false: the phase did not complete within about a second of the preceding kernel's end, or another role of the CTA has given up
__device__ __noinline__ bool qs_wait_long(uint32_t bar, uint32_t parity, volatile uint32_t* gave_up, unsigned int* error, uint32_t code) {
    uint64_t t0 = 0;
    for (uint32_t tries = 0; !qs_try(bar, parity); ++tries) {
        if ((tries & 255u) != 255u) continue;                                // (reading the timer is slow)
        if (*gave_up) return false;
        if (!t0) pdl_wait();                                                 // the time of a kernel that this one depends on does not count
        uint64_t t1;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
        if (!t0) t0 = t1;
        if (t1 - t0 > 1000000000ull) {
            *gave_up = 1;
            report_wait_error(error, code);
            return false;
        }
    }
    return true;
}
// all lanes of a warp wait; the answer is the warp's
__device__ __forceinline__ bool qs_wait(uint32_t bar, uint32_t parity, volatile uint32_t* gave_up, unsigned int* error, uint32_t code) {
    if (__all_sync(0xffffffffu, qs_try(bar, parity))) return true;
    return __all_sync(0xffffffffu, qs_wait_long(bar, parity, gave_up, error, code));
}
// after a wait that ran out: what is in flight ends before the CTA does
__device__ __forceinline__ void qs_settle(uint32_t bar, uint32_t parity) {
    for (uint32_t n = 0; n < 4096 && !qs_try(bar, parity); ++n) {}
}
__device__ __forceinline__ void qs_tma_2d(uint32_t dst, const CUtensorMap* map, uint32_t x, uint32_t y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ bool qs_elect() {                                 // one lane of a converged warp
    uint32_t p = 0;
    asm volatile("{ .reg .pred q; .reg .b32 r; elect.sync r|q, 0xffffffff; @q mov.u32 %0, 1; }" : "+r"(p));
    return p != 0;
}
__device__ __forceinline__ void qs_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void qs_mma(uint32_t d, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{ .reg .pred p; setp.ne.b32 p, %4, 0; tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p; }" ::"r"(d), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
                 : "memory");
}
__device__ __forceinline__ void qs_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void qs_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void qs_cluster_sync() { asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void qs_tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]),
                 "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
                 : "memory");
}
__device__ __forceinline__ void qs_tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]),
          "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ __nv_bfloat162 qs_b2(uint32_t v) { return *reinterpret_cast<__nv_bfloat162*>(&v); }
__device__ __forceinline__ uint32_t qs_u(__nv_bfloat162 v) { return *reinterpret_cast<uint32_t*>(&v); }

// d (two exact integers code - zp) -> hi = bf16(s d), lo = s d - hi, exact
__device__ __forceinline__ void qs_planes(__nv_bfloat162 d, uint32_t s2, uint32_t& hi, uint32_t& lo) {
    const __nv_bfloat162 h = __hmul2(qs_b2(s2), d);
    hi = qs_u(h);
    lo = qs_u(__hfma2(qs_b2(s2), d, __hneg2(h)));
}
// 8 four-bit codes (k order: nibble 0 first) -> four words of bf16 pairs per plane; z2 = (128 + zp) twice. Nibbles p and p + 4 of a word are 16 bits
// apart: one shift and one LOP3 give the pair 128 + e, PRMT puts the pairs back into k order.
__device__ __forceinline__ void qs_dequant4(uint32_t q, uint32_t z2, uint32_t s2, uint32_t* hi, uint32_t* lo) {
    uint32_t h[4], l[4];
#pragma unroll
    for (int p = 0; p < 4; ++p) qs_planes(__hsub2(qs_b2(((q >> (4 * p)) & 0x000F000Fu) | 0x43004300u), qs_b2(z2)), s2, h[p], l[p]);
    hi[0] = __byte_perm(h[0], h[1], 0x5410); hi[1] = __byte_perm(h[2], h[3], 0x5410); hi[2] = __byte_perm(h[0], h[1], 0x7632); hi[3] = __byte_perm(h[2], h[3], 0x7632);
    lo[0] = __byte_perm(l[0], l[1], 0x5410); lo[1] = __byte_perm(l[2], l[3], 0x5410); lo[2] = __byte_perm(l[0], l[1], 0x7632); lo[3] = __byte_perm(l[2], l[3], 0x7632);
}
// 4 eight-bit codes -> two words per plane; a code is 16 high + low nibble, and so is its zero point: 16 (h - zh) + (l - zl) is exact (|.| <= 255)
__device__ __forceinline__ void qs_dequant8(uint32_t q, uint32_t zh2, uint32_t zl2, uint32_t s2, uint32_t* hi, uint32_t* lo) {
    uint32_t h[2], l[2];                                                     // bytes (0, 2) and (1, 3)
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        const __nv_bfloat162 dl = __hsub2(qs_b2(((q >> (8 * p)) & 0x000F000Fu) | 0x43004300u), qs_b2(zl2));
        const __nv_bfloat162 dh = __hsub2(qs_b2(((q >> (8 * p + 4)) & 0x000F000Fu) | 0x43004300u), qs_b2(zh2));
        qs_planes(__hfma2(qs_b2(0x41804180u), dh, dl), s2, h[p], l[p]);
    }
    hi[0] = __byte_perm(h[0], h[1], 0x5410); hi[1] = __byte_perm(h[0], h[1], 0x7632);
    lo[0] = __byte_perm(l[0], l[1], 0x5410); lo[1] = __byte_perm(l[0], l[1], 0x7632);
}
// The same codes as integers code - zp, exact in bf16, times 2^-11 (bytes: 2^-15): a chain of 128 of them then adds up to no more than the largest
// activation, so an unscaled sum is never out of range where the product is in range. The nibble lies behind the bits of 2^-4 (2^-8) instead of 128.0.
template <int BITS> constexpr uint32_t qs_base = BITS == 4 ? 0x3D80u : 0x3B80u;
template <int BITS> constexpr float qs_unit = BITS == 4 ? 2048.0f : 32768.0f;      // 1 / the integers' factor
__device__ __forceinline__ void qs_integers4(uint32_t q, uint32_t z2, uint32_t* v) {
    uint32_t d[4];
#pragma unroll
    for (int p = 0; p < 4; ++p) d[p] = qs_u(__hsub2(qs_b2(((q >> (4 * p)) & 0x000F000Fu) | qs_base<4> * 0x00010001u), qs_b2(z2)));
    v[0] = __byte_perm(d[0], d[1], 0x5410); v[1] = __byte_perm(d[2], d[3], 0x5410); v[2] = __byte_perm(d[0], d[1], 0x7632); v[3] = __byte_perm(d[2], d[3], 0x7632);
}
__device__ __forceinline__ void qs_integers8(uint32_t q, uint32_t zh2, uint32_t zl2, uint32_t* v) {
    uint32_t d[2];
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        const __nv_bfloat162 dl = __hsub2(qs_b2(((q >> (8 * p)) & 0x000F000Fu) | qs_base<8> * 0x00010001u), qs_b2(zl2));
        const __nv_bfloat162 dh = __hsub2(qs_b2(((q >> (8 * p + 4)) & 0x000F000Fu) | qs_base<8> * 0x00010001u), qs_b2(zh2));
        d[p] = qs_u(__hfma2(qs_b2(0x41804180u), dh, dl));
    }
    v[0] = __byte_perm(d[0], d[1], 0x5410); v[1] = __byte_perm(d[0], d[1], 0x7632);
}
static decltype(&cuTensorMapEncodeTiled) tensor_map_encoder() {
    static decltype(&cuTensorMapEncodeTiled) fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) f = nullptr;
        cudaGetLastError();
        return (decltype(&cuTensorMapEncodeTiled))f;
    }();
    return fn;
}
static bool tensor_map(CUtensorMap* map, CUtensorMapDataType type, uint64_t addr, uint64_t inner, uint64_t outer, uint64_t pitch, uint32_t box_inner, uint32_t box_outer) {
    const cuuint64_t dims[2] = {inner, outer}, strides[1] = {pitch};
    const cuuint32_t box[2] = {box_inner, box_outer}, steps[2] = {1, 1};
    return tensor_map_encoder()(map, type, 2, (void*)addr, dims, strides, box, steps, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

// more than 64 rows of 4-bit ZeroPoint / Symmetric weights in groups of 128 and more (qmm_wide.cu)
struct QwPlan { uint32_t width = 0; float cost = 1e30f; };
QwPlan qw_plan(uint32_t m, uint32_t n, uint32_t nkb, uint32_t sms);
void encode_qmm_wide(uzu_command_buffer* cmd, const uzu_matmul_args& a, QsParams p, uint32_t width);

}  // namespace uzu
