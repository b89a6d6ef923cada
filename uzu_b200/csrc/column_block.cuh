// Blocks of four tokens for the recurrences with independent state columns (gated_delta.cu, general_delta.cu). What the four tokens of a block do
// to one another depends on their vectors alone, not on the state, so it is worked out ahead by producer warps; the consumer warps, which hold the state
// in registers, then take all dot products of a block against the state at its start. One reduction over lanes, one exchange and one update serve four
// tokens instead of one, and a vector that is read from shared memory serves Q columns.
// L lanes own a group of Q columns, lane `part` of them the channels {4 (i L + part) .. + 3}, i < NV.
#pragma once
#include "column_scan.cuh"

namespace uzu {

constexpr int CB_TOKENS = 4;                          // tokens of a block
constexpr int CB_BLOCKS = 4;                          // blocks between two CTA barriers; one producer warp each
constexpr int CB_WARPS = 4;                           // consumer warps
constexpr int CB_THREADS = (CB_WARPS + CB_BLOCKS) * 32;

// two f32 in one 64-bit register: fma.rn.f32x2 rounds each half as fmaf does, for one issue slot
using cb_f2 = unsigned long long;
__device__ __forceinline__ cb_f2 cb_fma2(cb_f2 a, cb_f2 b, cb_f2 c) {
    cb_f2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ cb_f2 cb_mul2(cb_f2 a, cb_f2 b) {
    cb_f2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ cb_f2 cb_pack(float lo, float hi) {
    cb_f2 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ float cb_lo(cb_f2 x) { return __uint_as_float((uint32_t)x); }
__device__ __forceinline__ float cb_hi(cb_f2 x) { return __uint_as_float((uint32_t)(x >> 32)); }
__device__ __forceinline__ float cb_sum2(cb_f2 x) { return cb_lo(x) + cb_hi(x); }

// four channels
struct cb_f4 {
    cb_f2 a, b;
};
__device__ __forceinline__ cb_f4 cb_load4(const float* p) {
    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
    return {v.x, v.y};
}
__device__ __forceinline__ void cb_store4(float* p, const cb_f4& x) { *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(x.a, x.b); }
__device__ __forceinline__ cb_f4 cb_set4(float x) { return {cb_pack(x, x), cb_pack(x, x)}; }
__device__ __forceinline__ cb_f4 cb_mul(const cb_f4& x, const cb_f4& y) { return {cb_mul2(x.a, y.a), cb_mul2(x.b, y.b)}; }
__device__ __forceinline__ cb_f4 cb_scale(const cb_f4& x, cb_f2 s) { return {cb_mul2(x.a, s), cb_mul2(x.b, s)}; }
__device__ __forceinline__ float cb_dot(const cb_f4& x, const cb_f4& y) { return cb_sum2(cb_fma2(x.b, y.b, cb_mul2(x.a, y.a))); }
__device__ __forceinline__ void cb_fma(cb_f4& acc, const cb_f4& x, cb_f2 s) {
    acc.a = cb_fma2(x.a, s, acc.a);
    acc.b = cb_fma2(x.b, s, acc.b);
}

// (j, i) of entry e of a lower triangle stored by rows, without (strict) or with its diagonal
__device__ __forceinline__ void cb_strict(uint32_t e, uint32_t& j, uint32_t& i) {
    j = e >= 3 ? 3u : e >= 1 ? 2u : 1u;
    i = e - j * (j - 1) / 2;
}
__device__ __forceinline__ void cb_lower(uint32_t e, uint32_t& j, uint32_t& i) {
    j = e >= 6 ? 3u : e >= 3 ? 2u : e >= 1 ? 1u : 0u;
    i = e - j * (j + 1) / 2;
}

// T of (1 - n) x = b  <=>  x = T b, for the strictly lower n of four tokens: n = {10, 20, 21, 30, 31, 32}, T in the same places
__device__ __forceinline__ void cb_invert(const float (&n)[6], float (&t)[6]) {
    t[0] = n[0];
    t[2] = n[2];
    t[5] = n[5];
    t[1] = fmaf(n[2], t[0], n[1]);
    t[4] = fmaf(n[5], t[2], n[4]);
    t[3] = fmaf(n[5], t[1], fmaf(n[4], t[0], n[3]));
}

// Q neighbouring values of shared memory, each stored twice
template <int Q>
__device__ __forceinline__ void cb_load(cb_f2 (&x)[Q], const float* p) {
    if constexpr (Q == 2) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
        x[0] = v.x;
        x[1] = v.y;
    } else {
        x[0] = *reinterpret_cast<const cb_f2*>(p);
    }
}

// the lane's part of the dot products of four vectors with its Q columns, in the order (vector, column)
template <int NV, int Q>
__device__ __forceinline__ void cb_dots(float (&o)[CB_TOKENS * Q], const cb_f4 (&x)[CB_TOKENS][NV], const cb_f4 (&s)[Q][NV]) {
#pragma unroll
    for (int j = 0; j < CB_TOKENS; ++j)
#pragma unroll
        for (int c = 0; c < Q; ++c) {
            cb_f2 y = cb_fma2(x[j][0].b, s[c][0].b, cb_mul2(x[j][0].a, s[c][0].a));
#pragma unroll
            for (int n = 1; n < NV; ++n) y = cb_fma2(x[j][n].b, s[c][n].b, cb_fma2(x[j][n].a, s[c][n].a, y));
            o[j * Q + c] = cb_sum2(y);
        }
}

// S += x_j y_j^T over the tokens of a block
template <int NV, int Q>
__device__ __forceinline__ void cb_update(cb_f4 (&s)[Q][NV], const cb_f4 (&x)[CB_TOKENS][NV], const cb_f2 (&y)[CB_TOKENS][Q]) {
#pragma unroll
    for (int j = 0; j < CB_TOKENS; ++j)
#pragma unroll
        for (int c = 0; c < Q; ++c)
#pragma unroll
            for (int n = 0; n < NV; ++n) cb_fma(s[c][n], x[j][n], y[j][c]);
}

// x = T b over the tokens of a block, for Q columns; t = {10, 20, 21, 30, 31, 32}, each stored twice
template <int Q>
__device__ __forceinline__ void cb_solve(cb_f2 (&x)[CB_TOKENS][Q], const cb_f2 (&b)[CB_TOKENS][Q], const float* t) {
    const cb_f4 t0 = cb_load4(t), t1 = cb_load4(t + 4), t2 = cb_load4(t + 8);
#pragma unroll
    for (int c = 0; c < Q; ++c) {
        x[0][c] = b[0][c];
        x[1][c] = cb_fma2(t0.a, b[0][c], b[1][c]);
        x[2][c] = cb_fma2(t1.a, b[1][c], cb_fma2(t0.b, b[0][c], b[2][c]));
        x[3][c] = cb_fma2(t2.b, b[2][c], cb_fma2(t2.a, b[1][c], cb_fma2(t1.b, b[0][c], b[3][c])));
    }
}
__device__ __forceinline__ void cb_store_solve(float* p, const float (&t)[6]) {
#pragma unroll
    for (int e = 0; e < 6; e += 2) *reinterpret_cast<float4*>(p + 2 * e) = make_float4(t[e], t[e], t[e + 1], t[e + 1]);
}

// one of a lane's columns, which differs between lanes
template <int Q>
__device__ __forceinline__ float cb_pick(const cb_f2 (&x)[Q], uint32_t c) {
    return Q == 2 && c ? cb_lo(x[Q - 1]) : cb_lo(x[0]);
}

// acc + the sum over i < n of row[i] x[i]
__device__ __forceinline__ float cb_upto(float acc, const float4& row, const float (&x)[CB_TOKENS], uint32_t n) {
    if (n > 0) acc = fmaf(row.x, x[0], acc);
    if (n > 1) acc = fmaf(row.y, x[1], acc);
    if (n > 2) acc = fmaf(row.z, x[2], acc);
    if (n > 3) acc = fmaf(row.w, x[3], acc);
    return acc;
}

}  // namespace uzu
