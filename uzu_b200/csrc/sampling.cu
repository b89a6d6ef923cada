// UnifiedSamplingKernel: bitmask -> temperature -> top-k / top-p / min-p -> Gumbel-max -> argmax.
// Spec: backends/cpu/kernel/sampling/unified_sampling.rs:22-98; RNG stream layout
// encodable_block/sampling/gumbel.rs:1-81 (Philox4x32-10, key = 64-bit seed, counter = [offset,0,0,0],
// logit i -> (offset, word) = revidx(i, vocab)). Counter-based, so any thread layout reproduces the
// reference's per-logit noise; ties resolve to the lowest index (unified_sampling.rs:90-95).
//
// Two code paths:
//   * no filters (greedy, or temperature + Gumbel): multi-CTA argmax over a packed (value, ~index)
//     64-bit key, last CTA (ticket) merges -> one launch, ~V*2 bytes read at HBM/L2 speed;
//   * with top-k / top-p / min-p: the kept set is a prefix of the (value desc, index asc) order, and equal values are equally likely, so
//     what is kept follows from how often each of the 65536 bf16 values occurs. A cluster of 8 CTAs per row counts them in shared memory
//     (a slice of the row per CTA, 16-bit counts), CTA c adds up the counts of an eighth of the values over distributed shared memory,
//     and the cluster finds the one value at which the kept set ends and how many elements of that value are kept. Noise is then drawn
//     for kept elements only. Sums of probabilities are f64 over exact counts: the same whatever the order of the atomics.
//     Rows whose largest logit is not finite (everything masked, infinities, NaN) walk the candidates one by one instead
//     (sampling_walk: take the best post-noise element of the current set, accept it if its rank and the mass before it pass, otherwise
//     shrink the set to the elements ranked before it; metal/kernel/sampling/unified_sampling.metal:154-238), as do small vocabularies
//     and many rows, where the walk is faster, and a vocabulary whose slice does not fit 16-bit counts.
#include "common.cuh"

namespace uzu {

__device__ __forceinline__ void philox_round(uint32_t (&c)[4], const uint32_t (&k)[2]) {
    const uint32_t hi0 = __umulhi(0xD2511F53u, c[0]), lo0 = 0xD2511F53u * c[0];
    const uint32_t hi1 = __umulhi(0xCD9E8D57u, c[2]), lo1 = 0xCD9E8D57u * c[2];
    const uint32_t n0 = hi1 ^ c[1] ^ k[0], n1 = lo1, n2 = hi0 ^ c[3] ^ k[1], n3 = lo0;
    c[0] = n0; c[1] = n1; c[2] = n2; c[3] = n3;
}

__device__ __forceinline__ float gumbel_noise(uint64_t seed, uint32_t i, uint32_t vocab) {
    // revidx (gumbel.rs:69-81)
    const uint32_t thread_idx = i % 1024u;
    const uint32_t thread_offset = ((vocab + 4095u) / 4096u) * thread_idx;
    const uint32_t block_idx = i / 1024u;
    const uint32_t offset = thread_offset + block_idx / 4u, word = block_idx % 4u;
    uint32_t c[4] = {offset, 0u, 0u, 0u};
    uint32_t k[2] = {(uint32_t)seed, (uint32_t)(seed >> 32)};
    philox_round(c, k);
#pragma unroll
    for (int r = 0; r < 9; ++r) {
        k[0] += 0x9E3779B9u;
        k[1] += 0xBB67AE85u;
        philox_round(c, k);
    }
    const uint32_t w = c[word] >> 8;
    const float u = (float)(w < 1u ? 1u : w) * (1.0f / 16777216.0f);  // unit_interval (gumbel.rs:55-57)
    return -logf(-logf(u));
}

__device__ __forceinline__ float filtered_logit(const uzu_unified_sampling_args& a, const __nv_bfloat16* logits, const uint32_t* bitmask,
                                                float recip_t, uint32_t i) {
    float l = bf2f(logits[i]);
    if (a.has_bitmask && ((bitmask[i >> 5] >> (i & 31)) & 1u) == 0u) l = -INFINITY;
    if (a.has_temperature) l *= recip_t;
    return l;
}

// total order: larger value first, then lower index
__device__ __forceinline__ unsigned long long pack_key(float v, uint32_t i) {
    uint32_t u = __float_as_uint(v);
    if (v != v) u = 0u;  // NaN never wins (the reference's partial_cmp -> Equal keeps the earlier element)
    else u = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
    return ((unsigned long long)u << 32) | (unsigned long long)(0xFFFFFFFFu - i);
}
__device__ __forceinline__ unsigned long long warp_max_u64(unsigned long long k) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long other = __shfl_xor_sync(0xffffffffu, k, o);
        k = other > k ? other : k;
    }
    return k;
}

constexpr uint32_t SAMPLING_WS_SLOTS = 7168;   // u64 partial keys
constexpr uint32_t SAMPLING_MAX_BLOCKS = 28;
constexpr uint32_t SAMPLING_ROWS_PER_LAUNCH = 256;

// rows of whole 16-byte pieces: eight logits per read, their eight mask bits in one word
static bool sampling_whole_pieces(const uzu_unified_sampling_args& a) { return a.vocab_size % 8u == 0 && !(a.logits & 15u); }
// eight logits as they count: masked ones are -inf
__device__ __forceinline__ uint4 masked_piece(const uint16_t* logits, const uint32_t* bitmask, uint32_t i) {
    uint4 x = *reinterpret_cast<const uint4*>(logits + i);
    if (bitmask) {
        const uint32_t on = bitmask[i >> 5] >> (i & 31u);
        uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (!((on >> (2 * j)) & 1u)) w[j] = (w[j] & 0xFFFF0000u) | 0xFF80u;
            if (!((on >> (2 * j + 1)) & 1u)) w[j] = (w[j] & 0xFFFFu) | 0xFF800000u;
        }
        x = make_uint4(w[0], w[1], w[2], w[3]);
    }
    return x;
}
__device__ __forceinline__ uint16_t piece_bits(const uint4& x, int j) {
    const uint32_t w = j < 2 ? x.x : j < 4 ? x.y : j < 6 ? x.z : x.w;
    return (uint16_t)(w >> (16 * (j & 1)));
}

// VEC: a thread's logits come in one or two 16-byte reads instead of a chain of 2-byte ones. Bound: latency (a read, the block's and the grid's maximum;
// with seeds the noise of a thread's logits, one behind another). With seeds a short rest behind whole rounds of pieces is dealt out singly: 1 row of 248320
// logits, 18944 of them such a rest, 12.4 us (as without VEC) against 16.5 with a second piece for some threads, 8 rows 20.6 against 24.6 (22.6 without VEC).
// A rest of six logits a thread and more is as well off as pieces: 400000 logits 16.4 us both ways, 16 rows 51.5 singly, 43.1 as pieces.
template <bool VEC>
__global__ void __launch_bounds__(1024) sampling_argmax_kernel(const uzu_unified_sampling_args a, uint32_t row0, unsigned long long* ws,
                                                               unsigned int* tickets) {
    __shared__ unsigned long long red[32];
    __shared__ unsigned int sm_ticket;
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t row = row0 + blockIdx.y, V = a.vocab_size;
    const __nv_bfloat16* logits = reinterpret_cast<const __nv_bfloat16*>(a.logits) + (size_t)row * V;
    const uint32_t* bitmask = a.has_bitmask ? reinterpret_cast<const uint32_t*>(a.bitmask) + (size_t)row * ((V + 31) / 32) : nullptr;
    const float recip_t = a.has_temperature ? 1.0f / a.temperature : 1.0f;
    const uint64_t seed = a.is_stochastic ? reinterpret_cast<const unsigned long long*>(a.seeds)[row] : 0ull;
    unsigned long long best = 0ull;
    auto offer = [&](float v, uint32_t i) {
        if (a.is_stochastic) v += gumbel_noise(seed, i, V);
        const unsigned long long k = pack_key(v, i);
        best = k > best ? k : best;
    };
    if constexpr (VEC) {
        const uint32_t threads = gridDim.x * blockDim.x, me = blockIdx.x * blockDim.x + threadIdx.x, rest = V % (threads * 8u);
        const uint32_t whole = a.is_stochastic && V > rest && rest <= threads * 5u ? V - rest : V;
        for (uint32_t i = me * 8u; i < whole; i += threads * 8u) {
            const uint4 x = masked_piece(reinterpret_cast<const uint16_t*>(logits), bitmask, i);
#pragma unroll
            for (int j = 0; j < 8; ++j) offer(a.has_temperature ? bf16_bits_to_f32(piece_bits(x, j)) * recip_t : bf16_bits_to_f32(piece_bits(x, j)), i + j);
        }
        for (uint32_t i = whole + me; i < V; i += threads) offer(filtered_logit(a, logits, bitmask, recip_t, i), i);
    } else {
        for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < V; i += gridDim.x * blockDim.x) offer(filtered_logit(a, logits, bitmask, recip_t, i), i);
    }
    best = warp_max_u64(best);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) red[warp] = best;
    __syncthreads();
    if (warp == 0) {
        best = red[lane];
        best = warp_max_u64(best);
        if (lane == 0) {
            if (gridDim.x == 1) {
                reinterpret_cast<uint32_t*>(a.output)[row] = V ? 0xFFFFFFFFu - (uint32_t)(best & 0xFFFFFFFFull) : 0u;
            } else {
                ws[(size_t)blockIdx.y * gridDim.x + blockIdx.x] = best;
                __threadfence();
                sm_ticket = atomicAdd(&tickets[blockIdx.y], 1u);
            }
        }
    }
    if (gridDim.x == 1) return;
    __syncthreads();
    if (sm_ticket != gridDim.x - 1 || warp != 0) return;
    __threadfence();
    unsigned long long k = lane < gridDim.x ? __ldcg(&ws[(size_t)blockIdx.y * gridDim.x + lane]) : 0ull;
    k = warp_max_u64(k);
    if (lane == 0) {
        reinterpret_cast<uint32_t*>(a.output)[row] = 0xFFFFFFFFu - (uint32_t)(k & 0xFFFFFFFFull);
        tickets[blockIdx.y] = 0;
    }
}

// "ranked before c": strictly better in (value desc, index asc)
__device__ __forceinline__ bool ranked_before(float lj, uint32_t j, float lc, uint32_t c) { return lj > lc || (lj == lc && j < c); }

// one CTA of 1024 threads: the candidates of row `row` one by one
__device__ __forceinline__ void sampling_walk(const uzu_unified_sampling_args& a, uint32_t row) {
    __shared__ float redf[32];
    __shared__ unsigned long long redk[32];
    __shared__ unsigned int redc[32];
    __shared__ unsigned long long s_key;
    __shared__ float s_f;
    __shared__ unsigned int s_c;
    const uint32_t V = a.vocab_size;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const __nv_bfloat16* logits = reinterpret_cast<const __nv_bfloat16*>(a.logits) + (size_t)row * V;
    const uint32_t* bitmask = a.has_bitmask ? reinterpret_cast<const uint32_t*>(a.bitmask) + (size_t)row * ((V + 31) / 32) : nullptr;
    const float recip_t = a.has_temperature ? 1.0f / a.temperature : 1.0f;
    const uint64_t seed = a.is_stochastic ? reinterpret_cast<const unsigned long long*>(a.seeds)[row] : 0ull;

    auto block_max_key = [&](unsigned long long k) {
        k = warp_max_u64(k);
        __syncthreads();
        if (lane == 0) redk[warp] = k;
        __syncthreads();
        if (warp == 0) {
            unsigned long long t = lane < nw ? redk[lane] : 0ull;
            t = warp_max_u64(t);
            if (lane == 0) s_key = t;
        }
        __syncthreads();
        return s_key;
    };
    auto block_sum_f = [&](float v) {
        v = warp_sum(v);
        __syncthreads();
        if (lane == 0) redf[warp] = v;
        __syncthreads();
        if (warp == 0) {
            float t = lane < nw ? redf[lane] : 0.0f;
            t = warp_sum(t);
            if (lane == 0) s_f = t;
        }
        __syncthreads();
        return s_f;
    };
    auto block_sum_u = [&](unsigned int v) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        __syncthreads();
        if (lane == 0) redc[warp] = v;
        __syncthreads();
        if (warp == 0) {
            unsigned int t = lane < nw ? redc[lane] : 0u;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            if (lane == 0) s_c = t;
        }
        __syncthreads();
        return s_c;
    };

    // pass 0: max of the filtered logits, softmax normaliser, best post-noise candidate over everything
    unsigned long long kmax = 0ull, kcand = 0ull;
    for (uint32_t i = threadIdx.x; i < V; i += blockDim.x) {
        const float l = filtered_logit(a, logits, bitmask, recip_t, i);
        const unsigned long long k = pack_key(l, i);
        kmax = k > kmax ? k : kmax;
        const float v = a.is_stochastic ? l + gumbel_noise(seed, i, V) : l;
        const unsigned long long kc = pack_key(v, i);
        kcand = kc > kcand ? kc : kcand;
    }
    kmax = block_max_key(kmax);
    kcand = block_max_key(kcand);
    const uint32_t imax = 0xFFFFFFFFu - (uint32_t)(kmax & 0xFFFFFFFFull);
    const float lmax = filtered_logit(a, logits, bitmask, recip_t, imax);
    float part = 0.0f;
    for (uint32_t i = threadIdx.x; i < V; i += blockDim.x) part += expf(filtered_logit(a, logits, bitmask, recip_t, i) - lmax);
    const float norm = block_sum_f(part);
    const float min_p_thr = a.has_min_p ? lmax + logf(a.min_p) : -INFINITY;

    uint32_t cand = 0xFFFFFFFFu - (uint32_t)(kcand & 0xFFFFFFFFull);
    uint32_t result = 0;
    for (uint32_t iter = 0; iter <= V; ++iter) {
        const float lc = filtered_logit(a, logits, bitmask, recip_t, cand);
        // one pass: rank and preceding mass of `cand`, plus the best post-noise element ranked before it
        unsigned int cnt = 0;
        float mass = 0.0f;
        unsigned long long knext = 0ull;
        for (uint32_t j = threadIdx.x; j < V; j += blockDim.x) {
            const float lj = filtered_logit(a, logits, bitmask, recip_t, j);
            if (ranked_before(lj, j, lc, cand)) {
                cnt++;
                mass += expf(lj - lmax) / norm;
                const float v = a.is_stochastic ? lj + gumbel_noise(seed, j, V) : lj;
                const unsigned long long k = pack_key(v, j);
                knext = k > knext ? k : knext;
            }
        }
        const unsigned int rank = block_sum_u(cnt);
        const float mass_before = block_sum_f(mass);
        knext = block_max_key(knext);
        const bool kept = !((a.has_top_k && rank >= a.top_k) || (a.has_top_p && mass_before >= a.top_p) || (a.has_min_p && lc < min_p_thr));
        if (kept) { result = cand; break; }
        if (rank == 0) { result = 0; break; }   // nothing survives the filters: all -inf, argmax = index 0
        cand = 0xFFFFFFFFu - (uint32_t)(knext & 0xFFFFFFFFull);
    }
    if (threadIdx.x == 0) reinterpret_cast<uint32_t*>(a.output)[row] = result;
}

__global__ void __launch_bounds__(1024) sampling_walk_kernel(const uzu_unified_sampling_args a) { sampling_walk(a, blockIdx.x); }
__device__ __noinline__ void sampling_walk_call(const uzu_unified_sampling_args& a, uint32_t row) { sampling_walk(a, row); }

// order-preserving 16-bit key of a bf16 logit; -0 counts as +0 (they compare equal)
__device__ __forceinline__ uint32_t bf16_key(uint16_t bits) {
    if (bits == 0x8000u) bits = 0;
    return (bits & 0x8000u) ? (uint32_t)(uint16_t)~bits : (uint32_t)bits | 0x8000u;
}
__device__ __forceinline__ float key_value(uint32_t key) {
    return bf16_bits_to_f32((key & 0x8000u) ? (uint16_t)(key & 0x7FFFu) : (uint16_t)~key);
}

constexpr uint32_t SF_CTAS = 8, SF_THREADS = 1024;
constexpr uint32_t SF_KEYS = 65536, SF_OWNED = SF_KEYS / SF_CTAS, SF_PER = SF_OWNED / SF_THREADS;    // keys per CTA and per thread when they are added up
constexpr uint32_t SF_PIECES = 4;                    // 16-byte pieces of logits that a thread keeps
constexpr size_t SF_SMEM = SF_KEYS * sizeof(uint16_t);
static_assert(SF_PER == 8, "a thread adds up eight neighbouring keys: one 16-byte read per CTA");

// Bound: latency (a few cluster barriers, one pass over a 128 KB count table). VEC: rows of whole 16-byte pieces, one for every thread and at most four (65536
// to 262144 logits), stay in registers, one read each; otherwise the logits are read twice, two bytes at a time. Below that some threads would count eight
// logits and others none: 1 row of 32768, top-k 50, 21.5 us without VEC and 22.9 with it, 8 rows of 8192 20.6 and 24.6, 1 row of 65536 26.7 and 25.0. 8 rows, temperature, top-k 50, top-p 0.95: 34 us at 128256 logits (40 with the
// two-byte reads), 47 at 248320 (67); 16 rows of 128256 67 us (82).
template <bool VEC>
__global__ void __cluster_dims__(SF_CTAS, 1, 1) __launch_bounds__(SF_THREADS, 1) sampling_filtered_kernel(const uzu_unified_sampling_args a) {
    extern __shared__ __align__(16) uint16_t sf_counts[];
    // what the CTAs of the cluster tell one another, slot = the sender
    __shared__ uint32_t x_top[SF_CTAS], x_n[SF_CTAS], x_edge[SF_CTAS], x_kept[SF_CTAS], x_bad[SF_CTAS];
    __shared__ double x_mass[SF_CTAS];
    __shared__ unsigned long long x_best[SF_CTAS];
    __shared__ double red_d[32];
    __shared__ uint32_t red_u[32];
    __shared__ unsigned long long red_k[32];
    pdl_launch_dependents();
    for (uint32_t i = threadIdx.x; i < SF_KEYS / 8; i += SF_THREADS) reinterpret_cast<uint4*>(sf_counts)[i] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    pdl_wait();
    const uint32_t V = a.vocab_size, row = blockIdx.y, rank = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint16_t* logits = reinterpret_cast<const uint16_t*>(a.logits) + (size_t)row * V;
    const uint32_t* bitmask = a.has_bitmask ? reinterpret_cast<const uint32_t*>(a.bitmask) + (size_t)row * ((V + 31) / 32) : nullptr;
    const float recip_t = a.has_temperature ? 1.0f / a.temperature : 1.0f;
    const uint32_t slice = VEC ? ((V / 8u + SF_CTAS - 1) / SF_CTAS) * 8u : (V + SF_CTAS - 1) / SF_CTAS, lo = min(rank * slice, V), hi = min(lo + slice, V);
    auto masked_bits = [&](uint32_t i) -> uint16_t {
        const bool off = bitmask && ((bitmask[i >> 5] >> (i & 31)) & 1u) == 0u;
        return off ? (uint16_t)0xFF80u : logits[i];
    };
    auto cluster_sync = [] { asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory"); };
    auto remote = [](const void* p, uint32_t cta) {
        uint32_t r;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(cta));
        return r;
    };
    auto tell_u32 = [&](uint32_t* slots, uint32_t v) {      // thread c < SF_CTAS tells CTA c
        if (tid < SF_CTAS) asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(remote(slots + rank, tid)), "r"(v) : "memory");
    };
    auto tell_u64 = [&](void* slot, unsigned long long v) {
        if (tid < SF_CTAS) asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(remote(slot, tid)), "l"(v) : "memory");
    };
    auto block_max_u = [&](uint32_t v) {
        v = __reduce_max_sync(0xffffffffu, v);
        __syncthreads();
        if (lane == 0) red_u[warp] = v;
        __syncthreads();
        return __reduce_max_sync(0xffffffffu, red_u[lane]);
    };
    // exclusive sum over the threads AFTER this one (keys rise with the thread, ranks with falling keys) and the total
    auto suffix_u = [&](uint32_t v, uint32_t& total) {
        uint32_t s = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const uint32_t t = __shfl_down_sync(0xffffffffu, s, o); if (lane + o < 32) s += t; }
        __syncthreads();
        if (lane == 0) red_u[warp] = s;
        __syncthreads();
        uint32_t w = red_u[lane], ws = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const uint32_t t = __shfl_down_sync(0xffffffffu, ws, o); if (lane + o < 32) ws += t; }
        total = __shfl_sync(0xffffffffu, ws, 0);
        return s - v + __shfl_sync(0xffffffffu, ws - w, warp);
    };
    auto suffix_d = [&](double v, double& total) {
        double s = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const double t = __shfl_down_sync(0xffffffffu, s, o); if (lane + o < 32) s += t; }
        const double after = __shfl_down_sync(0xffffffffu, s, 1);
        __syncthreads();
        if (lane == 0) red_d[warp] = s;
        __syncthreads();
        double ws = red_d[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const double t = __shfl_down_sync(0xffffffffu, ws, o); if (lane + o < 32) ws += t; }
        total = __shfl_sync(0xffffffffu, ws, 0);
        const double warps_after = __shfl_down_sync(0xffffffffu, ws, 1);      // lane w: sum of the warps after w
        const double mine = __shfl_sync(0xffffffffu, lane == 31 ? 0.0 : warps_after, warp);
        return (lane == 31 ? 0.0 : after) + mine;
    };

    // 1. count the values of this CTA's slice
    uint32_t bad = 0;
    auto count = [&](uint16_t bits) {
        bad |= (uint32_t)((bits & 0x7FFFu) > 0x7F80u) | (uint32_t)(bits == 0x7F80u);       // NaN, +inf
        const uint32_t key = bf16_key(bits);
        atomicAdd(reinterpret_cast<uint32_t*>(sf_counts) + (key >> 1), (key & 1u) ? 0x10000u : 1u);
    };
    uint4 x[VEC ? SF_PIECES : 1];
    if constexpr (VEC) {
#pragma unroll
        for (uint32_t v = 0; v < SF_PIECES; ++v) {
            const uint32_t i = lo + (v * SF_THREADS + tid) * 8u;
            if (i < hi) x[v] = masked_piece(logits, bitmask, i);
        }
#pragma unroll
        for (uint32_t v = 0; v < SF_PIECES; ++v)
            if (lo + (v * SF_THREADS + tid) * 8u < hi) {
#pragma unroll
                for (int j = 0; j < 8; ++j) count(piece_bits(x[v], j));
            }
    } else {
        for (uint32_t i = lo + tid; i < hi; i += SF_THREADS) count(masked_bits(i));
    }
    bad = (uint32_t)__syncthreads_or((int)bad);
    cluster_sync();
    // 2. add up the eight keys this thread owns over the CTAs' tables
    uint32_t n[SF_PER];
#pragma unroll
    for (uint32_t j = 0; j < SF_PER; ++j) n[j] = 0;
    const uint32_t key0 = rank * SF_OWNED + tid * SF_PER;
#pragma unroll
    for (uint32_t c = 0; c < SF_CTAS; ++c) {
        uint4 v;
        asm volatile("ld.shared::cluster.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(remote(sf_counts + key0, c)));
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) { n[2 * j] += w[j] & 0xFFFFu; n[2 * j + 1] += w[j] >> 16; }
    }
    uint32_t top = 0, mine = 0;
#pragma unroll
    for (uint32_t j = 0; j < SF_PER; ++j) {
        if (n[j]) top = key0 + j;
        mine += n[j];
    }
    uint32_t cta_n;
    const uint32_t after_n = suffix_u(mine, cta_n);
    top = block_max_u(top);
    tell_u32(x_top, top);
    tell_u32(x_n, cta_n);
    tell_u32(x_bad, bad);
    cluster_sync();
    top = 0;
    uint32_t rank0 = after_n;                        // elements with a larger key than this thread's
    for (uint32_t c = 0; c < SF_CTAS; ++c) {
        top = max(top, x_top[c]);
        bad |= x_bad[c];
        if (c > rank) rank0 += x_n[c];
    }
    const float lmax = key_value(top) * recip_t;
    // not finite, or a temperature that could make different values equal: the general walk
    if (bad || !(fabsf(lmax) < INFINITY) || !(recip_t > 1.52587890625e-5f && recip_t < 65536.0f)) {
        if (rank == 0) sampling_walk_call(a, row);
        return;                                      // (uniform over the cluster; no CTA reads another's memory any more)
    }
    // 3. probabilities: f64 sums of counts * exp(l - lmax)
    double e[SF_PER], mass = 0.0;
#pragma unroll
    for (uint32_t j = 0; j < SF_PER; ++j) {
        e[j] = n[j] ? (double)expf(key_value(key0 + j) * recip_t - lmax) : 0.0;
        mass += (double)n[j] * e[j];
    }
    double cta_mass;
    double mass0 = suffix_d(mass, cta_mass);
    tell_u64(x_mass + rank, (unsigned long long)__double_as_longlong(cta_mass));
    cluster_sync();
    double norm = 0.0;
    for (uint32_t c = 0; c < SF_CTAS; ++c) {
        norm += x_mass[c];
        if (c > rank) mass0 += x_mass[c];
    }
    // 4. the kept elements of each value: those of rank < top_k, mass before < top_p, value >= min_p threshold. The kept set ends at the
    //    largest key that is not kept as a whole.
    const float min_p_thr = a.has_min_p ? lmax + logf(a.min_p) : -INFINITY;
    const double limit = (double)a.top_p * norm;
    uint32_t edge = 0, kept_at_edge = 0;             // edge = key + 1, 0 = none
#pragma unroll
    for (int j = (int)SF_PER - 1; j >= 0; --j) {
        if (n[j] && !edge) {
            uint32_t q = n[j];
            if (a.has_top_k) q = rank0 >= a.top_k ? 0u : min(q, a.top_k - rank0);
            if (a.has_top_p) {                       // element i of this value is kept while mass0 + i e < limit
                const double room = limit - mass0;
                if (room <= 0.0) q = 0;              // (a top_p that is NaN cuts nothing off)
                else if (e[j] > 0.0 && room < e[j] * (double)q) q = min(q, (uint32_t)ceil(room / e[j]));
            }
            if (a.has_min_p && key_value(key0 + j) * recip_t < min_p_thr) q = 0;
            if (q < n[j]) { edge = key0 + j + 1; kept_at_edge = q; }
        }
        rank0 += n[j];
        mass0 += (double)n[j] * e[j];
    }
    const uint32_t cta_edge = block_max_u(edge);
    __syncthreads();                                 // all have read red_u
    if (cta_edge && edge == cta_edge) red_u[0] = kept_at_edge;       // (one thread owns the key)
    __syncthreads();
    kept_at_edge = red_u[0];
    tell_u32(x_edge, cta_edge);
    tell_u32(x_kept, kept_at_edge);
    cluster_sync();
    edge = 0;
    uint32_t quota = 0;
    for (uint32_t c = 0; c < SF_CTAS; ++c)
        if (x_edge[c] > edge) { edge = x_edge[c]; quota = x_kept[c]; }
    // 5. elements of the edge value are kept by rising index: the slices before this CTA's come first
    const uint32_t edge_key = edge - 1;              // (edge = 0: every element is kept)
    for (uint32_t c = 0; edge && c < rank; ++c) {    // (their tables stay: no CTA leaves before the last barrier)
        uint16_t same;
        asm volatile("ld.shared::cluster.u16 %0, [%1];" : "=h"(same) : "r"(remote(sf_counts + edge_key, c)));
        quota -= min(quota, (uint32_t)same);
    }
    const uint64_t seed = a.is_stochastic ? reinterpret_cast<const unsigned long long*>(a.seeds)[row] : 0ull;
    unsigned long long best = 0ull;
    auto offer = [&](uint32_t i, uint16_t bits) {
        float v = bf16_bits_to_f32(bits) * recip_t;
        if (a.is_stochastic) v += gumbel_noise(seed, i, V);
        const unsigned long long k = pack_key(v, i);
        best = k > best ? k : best;
    };
    const bool count_equal = edge != 0 && quota != 0 && quota < sf_counts[edge_key];     // (uniform over the CTA)
    if constexpr (VEC) {
#pragma unroll
        for (uint32_t v = 0; v < SF_PIECES; ++v) {
            const uint32_t i = lo + (v * SF_THREADS + tid) * 8u;
            uint32_t equal = 0, keep = 0;            // a bit per logit of the piece
            if (i < hi) {
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const uint32_t key = bf16_key(piece_bits(x[v], j)) + 1u;
                    keep |= (uint32_t)(key > edge) << j;
                    equal |= (uint32_t)(edge != 0 && key == edge) << j;
                }
            }
            if (count_equal) {
                const uint32_t own = (uint32_t)__popc(equal);
                uint32_t upto = own;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) { const uint32_t t = __shfl_up_sync(0xffffffffu, upto, o); if (lane >= o) upto += t; }
                __syncthreads();
                if (lane == 31) red_u[warp] = upto;
                __syncthreads();
                const uint32_t w = red_u[lane], all = __reduce_add_sync(0xffffffffu, w);
                uint32_t left = __reduce_add_sync(0xffffffffu, lane < warp ? w : 0u) + upto - own;       // equal ones before this piece
                left = quota > left ? quota - left : 0u;
                for (uint32_t m = equal; m && left; m &= m - 1u, --left) keep |= m & (0u - m);
                quota -= min(quota, all);
            } else if (quota != 0) keep |= equal;
            for (; keep; keep &= keep - 1u) {
                const int j = __ffs(keep) - 1;
                offer(i + j, piece_bits(x[v], j));
            }
        }
    }
    for (uint32_t i0 = VEC ? hi : lo; i0 < hi; i0 += SF_THREADS) {
        const uint32_t i = i0 + tid;
        const uint16_t bits = i < hi ? masked_bits(i) : (uint16_t)0xFF80u;
        const uint32_t key = i < hi ? bf16_key(bits) + 1u : 0u;
        bool keep = i < hi && key > edge;
        const bool equal = edge != 0 && key == edge;
        if (count_equal) {
            const uint32_t b = __ballot_sync(0xffffffffu, equal);
            __syncthreads();
            if (lane == 0) red_u[warp] = (uint32_t)__popc(b);
            __syncthreads();
            const uint32_t w = red_u[lane];
            const uint32_t before = __reduce_add_sync(0xffffffffu, lane < warp ? w : 0u) + (uint32_t)__popc(b & ((1u << lane) - 1u));
            const uint32_t all = __reduce_add_sync(0xffffffffu, w);
            if (equal && before < quota) keep = true;
            quota -= min(quota, all);
        } else if (equal && quota != 0) keep = true;
        if (keep) offer(i, bits);
    }
    best = warp_max_u64(best);
    if (lane == 0) red_k[warp] = best;
    __syncthreads();
    best = warp_max_u64(red_k[lane]);
    if (tid == 0) asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(remote(x_best + rank, 0)), "l"(best) : "memory");
    cluster_sync();
    if (rank == 0 && warp == 0) {
        best = warp_max_u64(lane < SF_CTAS ? x_best[lane] : 0ull);
        if (lane == 0) reinterpret_cast<uint32_t*>(a.output)[row] = best ? 0xFFFFFFFFu - (uint32_t)(best & 0xFFFFFFFFull) : 0u;   // nothing kept: index 0
    }
}

}  // namespace uzu

extern "C" {

void uzu_unified_sampling_encode(uzu_command_buffer* cmd, const uzu_unified_sampling_args* a) {
    if (!uzu::encodable(cmd, "unified_sampling")) return;
    if (!a->logits || !a->output || (a->is_stochastic && !a->seeds) || (a->has_bitmask && !a->bitmask) || a->vocab_size == 0 ||
        (a->has_temperature && !(a->temperature > 0.0f))) {
        cmd->record_error(UZU_ERROR_INVALID_ARGUMENT, "unified_sampling: inconsistent arguments");
        return;
    }
    if (a->batch_size == 0) return;
    uzu_context* ctx = cmd->ctx;
    if (a->has_top_k || a->has_top_p || a->has_min_p) {
        // us of both forms: counting takes about 18 us for each 15 rows (as many clusters fit the chip at a time), the walk one pass over the row per
        // candidate, more of them in the unluckiest of several rows. Walk / count: 1 row of 4096 logits 14 / 21, of 16384 34 / 21; 16 rows of 8192 37 / 37, of
        // 32768 80 / 42; 64 rows of 32768 72 / 104, of 65536 155 / 117.
        const float count_us = 3.0f + (float)((a->batch_size + 14u) / 15u) * (18.0f + 8e-5f * a->vocab_size);
        const float walk_us = 9.0f + (a->batch_size == 1 ? 0.0015f : 0.0019f) * a->vocab_size;
        if (walk_us < count_us || a->vocab_size > uzu::SF_CTAS * 65535u) {      // (16-bit counts per slice)
            uzu::sampling_walk_kernel<<<a->batch_size, 1024, 0, ctx->stream>>>(*a);
            uzu::after_launch(cmd, "sampling_walk_kernel");
            return;
        }
        constexpr uint32_t piece_each = uzu::SF_CTAS * uzu::SF_THREADS * 8u;
        const bool pieces = uzu::sampling_whole_pieces(*a) && a->vocab_size >= piece_each && a->vocab_size <= piece_each * uzu::SF_PIECES;
        const auto kernel = pieces ? uzu::sampling_filtered_kernel<true> : uzu::sampling_filtered_kernel<false>;
        static std::atomic<uint64_t> smem_opt_in[2];
        uzu::opt_in_dynamic_smem(cmd, kernel, (int)uzu::SF_SMEM, smem_opt_in[pieces]);
        for (uint32_t row0 = 0; row0 < a->batch_size; row0 += 65535u) {      // (rows are the grid's y axis)
            uzu_unified_sampling_args b = *a;
            b.logits += (uint64_t)row0 * a->vocab_size * 2; b.output += (uint64_t)row0 * 4; b.seeds += a->is_stochastic ? (uint64_t)row0 * 8 : 0;
            b.bitmask += a->has_bitmask ? (uint64_t)row0 * ((a->vocab_size + 31) / 32) * 4 : 0;
            b.batch_size = std::min(65535u, a->batch_size - row0);
            uzu::launch(cmd, "sampling_filtered_kernel", kernel, dim3(uzu::SF_CTAS, b.batch_size), dim3(uzu::SF_THREADS), uzu::SF_SMEM, b);
        }
        return;
    }
    uint32_t nblocks = std::min(uzu::SAMPLING_MAX_BLOCKS, (a->vocab_size + 8191u) / 8192u);
    nblocks = std::max(nblocks, 1u);
    unsigned int* tickets = reinterpret_cast<unsigned int*>(ctx->sampling_ws + uzu::SAMPLING_WS_SLOTS);
    for (uint32_t row0 = 0; row0 < a->batch_size; row0 += uzu::SAMPLING_ROWS_PER_LAUNCH) {
        const uint32_t rows = std::min(uzu::SAMPLING_ROWS_PER_LAUNCH, a->batch_size - row0);
        dim3 grid(nblocks, rows);
        uzu::launch(cmd, "sampling_argmax_kernel", uzu::sampling_whole_pieces(*a) ? uzu::sampling_argmax_kernel<true> : uzu::sampling_argmax_kernel<false>, grid, dim3(1024), 0, *a, row0, ctx->sampling_ws, tickets);
    }
}

}  // extern "C"
