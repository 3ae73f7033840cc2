// On-device token choice (crates/runtime/src/sampler.rs:148-170): greedy argmax.
#include <math.h>

#include "brasa_internal.h"

namespace {

struct Best {
    float v;
    uint32_t i;
};
// larger value wins; equal values keep the smaller index (first maximum)
__device__ __forceinline__ Best better(Best a, Best b) { return (b.v > a.v || (b.v == a.v && b.i < a.i)) ? b : a; }

__device__ Best block_best(Best b, Best *sh) {
    for (int o = 16; o > 0; o >>= 1) {
        Best other{__shfl_xor_sync(0xffffffffu, b.v, o), __shfl_xor_sync(0xffffffffu, b.i, o)};
        b = better(b, other);
    }
    int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) sh[warp] = b;
    __syncthreads();
    if (warp == 0) {
        b = lane < (int)(blockDim.x >> 5) ? sh[lane] : Best{-INFINITY, 0xffffffffu};
        for (int o = 16; o > 0; o >>= 1) {
            Best other{__shfl_xor_sync(0xffffffffu, b.v, o), __shfl_xor_sync(0xffffffffu, b.i, o)};
            b = better(b, other);
        }
    }
    return b;  // valid in warp 0
}

// NaN never compares greater, so it never wins; an all -inf (or empty) input yields index 0.
__global__ void __launch_bounds__(256) argmax_kernel(const float *v, uint32_t n, uint32_t *out, Best *partial, uint32_t *counter) {
    __shared__ Best sh[8];
    __shared__ bool last;
    Best b{-INFINITY, 0xffffffffu};
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float x = v[i];
        if (x > b.v) b = Best{x, i};
    }
    b = block_best(b, sh);
    if (threadIdx.x == 0) {
        partial[blockIdx.x] = b;
        __threadfence();
        last = atomicAdd(counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    Best f{-INFINITY, 0xffffffffu};
    for (uint32_t i = threadIdx.x; i < gridDim.x; i += blockDim.x) {
        Best pb;
        pb.v = __ldcg(&partial[i].v);
        pb.i = __ldcg(&partial[i].i);
        f = better(f, pb);
    }
    f = block_best(f, sh);
    if (threadIdx.x == 0) {
        *out = (f.v == -INFINITY || f.i == 0xffffffffu) ? 0u : f.i;
        *counter = 0;
    }
}

// End of a decode step: the chosen token becomes the next input, is appended to the output list, and
// the position advances. One thread.
__global__ void advance_kernel(uint32_t *ids, const uint32_t *next, uint32_t *out_ids, uint32_t *out_count, uint32_t out_cap, uint32_t *pos) {
    uint32_t tok = *next;
    ids[0] = tok;
    uint32_t n = *out_count;
    if (n < out_cap) out_ids[n] = tok;
    *out_count = n + 1;
    *pos += 1;
}


// ---- temperature / top-k / top-p sampling on the device (crates/runtime/src/sampler.rs:60-146) ----------------
// The reference sorts the candidates (descending logit, f32 total order), turns them into weights
// exp((l - max) / T), keeps the shortest prefix whose normalised mass reaches top_p and walks that prefix with one
// PCG32 draw. Here nothing is sorted: a prefix of the sorted order is the set {key > t, or key = t and id <= i}, and the
// three prefixes the algorithm needs (the top_k-th candidate, the top_p cut, the drawn token) are each found in five
// steps: among 256 steps of (max - l) / T first (logits of one vocabulary share two or three values of their key's top byte: a
// histogram over that byte is one long queue on the same word), then by histograms over the four bytes of the 32-bit order key among the
// candidates of the chosen step. A count over ascending ids settles equal logits (they keep ascending id, as in the host sampler).
// Masses are 64-bit fixed point (weight x 2^k with n 2^k <= 2^62, truncated): sums do not depend on the order of the
// additions, and what truncation loses is below 2^-26 of the largest weight for 2^18 candidates, a quarter of one rounding
// of the f32 sums the reference forms.
// A row is one cluster of eight blocks, each with an eighth of the ids, or one block (see sample_launch); a cluster's histograms meet through
// distributed shared memory, one cluster barrier per histogram. The logits are read twice, for the maximum and for the first histogram, which also leaves every id's step as a
// byte in shared memory; the later passes look at four steps per word and touch the few logits that match (vocabularies too long for
// that work the step out again). Bound: latency, some ten passes of a barrier each. One row of 151 936: 79 us (3 840 with one block a row
// that bisected over the whole row, 158 with every pass over the logits); a step of 64 rows 113 us (240 as eleven launches).
struct Prefix {
    uint32_t t;   // candidates with key > t are in
    uint32_t id;  // candidates with key == t are in when their id <= id
};

__device__ __forceinline__ uint32_t order_key(float f) {  // larger key = earlier in the descending total order
    int32_t b = __float_as_int(f);
    b ^= (int32_t)(((uint32_t)(b >> 31)) >> 1);
    return (uint32_t)b ^ 0x80000000u;
}
__device__ __forceinline__ float key_value(uint32_t k) {  // inverse of order_key
    int32_t b = (int32_t)(k ^ 0x80000000u);
    b ^= (int32_t)(((uint32_t)(b >> 31)) >> 1);
    return __int_as_float(b);
}
__device__ __forceinline__ bool in_prefix(uint32_t key, uint32_t id, Prefix p) { return key > p.t || (key == p.t && id <= p.id); }

constexpr int SM_THREADS = 512, SM_WARPS = SM_THREADS / 32, SM_CLUSTER = 8;  // (a row's blocks: CL, 1 or SM_CLUSTER)

template <int CL>
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r = 0;
    if (CL > 1) asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
template <int CL>
__device__ __forceinline__ void cluster_sync() {
    if (CL == 1) {
        __syncthreads();
        return;
    }
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
template <int CL>
__device__ __forceinline__ unsigned long long cluster_load(const unsigned long long *local, uint32_t rank) {  // the same word of block `rank`
    if (CL == 1) return *local;
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(local);
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(a), "r"(rank));
    unsigned long long v;
    asm volatile("ld.shared::cluster.u64 %0, [%1];" : "=l"(v) : "r"(remote) : "memory");
    return v;
}

struct SampleShared {
    unsigned long long wh[SM_WARPS][256];  // a histogram per warp
    unsigned long long hist[2][256];       // the block's, read by the cluster; two, so that one barrier per pass is enough
    unsigned long long word[2];            // one number per block, likewise
    unsigned long long mass[256], count[256];  // of the steps, over the cluster and the kept candidates
    unsigned long long wtot[8], bound, above, hit;
    uint32_t wcnt[SM_WARPS], bin, pass;
};

// The sum over the cluster of one number per block, and the sum over the blocks before this one.
template <int CL>
__device__ unsigned long long cluster_sum(SampleShared &s, unsigned long long mine, unsigned long long &before) {
    const uint32_t buf = s.pass & 1, me = cluster_rank<CL>();
    if (threadIdx.x == 0) s.word[buf] = mine;
    cluster_sync<CL>();
    unsigned long long all = 0;
    before = 0;
    for (uint32_t r = 0; r < CL; ++r) {
        const unsigned long long v = cluster_load<CL>(&s.word[buf], r);
        all += v;
        if (r < me) before += v;
    }
    __syncthreads();
    if (threadIdx.x == 0) ++s.pass;
    __syncthreads();
    return all;
}

struct SampleRow {
    const float *l;
    uint32_t lo, hi;    // this block's ids
    const uint8_t *steps;  // of this block's ids, in shared memory; null: worked out again
    float mx, temperature, per_step, fix;
    __device__ __forceinline__ unsigned long long weight(float v) const {
        const float w = expf((v - mx) / temperature) * fix;
        return w > 0.0f ? __float2ull_rz(w) : 0ull;  // (a NaN weighs nothing)
    }
    __device__ __forceinline__ uint32_t step(float v) const {  // never larger for a larger logit
        const float x = (mx - v) * per_step;
        return x < 255.0f ? (uint32_t)x : 255u;
    }
    // bit j: id lo + i + j (four from i, a multiple of four) belongs to this step
    __device__ __forceinline__ uint32_t four(uint32_t i, uint32_t at) const {
        const uint32_t n = hi - lo;
        if (i >= n) return 0u;
        uint32_t m = 0;
        if (steps) {
            const uint32_t eq = __vcmpeq4(*reinterpret_cast<const uint32_t *>(steps + i), at * 0x01010101u);
            m = (eq & 1u) | ((eq >> 7) & 2u) | ((eq >> 14) & 4u) | ((eq >> 21) & 8u);
        } else {
            for (uint32_t j = 0; j < 4; ++j) m |= (i + j < n && step(l[lo + i + j]) == at ? 1u : 0u) << j;
        }
        return i + 4 <= n ? m : m & ((1u << (n - i)) - 1u);
    }
};

// s.hist[buf] = the sum over the warps' histograms
__device__ __forceinline__ void block_hist(SampleShared &s, uint32_t buf) {
    __syncthreads();
    if (threadIdx.x < 256) {
        unsigned long long a = 0;
#pragma unroll
        for (int w = 0; w < SM_WARPS; ++w) a += s.wh[w][threadIdx.x];
        s.hist[buf][threadIdx.x] = a;
    }
}
template <int CL>
__device__ __forceinline__ unsigned long long cluster_bin(const SampleShared &s, uint32_t buf) {  // thread < 256: its bin over the cluster
    unsigned long long h = 0;
#pragma unroll
    for (uint32_t r = 0; r < CL; ++r) h += cluster_load<CL>(&s.hist[buf][threadIdx.x], r);
    return h;
}
// The first bin at which `above` and the bins so far reach s.bound: into s.bin, what lies before it into s.above. h: thread's bin (thread
// < 256). Sets s.bound first when `share` does (from the sum over the bins).
template <typename Bound>
__device__ __forceinline__ void pick_bin(SampleShared &s, unsigned long long h, bool first, Bound bound_of) {
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    unsigned long long v = h;
    if (tid < 256) {
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long up = __shfl_up_sync(0xffffffffu, v, o);
            if ((int)lane >= o) v += up;
        }
        if (lane == 31) s.wtot[warp] = v;
    }
    __syncthreads();
    if (tid == 0 && first) {
        unsigned long long total = 0;
        for (int w = 0; w < 8; ++w) total += s.wtot[w];
        const unsigned long long bound = bound_of(total);
        s.bound = bound < 1 ? 1 : bound;  // (a draw of 0 takes the first candidate)
        s.above = 0;
    }
    __syncthreads();
    const unsigned long long bound = s.bound, above = s.above;
    if (tid < 256) {
        for (uint32_t w = 0; w < warp; ++w) v += s.wtot[w];
        v += above;
    }
    __syncthreads();  // everyone has read `above`
    if (tid < 256 && v >= bound && v - h < bound) {  // exactly one bin
        s.bin = tid;
        s.above = v - h;
    }
    __syncthreads();
}

enum SampleBound { BOUND_COUNT, BOUND_SHARE, BOUND_DRAW };

// Narrows `inside` to its shortest prefix whose mass reaches the bound (top_k candidates; top_p of its mass; u24 / 2^24 of
// its mass, at least one unit). s.mass and s.count are those of `inside`, and of the narrowed one afterwards unless it is the draw.
template <SampleBound KIND, int CL>
__device__ Prefix select_prefix(SampleShared &s, const SampleRow &row, Prefix inside, uint32_t top_k, float top_p, uint32_t u24) {
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, len = row.hi - row.lo;
    pick_bin(s, tid < 256 ? (KIND == BOUND_COUNT ? s.count[tid] : s.mass[tid]) : 0ull, true, [&](unsigned long long total) -> unsigned long long {
        if (KIND == BOUND_COUNT) return top_k;
        if (KIND == BOUND_SHARE) {
            const double b = ceil((double)total * (double)top_p);
            return b >= (double)total ? total : (unsigned long long)b;
        }
        const unsigned long long hi64 = __umul64hi(total, (unsigned long long)u24), lo64 = total * (unsigned long long)u24;  // ceil(total u24 / 2^24)
        return ((hi64 << 40) | (lo64 >> 24)) + ((lo64 & 0xffffffull) ? 1 : 0);
    });
    const uint32_t step = s.bin;
    uint32_t pref = 0;
    for (int shift = 24; shift >= 0; shift -= 8) {
        const uint32_t buf = s.pass & 1;
        for (uint32_t i = tid; i < SM_WARPS * 256; i += SM_THREADS) (&s.wh[0][0])[i] = 0;
        __syncthreads();
        for (uint32_t i = 4 * tid; i < len; i += 4 * SM_THREADS) {
            for (uint32_t m = row.four(i, step); m; m &= m - 1) {
                const uint32_t id = row.lo + i + __ffs(m) - 1;
                const float v = row.l[id];
                const uint32_t k = order_key(v);
                if (shift < 24 && (k >> (shift + 8)) != (pref >> (shift + 8))) continue;
                if (!in_prefix(k, id, inside)) continue;
                const unsigned long long w = KIND == BOUND_COUNT ? 1ull : row.weight(v);
                if (w) atomicAdd(&s.wh[warp][255u - ((k >> shift) & 255u)], w);
            }
        }
        block_hist(s, buf);
        cluster_sync<CL>();
        const unsigned long long h = tid < 256 ? cluster_bin<CL>(s, buf) : 0ull;
        __syncthreads();
        if (tid == 0) ++s.pass;
        pick_bin(s, h, false, [](unsigned long long) { return 0ull; });
        pref |= (255u - s.bin) << shift;
        __syncthreads();
    }
    // the prefix ends with the m-th, in ascending id order, of the candidates whose key is `pref`
    const unsigned long long wt = KIND == BOUND_COUNT ? 1ull : row.weight(key_value(pref)), m = (s.bound - s.above + wt - 1) / wt;
    const uint32_t span = ((len + SM_WARPS - 1) / SM_WARPS + 3) & ~3u, b = min(len, warp * span), e = min(len, b + span);
    auto equals = [&](uint32_t i) {  // of the four ids from i, those with that key
        uint32_t has = 0;
        for (uint32_t c = i < e ? row.four(i, step) : 0u; c; c &= c - 1) {
            const uint32_t j = __ffs(c) - 1, id = row.lo + i + j;
            if (order_key(row.l[id]) == pref && in_prefix(pref, id, inside)) has |= 1u << j;
        }
        return has;
    };
    uint32_t cnt = 0;
    for (uint32_t i0 = b; i0 < e; i0 += 128) cnt += __popc(equals(i0 + 4 * lane));
    for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    if (lane == 0) s.wcnt[warp] = cnt;
    __syncthreads();
    uint32_t mine = 0, before_warp = 0;
    for (uint32_t w = 0; w < SM_WARPS; ++w) {
        if (w < warp) before_warp += s.wcnt[w];
        mine += s.wcnt[w];
    }
    unsigned long long before;
    cluster_sum<CL>(s, mine, before);
    before += before_warp;
    if (tid == 0) s.hit = 0;
    __syncthreads();
    if (before < m && m <= before + cnt) {  // one warp of the cluster
        uint32_t left = (uint32_t)(m - before);
        for (uint32_t i0 = b; i0 < e; i0 += 128) {
            uint32_t has = equals(i0 + 4 * lane), incl = __popc(has);
            const uint32_t own = incl;
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t up = __shfl_up_sync(0xffffffffu, incl, o);
                if ((int)lane >= o) incl += up;
            }
            const uint32_t all = __shfl_sync(0xffffffffu, incl, 31);
            if (left <= all) {
                if (left > incl - own && left <= incl) {
                    for (uint32_t k = left - (incl - own); k > 1; --k) has &= has - 1;
                    s.hit = row.lo + i0 + 4 * lane + __ffs(has);  // id + 1
                }
                break;
            }
            left -= all;
        }
    }
    __syncthreads();
    unsigned long long unused;
    const unsigned long long id1 = cluster_sum<CL>(s, s.hit, unused);
    const Prefix cut{pref, (uint32_t)id1 - 1};
    if (KIND != BOUND_DRAW) {  // what the narrowed prefix holds of each step
        unsigned long long c = 0, w = 0;
        for (uint32_t i = 4 * tid; i < len; i += 4 * SM_THREADS)
            for (uint32_t f = row.four(i, step); f; f &= f - 1) {
                const uint32_t id = row.lo + i + __ffs(f) - 1;
                const float v = row.l[id];
                if (in_prefix(order_key(v), id, cut) && in_prefix(order_key(v), id, inside)) {
                    ++c;
                    w += row.weight(v);
                }
            }
        for (int o = 16; o > 0; o >>= 1) {
            c += __shfl_xor_sync(0xffffffffu, c, o);
            w += __shfl_xor_sync(0xffffffffu, w, o);
        }
        __syncthreads();
        if (lane == 0) {
            s.wh[warp][0] = c;
            s.wh[warp][1] = w;
        }
        __syncthreads();
        c = w = 0;
        for (int k = 0; k < SM_WARPS; ++k) {
            c += s.wh[k][0];
            w += s.wh[k][1];
        }
        c = cluster_sum<CL>(s, c, unused);
        w = cluster_sum<CL>(s, w, unused);
        if (tid < 256 && tid >= step) {
            s.count[tid] = tid == step ? c : 0ull;
            s.mass[tid] = tid == step ? w : 0ull;
        }
        __syncthreads();
    }
    return cut;
}

// Row r: logits[r n ..], the PCG32 state at rng + 2 r, the token at out + r. keep_steps: the dynamic shared memory holds a byte per id of
// a block. A kept candidate whose weight is NaN (a NaN among the logits, an infinite largest one, nothing but -inf) makes the reference's
// sums NaN, which no comparison stops: its walk ends at the last of the top_k kept candidates, and that is the token here.
template <int CL>
__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(SM_THREADS, 2)
    sample_kernel(const float *logits, uint32_t n, float temperature, uint32_t top_k, float top_p, float fix, bool keep_steps,
                  unsigned long long *rng, uint32_t *out) {
    extern __shared__ __align__(16) uint8_t step_bytes[];
    __shared__ SampleShared s;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, r = blockIdx.x / CL, me = cluster_rank<CL>();
    const uint32_t seg = (uint32_t)(((uint64_t)n + CL - 1) / CL);
    SampleRow row;
    row.l = logits + (size_t)r * n;
    row.lo = (uint32_t)min((uint64_t)n, (uint64_t)me * seg);
    row.hi = (uint32_t)min((uint64_t)n, (uint64_t)row.lo + seg);
    row.steps = keep_steps ? step_bytes : nullptr;
    row.temperature = temperature;
    row.per_step = 8.0f / temperature;
    row.fix = fix;
    if (tid == 0) s.pass = 0;
    uint32_t kmax = 0, kmin = 0xffffffffu;
#pragma unroll 8
    for (uint32_t i = row.lo + tid; i < row.hi; i += SM_THREADS) {
        const uint32_t k = order_key(row.l[i]);
        kmax = max(kmax, k);
        kmin = min(kmin, k);
    }
    kmax = __reduce_max_sync(0xffffffffu, kmax);
    kmin = __reduce_min_sync(0xffffffffu, kmin);
    if (lane == 0) s.mass[warp] = ((unsigned long long)kmax << 32) | kmin;
    for (uint32_t i = tid; i < SM_WARPS * 256; i += SM_THREADS) (&s.wh[0][0])[i] = 0;
    __syncthreads();
    for (uint32_t w = 0; w < SM_WARPS; ++w) {
        kmax = max(kmax, (uint32_t)(s.mass[w] >> 32));
        kmin = min(kmin, (uint32_t)s.mass[w]);
    }
    if (tid == 0) s.word[0] = ((unsigned long long)kmax << 32) | kmin;
    cluster_sync<CL>();
    for (uint32_t b = 0; b < CL; ++b) {
        const unsigned long long v = cluster_load<CL>(&s.word[0], b);
        kmax = max(kmax, (uint32_t)(v >> 32));
        kmin = min(kmin, (uint32_t)v);
    }
    if (tid == 0) s.pass = 1;
    __syncthreads();
    row.mx = key_value(kmax);
    const unsigned long long old = rng[2 * (size_t)r], inc = rng[2 * (size_t)r + 1];
    // below: every candidate whose key is smaller has a NaN for its weight. to_end: some kept candidate has, whatever top_k keeps. (Every
    // step is 255 where the largest logit or the temperature is no number, so that the count below needs no other form.)
    const uint32_t below = order_key(-INFINITY) + (isinf(temperature) ? 1u : 0u);
    const bool keep_all = top_k == 0 || top_k >= n, to_end = !isfinite(row.mx) || isnan(temperature) || (keep_all && kmin < below);
    const bool counted = !keep_all || to_end;
    // mass (and count) of every step
#pragma unroll 4
    for (uint32_t i = row.lo + tid; i < row.hi; i += SM_THREADS) {
        const float v = row.l[i];
        const uint32_t at = row.step(v);
        if (keep_steps) step_bytes[i - row.lo] = (uint8_t)at;
        const unsigned long long w = row.weight(v);
        if (w) atomicAdd(&s.wh[warp][at], w);
    }
    block_hist(s, 1);
    cluster_sync<CL>();
    if (tid < 256) s.mass[tid] = cluster_bin<CL>(s, 1);
    __syncthreads();
    if (tid == 0) s.pass = 2;
    if (counted) {
        for (uint32_t i = tid; i < SM_WARPS * 256; i += SM_THREADS) (&s.wh[0][0])[i] = 0;
        __syncthreads();
        for (uint32_t i = row.lo + tid; i < row.hi; i += SM_THREADS) atomicAdd(&s.wh[warp][keep_steps ? step_bytes[i - row.lo] : row.step(row.l[i])], 1ull);
        block_hist(s, 0);
        cluster_sync<CL>();
        if (tid < 256) s.count[tid] = cluster_bin<CL>(s, 0);
        __syncthreads();
        if (tid == 0) s.pass = 3;
    }
    __syncthreads();
    const uint32_t x = (uint32_t)(((old >> 18) ^ old) >> 27), rot = (uint32_t)(old >> 59);
    const uint32_t u24 = ((x >> rot) | (x << ((32 - rot) & 31))) >> 8;  // one PCG32 draw
    Prefix kept{0u, 0xffffffffu};  // everything
    if (counted) kept = select_prefix<BOUND_COUNT, CL>(s, row, kept, keep_all ? n : top_k, 0.0f, 0u);
    Prefix pick = kept;  // (its last candidate)
    if (!to_end && !(counted && kept.t < below)) {
        if (top_p < 1.0f) kept = select_prefix<BOUND_SHARE, CL>(s, row, kept, 0u, top_p, 0u);
        pick = select_prefix<BOUND_DRAW, CL>(s, row, kept, 0u, 0.0f, u24);
    }
    cluster_sync<CL>();  // every block has read the state, and the others' shared memory
    if (me == 0 && tid == 0) {
        out[r] = pick.id;
        rng[2 * (size_t)r] = old * 6364136223846793005ULL + inc;
    }
}

// greedy choice per row: first index of the maximum, NaN ignored, 0 when every logit is -inf
__global__ void __launch_bounds__(1024) argmax_rows_kernel(const float *logits, uint32_t n, uint32_t *out) {
    __shared__ Best sh[32];
    const float *v = logits + (size_t)blockIdx.x * n;
    Best b{-INFINITY, 0xffffffffu};
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
        float x = v[i];
        if (x > b.v) b = Best{x, i};
    }
    b = block_best(b, sh);
    if (threadIdx.x == 0) out[blockIdx.x] = (b.v == -INFINITY || b.i == 0xffffffffu) ? 0u : b.i;
}

}  // namespace

// Sampler::sample for `count` rows of n logits at once: row r uses the PCG32 state at rng + 2 r; out[r] receives its token.
static int32_t sample_launch(brasa_cmd *cmd, const float *logits, uint32_t n, uint32_t count, float temperature, uint32_t top_k, float top_p,
                             unsigned long long *rng, uint32_t *out) {
    brasa_ctx *ctx = cmd->ctx;
    int bits = 0;
    while (bits < 32 && (1ull << bits) < n) ++bits;
    // A row in one block saves the cluster barriers and a wave of blocks for every 37 rows; in a cluster it saves seven eighths of the walks over
    // the logits. us for one row, 64 and 200, one block and cluster: 50 logits 25, 39; 27, 84; 31, 254; 8 000 logits 39, 42; 43, 92; 52, 281;
    // 32 768 logits 102, 48; 104, 109; 129, 333. The steps of a long row do not fit one block's memory: a cluster then.
    auto step_bytes = [&](uint32_t blocks) { return (((size_t)n + blocks - 1) / blocks + 15) / 16 * 16; };
    auto fits = [&](uint32_t blocks) { return step_bytes(blocks) + sizeof(SampleShared) + 4096 <= ctx->smem_optin / 2; };  // (two blocks on an SM: many rows at once)
    const uint64_t waves = ((uint64_t)count * SM_CLUSTER + 2 * ctx->sm_count - 1) / (2 * ctx->sm_count);
    const uint32_t blocks = fits(1) && 25.0 + n / 425.0 < waves * (38.0 + n / 2900.0) ? 1 : SM_CLUSTER;
    const auto kernel = blocks == 1 ? sample_kernel<1> : sample_kernel<SM_CLUSTER>;
    const size_t bytes = step_bytes(blocks);
    const bool keep_steps = fits(blocks);
    if (keep_steps) BRASA_TRY(brasa_smem_optin(ctx, (const void *)kernel, bytes));
    kernel<<<count * blocks, SM_THREADS, keep_steps ? bytes : 0, ctx->stream>>>(logits, n, temperature, top_k, top_p, ldexpf(1.0f, 62 - bits), keep_steps, rng,
                                                                                out);
    return brasa_post_launch(cmd, "sample_top_p");
}

int32_t brasa_sample_batched_launch(brasa_cmd *cmd, const float *logits, uint32_t n, uint32_t count, float temperature, uint32_t top_k, float top_p,
                                    unsigned long long *rng, uint32_t *out) {
    brasa_ctx *ctx = cmd->ctx;
    if (count == 0) return BRASA_OK;
    if (temperature <= 0.0f) {
        argmax_rows_kernel<<<count, 1024, 0, ctx->stream>>>(logits, n, out);
        return brasa_post_launch(cmd, "argmax_rows");
    }
    BRASA_REQUIRE(ctx, top_p > 0.0f, "sample_top_p: top_p must be positive");
    return sample_launch(cmd, logits, n, count, temperature, top_k, top_p, rng, out);
}

int32_t brasa_advance_launch(brasa_cmd *cmd, uint32_t *ids, const uint32_t *next, uint32_t *out_ids, uint32_t *out_count, uint32_t out_cap,
                             uint32_t *pos) {
    advance_kernel<<<1, 1, 0, cmd->ctx->stream>>>(ids, next, out_ids, out_count, out_cap, pos);
    return brasa_post_launch(cmd, "advance");
}

int32_t brasa_argmax_launch(brasa_cmd *cmd, const float *logits, uint32_t n, uint32_t *out) {
    brasa_ctx *ctx = cmd->ctx;
    // scratch: 256 partials (8 bytes each) after the counter, inside the context's status block
    if (!ctx->argmax_scratch) {
        BRASA_CUDA(ctx, cudaMalloc(&ctx->argmax_scratch, 4096));
        BRASA_CUDA(ctx, cudaMemset(ctx->argmax_scratch, 0, 4096));
    }
    uint32_t grid = n == 0 ? 1 : std::min<uint32_t>(256, (n + 1023) / 1024);
    uint32_t *counter = (uint32_t *)ctx->argmax_scratch;
    Best *partial = (Best *)((uint8_t *)ctx->argmax_scratch + 64);
    argmax_kernel<<<grid, 256, 0, ctx->stream>>>(logits, n, out, partial, counter);
    return brasa_post_launch(cmd, "argmax");
}

extern "C" {

int32_t brasa_k_argmax(brasa_cmd *cmd, brasa_arg logits, uint32_t n, brasa_arg out_u32) {
    if (!cmd) return BRASA_EINVAL;
    brasa_ctx *ctx = cmd->ctx;
    BRASA_REQUIRE(ctx, arg_fits(logits, (uint64_t)n * 4) && arg_fits(out_u32, 4), "argmax: buffers too small");
    return brasa_argmax_launch(cmd, (const float *)arg_ptr(logits), n, (uint32_t *)arg_ptr(out_u32));
}


int32_t brasa_k_sample_top_p(brasa_cmd *cmd, brasa_arg logits, uint32_t n, float temperature, uint32_t top_k, float top_p, brasa_arg rng_state,
                             brasa_arg out_u32) {
    if (!cmd) return BRASA_EINVAL;
    brasa_ctx *ctx = cmd->ctx;
    BRASA_REQUIRE(ctx, n > 0 && arg_fits(logits, (uint64_t)n * 4) && arg_fits(out_u32, 4) && arg_fits(rng_state, 16) && rng_state.offset % 8 == 0,
                  "sample_top_p: buffers too small or misaligned");
    if (temperature <= 0.0f) return brasa_argmax_launch(cmd, (const float *)arg_ptr(logits), n, (uint32_t *)arg_ptr(out_u32));
    BRASA_REQUIRE(ctx, top_p > 0.0f, "sample_top_p: top_p must be positive");
    return sample_launch(cmd, (const float *)arg_ptr(logits), n, 1, temperature, top_k, top_p, (unsigned long long *)arg_ptr(rng_state), (uint32_t *)arg_ptr(out_u32));
}

int32_t brasa_k_sample_rows(brasa_cmd *cmd, brasa_arg logits, uint32_t n, uint32_t count, float temperature, uint32_t top_k, float top_p,
                            brasa_arg rng_states, brasa_arg scratch, brasa_arg out_u32) {
    if (!cmd) return BRASA_EINVAL;
    brasa_ctx *ctx = cmd->ctx;
    BRASA_REQUIRE(ctx, n > 0 && arg_fits(logits, (uint64_t)count * n * 4) && arg_fits(out_u32, (uint64_t)count * 4) &&
                           arg_fits(rng_states, (uint64_t)count * 16) && arg_fits(scratch, (uint64_t)count * n * 8),
                  "sample_rows: buffers too small");
    BRASA_REQUIRE(ctx, rng_states.offset % 8 == 0 && scratch.offset % 8 == 0, "sample_rows: misaligned");
    return brasa_sample_batched_launch(cmd, (const float *)arg_ptr(logits), n, count, temperature, top_k, top_p,
                                       (unsigned long long *)arg_ptr(rng_states), (uint32_t *)arg_ptr(out_u32));
}

void brasa_pcg32_seed(uint64_t seed, uint64_t state_inc[2]) {
    // Pcg32::new of the reference (sampler.rs:13-20): the state after seeding, and the increment
    uint64_t state = 0, inc = (0xda3e39cb94b95bdbULL << 1) | 1;
    state = state * 6364136223846793005ULL + inc;
    state += seed;
    state = state * 6364136223846793005ULL + inc;
    state_inc[0] = state;
    state_inc[1] = inc;
}

}  // extern "C"
