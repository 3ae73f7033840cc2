// What the two whole-token kernels (decode_token.cu, decode_token_mma.cu) share: the words activations cross blocks in, the bounded waits,
// the blocks' rows, and the attention of one token.
#pragma once
#include "attn_device.cuh"
#include "decode_token.h"
#include "gemv_device.cuh"

namespace brasa_dev {

constexpr int TK_WARPS = 16, TK_THREADS = TK_WARPS * 32;
constexpr uint32_t POLL_LIMIT = 1u << 20;  // polls of an activation word before the wait gives up
constexpr uint32_t EPOCH_SPAN = 1024;      // epochs of one launch; operations + 2 must stay below it
constexpr uint32_t VS_EMPTY = 0xffffffffu;  // an activation word nobody has written in this launch

// Words of a block's reduction area: the warps' sums of x^2 from word 0, each warp's best logit and its index, and the scale of the operation's
// outputs. The scale has a word of its own: every warp reads it behind the rows' barrier, and a warp without rows of the lm_head stores its best
// without another barrier.
constexpr uint32_t RED_BEST = TK_WARPS, RED_INDEX = 2 * TK_WARPS, RED_SCALE = 3 * TK_WARPS, RED_WORDS = RED_SCALE + 4;
static_assert(RED_WORDS % 4 == 0, "what follows the area is copied in 16-byte words");

enum { OP_GEMV = 0, OP_ATTN = 1 };
enum { IN_LL = 0, IN_EMBED = 1 };
enum { EPI_SCALE = 0, EPI_SWIGLU = 1, EPI_RESID = 2, EPI_LOGITS = 3 };

struct Best {
    float v;
    uint32_t i;
};
__device__ __forceinline__ Best better(Best a, Best b) { return (b.v > a.v || (b.v == a.v && b.i < a.i)) ? b : a; }

__device__ __forceinline__ void ll_store(unsigned long long *p, uint32_t bits, uint32_t epoch) {
    unsigned long long w = ((unsigned long long)epoch << 32) | bits;
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(w) : "memory");
}
__device__ __forceinline__ unsigned long long ll_load(const unsigned long long *p) {
    unsigned long long w;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(p) : "memory");
    return w;
}

// An activation word of this launch's copy, and the same word of the other copy emptied for the next launch.
__device__ __forceinline__ void vs_store(uint32_t *cur, uint32_t *alt, uint32_t bits) {
    if (bits == VS_EMPTY) bits = 0x7fffffffu;  // this one NaN pattern means "empty": another NaN takes its place
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(cur), "r"(bits) : "memory");
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(alt), "r"(VS_EMPTY) : "memory");
}
__device__ __forceinline__ uint32_t vs_load(const uint32_t *p) {
    uint32_t w;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(w) : "l"(p) : "memory");
    return w;
}
__device__ __forceinline__ uint4 vs_load4(const uint32_t *p) {  // four words, each indivisible on its own
    uint4 w;
    asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(w.x), "=r"(w.y), "=r"(w.z), "=r"(w.w) : "l"(p) : "memory");
    return w;
}

__device__ __forceinline__ bool vs_there(uint4 w) { return w.x != VS_EMPTY && w.y != VS_EMPTY && w.z != VS_EMPTY && w.w != VS_EMPTY; }

// Rows of block b: logical rows [r0, r1) of `total` (matrices one after another; SwiGLU: the rows of gate, up follows
// the same range), cut into per-matrix segments.
BRASA_HD inline void block_rows(uint32_t total, uint32_t nmat, const uint32_t rows[3], bool swiglu, uint32_t b, uint32_t G, uint32_t &r0,
                                uint32_t &r1, uint32_t first[3], uint32_t nrows[3]) {
    r0 = (uint32_t)((uint64_t)total * b / G);
    r1 = (uint32_t)((uint64_t)total * (b + 1) / G);
    uint32_t base = 0;
    const uint32_t nseg = swiglu ? 2 : nmat;
    for (int i = 0; i < 3; ++i) {
        first[i] = 0;
        nrows[i] = 0;
        if ((uint32_t)i < nseg) {
            if (swiglu) {
                first[i] = r0;
                nrows[i] = r1 - r0;
            } else {
                uint32_t lo = r0 > base ? r0 : base, hi = r1 < base + rows[i] ? r1 : base + rows[i];
                first[i] = lo > base ? lo - base : 0;
                nrows[i] = hi > lo ? hi - lo : 0;
                base += rows[i];
            }
        }
    }
}

// A wait ran out: remember it, stop waiting in this block.
template <class C>
__device__ __forceinline__ void give_up(const C &c, uint32_t code) {
    atomicExch(c.status_word(), code);
    *c.abort_flag() = 1;
}

// Four activation words at once: all loads in flight together, so a wait costs one round trip to L2 when the data is there.
template <class C>
__device__ __forceinline__ void ll_wait4(const C &c, const unsigned long long *p0, const unsigned long long *p1, const unsigned long long *p2,
                                         const unsigned long long *p3, uint32_t epoch, uint32_t out[4]) {
    for (uint32_t it = 0;; ++it) {
        const unsigned long long w0 = ll_load(p0), w1 = ll_load(p1), w2 = ll_load(p2), w3 = ll_load(p3);
        out[0] = (uint32_t)w0; out[1] = (uint32_t)w1; out[2] = (uint32_t)w2; out[3] = (uint32_t)w3;
        const bool ok = (uint32_t)(w0 >> 32) == epoch && (uint32_t)(w1 >> 32) == epoch && (uint32_t)(w2 >> 32) == epoch && (uint32_t)(w3 >> 32) == epoch;
        if (ok || *c.abort_flag()) break;
        if (it >= POLL_LIMIT) {
            give_up(c, 3);
            break;
        }
    }
}

// Four activation words of a vector (attention's q, k, v rows).
template <class C>
__device__ __forceinline__ void vs_wait4(const C &c, const uint32_t *p0, const uint32_t *p1, const uint32_t *p2, const uint32_t *p3, uint32_t out[4]) {
    for (uint32_t it = 0;; ++it) {
        out[0] = vs_load(p0); out[1] = vs_load(p1); out[2] = vs_load(p2); out[3] = vs_load(p3);
        const bool ok = out[0] != VS_EMPTY && out[1] != VS_EMPTY && out[2] != VS_EMPTY && out[3] != VS_EMPTY;
        if (ok || *c.abort_flag()) break;
        if (it >= POLL_LIMIT) {
            give_up(c, 3);
            break;
        }
    }
}

// Bounded wait for a ring slot's bytes. The block's abort flag is looked at only while the wait has to spin, so a slot
// that is already there costs one try. False when the limit ran out.
template <class C>
__device__ __forceinline__ bool slot_wait(const C &c, uint64_t *bar, uint32_t parity) {
    const uint32_t addr = smem_u32(bar);
    for (uint32_t it = 0; it < WAIT_LIMIT; ++it) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(addr), "r"(parity)
            : "memory");
        if (ok) return true;
        if ((it & 15) == 15 && *c.abort_flag()) return true;  // the block has given up: nobody waits any more
    }
    return false;
}

// ---- attention of this token over the cache, new row included ----
// Eight dims of a cached row as they lie there (segment seg of 0..15), and as floats; a q8_0 row's are its codes, whose scale
// goes with the dot product (with the probability) instead.
template <int KV> struct KvSeg;
template <> struct KvSeg<BRASA_KV_F16> {
    uint4 w;
    __device__ __forceinline__ void load(const uint8_t *row, uint32_t seg) { w = __ldcg(reinterpret_cast<const uint4 *>(row) + seg); }
    __device__ __forceinline__ void load_shared(const uint8_t *row, uint32_t seg) { w = reinterpret_cast<const uint4 *>(row)[seg]; }
    __device__ __forceinline__ float scale() const { return 1.0f; }
    __device__ __forceinline__ void four(int i, float v[4]) const {  // values 4 i .. 4 i + 3
        const uint32_t lo = i ? w.z : w.x, hi = i ? w.w : w.y;
        const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&lo)), b = __half22float2(*reinterpret_cast<const __half2 *>(&hi));
        v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
    }
};
template <> struct KvSeg<BRASA_KV_F32> {
    float4 w[2];
    __device__ __forceinline__ void load(const uint8_t *row, uint32_t seg) {
        w[0] = __ldcg(reinterpret_cast<const float4 *>(row) + 2 * seg);
        w[1] = __ldcg(reinterpret_cast<const float4 *>(row) + 2 * seg + 1);
    }
    __device__ __forceinline__ void load_shared(const uint8_t *row, uint32_t seg) {
        w[0] = reinterpret_cast<const float4 *>(row)[2 * seg];
        w[1] = reinterpret_cast<const float4 *>(row)[2 * seg + 1];
    }
    __device__ __forceinline__ float scale() const { return 1.0f; }
    __device__ __forceinline__ void four(int i, float v[4]) const { v[0] = w[i].x; v[1] = w[i].y; v[2] = w[i].z; v[3] = w[i].w; }
};
template <> struct KvSeg<BRASA_KV_Q8_0> {
    uint2 w;
    unsigned short d;
    __device__ __forceinline__ void load(const uint8_t *row, uint32_t seg) {
        w = __ldcg(reinterpret_cast<const uint2 *>(row) + seg);
        d = __ldcg(reinterpret_cast<const unsigned short *>(row + 128) + (seg >> 2));
    }
    __device__ __forceinline__ void load_shared(const uint8_t *row, uint32_t seg) {
        w = reinterpret_cast<const uint2 *>(row)[seg];
        d = reinterpret_cast<const unsigned short *>(row + 128)[seg >> 2];
    }
    __device__ __forceinline__ float scale() const { return __half2float(__ushort_as_half(d)); }
    __device__ __forceinline__ void four(int i, float v[4]) const {
        const uint32_t c = (i ? w.y : w.x) ^ 0x80808080u;  // code + 128
        // the float 2^23 + byte, minus 2^23 + 128: exact, and two instructions where a conversion takes a quarter-rate one
        v[0] = __uint_as_float(__byte_perm(c, 0x4B000000u, 0x7440)) - 8388736.0f;
        v[1] = __uint_as_float(__byte_perm(c, 0x4B000000u, 0x7441)) - 8388736.0f;
        v[2] = __uint_as_float(__byte_perm(c, 0x4B000000u, 0x7442)) - 8388736.0f;
        v[3] = __uint_as_float(__byte_perm(c, 0x4B000000u, 0x7443)) - 8388736.0f;
    }
};

// What the attention needs of the block: an area in shared memory, this launch's copy of the vectors.
struct AttnCtx {
    uint8_t *xfb;  // ATTN_AREA_BYTES
    volatile uint32_t *s_abort;
    uint32_t *status;
    uint32_t G, b, pos, par_cur, par_alt;
    __device__ __forceinline__ uint32_t *status_word() const { return status; }
    __device__ __forceinline__ volatile uint32_t *abort_flag() const { return s_abort; }
};
constexpr size_t ATTN_AREA_BYTES = (size_t)(TK_WARPS * (512 + 8) + 8 * 128) * 4 + 2 * 512;  // see attention_op

// Every warp walks keys of its own, four at a time, with a running maximum, sum and output in registers: sixteen lanes hold two keys, a
// lane 8 dims of them for four heads. Nothing is shared until a group of keys is done, so an item has two block barriers where a tile
// form (K and V tiles in shared memory, 64 keys between barriers) had four per 64 keys, and the next keys' rows are on their
// way while these are worked on. The bound is the multiply-adds (1 024 per key for four heads, 512 lanes). us a
// token of eight layers of 2 560 with 32 heads, the tile form's in brackets, behind 512 and 16 384 keys: f16 cache, 8 KV heads 238 (244), 366
// (506); 32 KV heads 265 (291), 763 (1 401); 4 KV heads, whose eight heads walk the keys twice, 256 (258), 366 (430); q8_0, 8 KV heads 242
// (249), 362 (571); 4 KV heads 259 (262), 373 (460).
template <int KV, class Op>
__device__ __forceinline__ void attention_op(const AttnCtx &c, const Op &op, uint32_t oi, uint32_t epoch, uint32_t heads,
                                          uint32_t kv_heads, uint32_t max_chunks, const float *cos_t, const float *sin_t,
                                          unsigned long long *partials, float attn_scale) {
    constexpr int RB = KvRow<KV>::BYTES;
    constexpr uint32_t C = KV == BRASA_KV_F32 ? 32 : 64;  // keys a group is cut by
    constexpr bool AHEAD = KV != BRASA_KV_F32;            // the next keys' rows fit the registers
    constexpr int QS_HEAD = 128;  // q of a head in shared memory: the first four values of every segment, then the other four
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t Gq = heads / kv_heads, pos = c.pos;
    const uint32_t lk = pos + 1, nchunks = (lk + C - 1) / C;
    float *osum = reinterpret_cast<float *>(c.xfb);               // [16 warps][4 heads][128]
    float *wm = osum + TK_WARPS * 512, *wl = wm + TK_WARPS * 4;   // [16 warps][4 heads]: running maximum and sum
    float *qs = wl + TK_WARPS * 4;                                // [8][QS_HEAD]
    uint8_t *krow = reinterpret_cast<uint8_t *>(qs + 8 * QS_HEAD), *vrow = krow + 512;  // this token's rows, in the cache's type
    const uint32_t kgrp = lane >> 4, seg = lane & 15;
    // A work item is (kv head, group of consecutive chunks): a dozen or so partial results per head to merge, however long the cache
    const uint32_t groups_max = max(1u, c.G / kv_heads);
    const uint32_t cpg = (nchunks + groups_max - 1) / groups_max, ngroups = (nchunks + cpg - 1) / cpg;
    const uint32_t nitems = kv_heads * ngroups;
#pragma unroll 1
    for (uint32_t item = c.b; item < nitems; item += c.G) {
        const uint32_t kh = item / ngroups, gi = item - kh * ngroups;
        const uint32_t k_lo = gi * cpg * C, k_hi = min(lk, k_lo + cpg * C);
        const uint32_t cached = min(k_hi, pos);  // the new row is not in the cache yet
        const uint8_t *kbase = op.kc + (size_t)kh * RB, *vbase = op.vc + (size_t)kh * RB;
        const size_t pitch = (size_t)kv_heads * RB;
#pragma unroll 1
        for (uint32_t g0 = 0; g0 < Gq; g0 += 4) {
            KvSeg<KV> kw[2]{}, vw[2]{};
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const uint32_t key = k_lo + 4 * warp + 2 * u + kgrp;
                if (key < cached) {  // (does not wait for this token's q)
                    kw[u].load(kbase + key * pitch, seg);
                    vw[u].load(vbase + key * pitch, seg);
                }
            }
            if (g0 == 0 && ((uint32_t)warp < Gq || ((uint32_t)warp < Gq + 2 && k_hi == lk))) {
                // warps 0 .. Gq-1: a query head (once per item); warp Gq: the new key row; warp Gq + 1: the new value row
                const uint32_t g = warp;
                const uint32_t *src = op.in + c.par_cur + (g < Gq ? (size_t)(kh * Gq + g) * 128 : (size_t)(heads + (g - Gq) * kv_heads + kh) * 128);
                float xv[4], y[4], wv[4], cs[2], sn[2];
                {   // what does not depend on this token's q, k, v first: norm weight, cos and sin of this position
                    const float *nw = g < Gq ? op.q_norm : op.k_norm;
                    for (int j = 0; j < 4; ++j) wv[j] = nw[lane + 32 * j];
                    for (int j = 0; j < 2; ++j) {
                        cs[j] = cos_t[(size_t)pos * 64 + lane + 32 * j];
                        sn[j] = sin_t[(size_t)pos * 64 + lane + 32 * j];
                    }
                    uint32_t raw[4];
                    vs_wait4(c, src + lane, src + lane + 32, src + lane + 64, src + lane + 96, raw);
                    for (int j = 0; j < 4; ++j) xv[j] = __uint_as_float(raw[j]);
                }
                if (g <= Gq) norm_rope_regs(xv, wv, cs, sn, op.eps, y);
                if (g < Gq) {
                    for (int j = 0; j < 4; ++j) {
                        const uint32_t e = lane + 32 * j;
                        qs[g * QS_HEAD + ((e >> 2) & 1) * 64 + (e >> 3) * 4 + (e & 3)] = y[j];
                    }
                } else {
                    const size_t grow = ((size_t)pos * kv_heads + kh) * RB;
                    if (g == Gq) put_row<KV>(op.kc + grow, krow, y, lane);
                    else put_row<KV>(op.vc + grow, vrow, xv, lane);
                }
            }
            __syncthreads();
            const float *q0 = qs + g0 * QS_HEAD + 4 * seg;
            float acc[4][8];
#pragma unroll
            for (int g = 0; g < 4; ++g)
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[g][i] = 0.0f;
            float m = -INFINITY, l = 0.0f;  // of head g0 + (seg / 2) % 4, over this half warp's keys
#pragma unroll 1
            for (uint32_t k0 = k_lo + 4 * warp; k0 < k_hi; k0 += 4 * TK_WARPS) {
                const uint32_t key0 = k0 + kgrp, next0 = key0 + 4 * TK_WARPS;  // this half warp's keys: key0, key0 + 2
                KvSeg<KV> kn[2]{}, vn[2]{};
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    if (AHEAD && next0 + 2 * u < cached) {
                        kn[u].load(kbase + (next0 + 2 * u) * pitch, seg);
                        vn[u].load(vbase + (next0 + 2 * u) * pitch, seg);
                    }
                    if (key0 + 2 * u == pos && pos < k_hi) {
                        kw[u].load_shared(krow, seg);
                        vw[u].load_shared(vrow, seg);
                    }
                }
                float s[2][4] = {};
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    float kf[2][4];
                    kw[0].four(i, kf[0]);
                    kw[1].four(i, kf[1]);
#pragma unroll
                    for (int g = 0; g < 4; ++g) {
                        const float4 qa = *reinterpret_cast<const float4 *>(q0 + g * QS_HEAD + 64 * i);
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            s[u][g] = fmaf(qa.x, kf[u][0], s[u][g]); s[u][g] = fmaf(qa.y, kf[u][1], s[u][g]);
                            s[u][g] = fmaf(qa.z, kf[u][2], s[u][g]); s[u][g] = fmaf(qa.w, kf[u][3], s[u][g]);
                        }
                    }
                }
                if (KV == BRASA_KV_Q8_0) {
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const float d = kw[u].scale();
#pragma unroll
                        for (int g = 0; g < 4; ++g) s[u][g] *= d;
                    }
                }
                // the sixteen lanes' shares meet: lane seg ends with key key0 + 2 (seg / 8), head (seg / 2) % 4 (each twice)
                const uint32_t mu = seg >> 3;
                float b[4];
#pragma unroll
                for (int g = 0; g < 4; ++g) {
                    b[g] = mu ? s[1][g] : s[0][g];
                    b[g] += __shfl_xor_sync(0xffffffffu, mu ? s[0][g] : s[1][g], 8);
                }
                float a0 = (seg & 4) ? b[2] : b[0], a1 = (seg & 4) ? b[3] : b[1];
                a0 += __shfl_xor_sync(0xffffffffu, (seg & 4) ? b[0] : b[2], 4);
                a1 += __shfl_xor_sync(0xffffffffu, (seg & 4) ? b[1] : b[3], 4);
                float sc = (seg & 2) ? a1 : a0;
                sc += __shfl_xor_sync(0xffffffffu, (seg & 2) ? a0 : a1, 2);
                sc += __shfl_xor_sync(0xffffffffu, sc, 1);
                const bool seen = key0 + 2 * mu < k_hi;
                sc = seen ? sc * attn_scale : -INFINITY;
                const float mn = fmaxf(m, fmaxf(sc, __shfl_xor_sync(0xffffffffu, sc, 8)));
                const float keep = m == -INFINITY ? 0.0f : expf(m - mn), pr = seen ? expf(sc - mn) : 0.0f;
                const bool moved = mn != m;
                l = l * keep + pr;
                m = mn;
                if (__any_sync(0xffffffffu, moved)) {
#pragma unroll
                    for (int g = 0; g < 4; ++g) {
                        const float kg = __shfl_sync(0xffffffffu, keep, (lane & 16) + 2 * g);
#pragma unroll
                        for (int i = 0; i < 8; ++i) acc[g][i] *= kg;
                    }
                }
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    float pg[4];
#pragma unroll
                    for (int g = 0; g < 4; ++g) {
                        pg[g] = __shfl_sync(0xffffffffu, pr, (lane & 16) + 8 * u + 2 * g);
                        if (KV == BRASA_KV_Q8_0) pg[g] *= vw[u].scale();
                    }
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        float vf[4];
                        vw[u].four(i, vf);
#pragma unroll
                        for (int g = 0; g < 4; ++g)
#pragma unroll
                            for (int e = 0; e < 4; ++e) acc[g][4 * i + e] = fmaf(pg[g], vf[e], acc[g][4 * i + e]);
                    }
                }
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    if (AHEAD) {
                        kw[u] = kn[u];
                        vw[u] = vn[u];
                    } else if (next0 + 2 * u < cached) {
                        kw[u].load(kbase + (next0 + 2 * u) * pitch, seg);
                        vw[u].load(vbase + (next0 + 2 * u) * pitch, seg);
                    }
                }
            }
            {   // the warp's halves meet: lane (kgrp, seg) ends with dims 8 seg .. of heads g0 + 2 kgrp and the next
                l += __shfl_xor_sync(0xffffffffu, l, 8);
                const float mw = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 16)), f = m == -INFINITY ? 0.0f : expf(m - mw);
                l *= f;
                l += __shfl_xor_sync(0xffffffffu, l, 16);
#pragma unroll
                for (int g = 0; g < 4; ++g) {
                    const float fg = __shfl_sync(0xffffffffu, f, (lane & 16) + 2 * g);
#pragma unroll
                    for (int i = 0; i < 8; ++i) acc[g][i] *= fg;
                }
#pragma unroll
                for (int g = 0; g < 2; ++g) {
                    float4 *dst = reinterpret_cast<float4 *>(osum + (warp * 4 + 2 * kgrp + g) * 128 + 8 * seg);
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float mine = kgrp ? acc[2 + g][i] : acc[g][i];
                        acc[g][i] = mine + __shfl_xor_sync(0xffffffffu, kgrp ? acc[g][i] : acc[2 + g][i], 16);
                    }
                    dst[0] = make_float4(acc[g][0], acc[g][1], acc[g][2], acc[g][3]);
                    dst[1] = make_float4(acc[g][4], acc[g][5], acc[g][6], acc[g][7]);
                }
                if (kgrp == 0 && (seg & 9) == 0) {
                    wm[warp * 4 + (seg >> 1)] = mw;
                    wl[warp * 4 + (seg >> 1)] = l;
                }
            }
            __syncthreads();
            {   // the warps meet: thread = (head, dim)
                const uint32_t hd = tid >> 7, d = tid & 127;
                const float mw = wm[(lane & 15) * 4 + hd];
                float M = mw;
                for (int o = 8; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
                const float f = mw == -INFINITY ? 0.0f : expf(mw - M);
                float L = wl[(lane & 15) * 4 + hd] * f;
                for (int o = 8; o > 0; o >>= 1) L += __shfl_xor_sync(0xffffffffu, L, o);
                float a = 0.0f;
#pragma unroll
                for (int w = 0; w < TK_WARPS; ++w) a = fmaf(osum[(w * 4 + hd) * 128 + d], __shfl_sync(0xffffffffu, f, w), a);
                if (g0 + hd < Gq) {
                    const uint32_t head = kh * Gq + g0 + hd;
                    if (ngroups == 1) {
                        uint32_t *o0 = op.out + (size_t)head * 128 + d;
                        vs_store(o0 + c.par_cur, o0 + c.par_alt, __float_as_uint(a / L));
                    } else {
                        unsigned long long *pp = partials + ((size_t)head * max_chunks + gi) * 130;
                        ll_store(pp + 2 + d, __float_as_uint(a), epoch);
                        if (d == 0) { ll_store(pp, __float_as_uint(M), epoch); ll_store(pp + 1, __float_as_uint(L), epoch); }
                    }
                }
            }
            if (g0 + 4 < Gq || item + c.G < nitems) __syncthreads();  // the next pass writes the same shared memory
        }
    }
    if (ngroups > 1) {
        // merge the groups of a head; heads go to the blocks at the far end of the grid (the work items start at block 0)
#pragma unroll 1
        for (uint32_t head = c.G - 1 - c.b; head < heads; head += c.G) {
            const unsigned long long *pp = partials + (size_t)head * max_chunks * 130;
            // thread (d, cg) merges the chunks cg, cg + 4, .. of output element d on its own (running maximum), four
            // chunks per round trip with m, l and the accumulator in flight together; the four classes meet below
            const uint32_t d = tid & 127, cg = tid >> 7;
            float M = -INFINITY, L = 0.0f, a = 0.0f;
#pragma unroll 1
            for (uint32_t ch = cg; ch < ngroups; ch += 16) {
                uint32_t cc[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) cc[j] = min(ch + 4 * j, ngroups - 1);
                unsigned long long w[12];
                for (uint32_t it = 0;; ++it) {
                    uint32_t bad = 0;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const unsigned long long *q = pp + (size_t)cc[j] * 130;
                        w[3 * j] = ll_load(q);
                        w[3 * j + 1] = ll_load(q + 1);
                        w[3 * j + 2] = ll_load(q + 2 + d);
                    }
#pragma unroll
                    for (int j = 0; j < 12; ++j) bad |= (uint32_t)(w[j] >> 32) ^ epoch;
                    if (bad == 0 || *c.abort_flag()) break;
                    if (it >= POLL_LIMIT) {
                        give_up(c, 3);
                        break;
                    }
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (ch + 4 * j < ngroups) {
                        const float mc = __uint_as_float((uint32_t)w[3 * j]), lc = __uint_as_float((uint32_t)w[3 * j + 1]);
                        const float ac = __uint_as_float((uint32_t)w[3 * j + 2]);
                        const float Mn = fmaxf(M, mc), so = expf(M - Mn), sn = expf(mc - Mn);  // M = -inf at first: so = 0
                        L = L * so + lc * sn;
                        a = a * so + ac * sn;
                        M = Mn;
                    }
                }
            }
            // classes with no chunk keep M = -inf, L = a = 0
            qs[cg * 128 + d] = a;
            if (d == 0) { qs[512 + cg] = L; qs[516 + cg] = M; }
            __syncthreads();
            if (tid < 128) {
                const float Mt = fmaxf(fmaxf(qs[516], qs[517]), fmaxf(qs[518], qs[519]));
                float A = 0.0f, Lt = 0.0f;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float wj = qs[516 + j] == -INFINITY ? 0.0f : expf(qs[516 + j] - Mt);
                    A = fmaf(qs[j * 128 + d], wj, A);
                    Lt = fmaf(qs[512 + j], wj, Lt);
                }
                vs_store(op.out + c.par_cur + (size_t)head * 128 + d, op.out + c.par_alt + (size_t)head * 128 + d, __float_as_uint(A / Lt));
            }
            __syncthreads();
        }
    }
}

inline uint32_t attn_chunk(int32_t kv) { return kv == BRASA_KV_F32 ? 32u : 64u; }

}  // namespace brasa_dev
