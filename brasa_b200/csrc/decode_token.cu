// One decode token as ONE persistent kernel (the token loop of crates/models/src/qwen3.rs:551-831 for a single
// token, plus the greedy choice of crates/runtime/src/sampler.rs:148-170).
//
// A token is a chain of about 180 small dependent operations (per layer: QKV GEMV, attention, o_proj GEMV, gate/up
// GEMV, down GEMV). Launched as separate kernels each link costs about 10 us on B200 although its bytes need 1-4 us,
// so the chain runs here inside one cooperative launch, one block per SM:
//   * Weights never wait. Every block owns the same share of rows of every matrix, known when the model is loaded,
//     so its weight traffic is a fixed list of byte ranges (slots). They stream through a shared-memory ring with
//     bulk async copies; the warp that is last to finish with a slot starts the copy that reuses it, across
//     operation boundaries. HBM keeps working while the blocks exchange activations.
//   * Activations cross blocks without barriers. Every operation has its own output vector in L2, twice (launches
//     alternate between the two copies). A word holds either the float or the bit pattern VS_EMPTY, a NaN no
//     arithmetic produces; a consumer polls the words it needs until none is empty. A 4-byte store is indivisible, so
//     no fence, flag or grid barrier is needed, and one round trip to L2 both synchronises and delivers the data.
//     The thread that writes a word of this launch's copy also empties the same word of the other copy, which the
//     launch before wrote and read and the next launch will fill: the end of the kernel orders that store before
//     every load of the next launch, so inside one launch a word changes exactly once, from empty to its value.
//     (Attention partials, the argmax candidates and the words that cross GPUs are 8-byte {float, epoch} words,
//     valid when they carry the epoch of the producing operation of this launch.)
//   * Every poll and every mbarrier wait is bounded. A wait that runs out sets the context's status word and a
//     block-wide flag after which the block stops waiting and runs to its end; the host reports BRASA_ETIMEOUT.
// decode_token_mma.cu takes the models whose products are worth integer tensor instructions (f16 and q8_0 caches, one GPU, hidden sizes
// of 768 to 3 072; brasa_token_mma_takes); this kernel has the narrower ones (bound by the exchanges either way), the wider ones (32B: rows that a tile
// of sixteen cannot hold in a slot), f32 caches and the shards of a tensor-parallel model.
// GEMV arithmetic, x conversion and epilogues are those of gemv.cu (with two byte planes of x for f16 and q8_0 caches, three there and
// for f32 caches); attention works on 64-key
// chunks (32 for an f32 cache) shared out over the blocks and is merged per head by the blocks at the far end of
// the grid.
#include <stdlib.h>

#include <memory>

#include "decode_token_mma.h"
#include "token_device.cuh"

using namespace brasa_dev;

namespace {

constexpr uint32_t SLOT_CAP = 24 * 1024;   // bytes of one ring slot
constexpr uint32_t DONE_PARITY = 1u << 31; // of a slot's count of warps that are done with it: whether it has been refilled an odd number of times
constexpr int R = 2;                       // rows a warp works on at a time
constexpr int NMAX = 5;                    // half blocks of x a lane keeps per column slice

struct SlotDesc {
    const uint8_t *src;
    uint32_t bytes;
    uint32_t part;  // 0: the bytes as they lie; else columns of a half row | rows << 16 | half << 24 (see issue_slot)
};

struct TokOp {
    uint32_t type, qtype, cols, nmat;
    uint32_t rows[3], total_rows;
    uint32_t epilogue, scaled, log2S, nact;
    uint32_t in_kind, in_op, save_resid, next_cols;  // next_cols: length of next_normw
    float eps;
    uint32_t xchg;  // tensor parallel: 1 + index of this residual add among the token's exchanges (0: no exchange)
    uint32_t fast;  // every lane's half blocks before its last iteration lie inside the row (see gemv_rows)
    uint32_t halves;  // 2: rows too wide for a slot and a lane's registers, taken as two halves of `cols` columns one after the other
    const uint8_t *w[3];
    const float *normw;
    const uint32_t *in;  // first copy; the second one lies TokParams::par_words further
    uint32_t *out;
    const float *q_norm, *k_norm;
    uint8_t *kc, *vc;
    const float *next_normw;  // norm weight of the operation after this one (null: none): staged in shared memory meanwhile
    uint64_t pad2;
};
constexpr uint32_t OP_WORDS = sizeof(TokOp) / 4;
constexpr uint32_t OPS_WORDS = OP_WORDS + 4;  // in shared memory the block's row counts follow the operation
static_assert(sizeof(TokOp) % 16 == 0, "TokOp is copied as words");

struct TokParams {
    const TokOp *ops;
    uint32_t nops;
    const SlotDesc *slots;
    const uint32_t *slot_begin;  // [grid + 1]
    const uint4 *block_ops;      // [nops][grid]: first output row, rows of segments 0 | 1 << 16, rows of segment 2, -
    uint32_t nslot, xf_bytes, part_floats, resid_floats, sdesc_n, nw_floats;
    uint32_t par_words;  // words of one copy of the activation vectors
    uint32_t *state, *ids, *next_id, *out_ids;
    uint32_t out_cap;
    const uint8_t *embed;
    uint32_t vocab, hidden, heads, kv_heads, max_chunks;
    const float *cos_t, *sin_t;
    float *logits;
    unsigned long long *cand;      // [grid][2]: best logit, its index
    unsigned long long *partials;  // [heads][max_chunks][130]
    float attn_scale;
    uint32_t *status;
    unsigned long long *trace;  // optional: block 0 stamps the phases of 16 operations from trace_op on (debugging aid)
    uint32_t trace_op;
    // tensor parallel (tp_world > 1): every rank's exchange area as seen from here, see brasa_tp_token_area
    uint32_t tp_world, tp_rank, tp_row0, tp_poll_limit;
    unsigned long long tp_stride;
    unsigned long long *tp_peer[BRASA_TP_MAX_RANKS];
};

// Words that cross GPUs (a peer's store into this rank's exchange area over NVLink): system scope.
__device__ __forceinline__ void xg_store(unsigned long long *p, uint32_t bits, uint32_t epoch) {
    unsigned long long w = ((unsigned long long)epoch << 32) | bits;
    asm volatile("st.relaxed.sys.global.u64 [%0], %1;" ::"l"(p), "l"(w) : "memory");
}
__device__ __forceinline__ unsigned long long xg_load(const unsigned long long *p) {
    unsigned long long w;
    asm volatile("ld.relaxed.sys.global.u64 %0, [%1];" : "=l"(w) : "l"(p) : "memory");
    return w;
}

// 16 values of row `row` of a tiled q6_0 table as the four quads of half block hbi (embed_kernel's arithmetic).
__device__ __forceinline__ void embed_half_block(const uint8_t *table, uint32_t row, uint32_t cols, uint32_t hbi, float4 q[4]) {
    const uint8_t *r = table + (size_t)row * tiled_row_bytes(BRASA_Q6_0, cols);
    const uint2 codes = *reinterpret_cast<const uint2 *>(r + hbi * 8);
    const uint32_t hb = *reinterpret_cast<const uint32_t *>(r + tiled_hi_off(cols) + hbi * 4);
    const float d = __half2float(*reinterpret_cast<const __half *>(r + tiled_scale_off(BRASA_Q6_0, cols) + (hbi >> 1) * 2));
    uint32_t a[4];
    a[0] = lop_and_or(hb, 0x30303030u, codes.x & 0x0F0F0F0Fu);
    a[1] = lop_and_or(hb >> 2, 0x30303030u, (codes.x >> 4) & 0x0F0F0F0Fu);
    a[2] = lop_and_or(hb << 2, 0x30303030u, codes.y & 0x0F0F0F0Fu);
    a[3] = lop_and_or(hb << 4, 0x30303030u, (codes.y >> 4) & 0x0F0F0F0Fu);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        q[j].x = d * (float)((int)(a[j] & 255u) - 32);
        q[j].y = d * (float)((int)((a[j] >> 8) & 255u) - 32);
        q[j].z = d * (float)((int)((a[j] >> 16) & 255u) - 32);
        q[j].w = d * (float)((int)(a[j] >> 24) - 32);
    }
}

#ifdef BRASA_TRACE_BUILD
#define TRACEB(i) do { if (c.trace && threadIdx.x == 0 && c.oi >= c.trace_op && c.oi < c.trace_op + 5) c.trace[512 + ((c.oi - c.trace_op) * 160 + c.b) * 4 + (i)] = gtime(); } while (0)
#define TRACE(i) do { if (c.trace && c.b == 0 && threadIdx.x == 0 && c.oi >= c.trace_op && c.oi < c.trace_op + 16) c.trace[16 + (c.oi - c.trace_op) * 16 + (i)] = (unsigned long long)clock64(); } while (0)
#else
#define TRACE(i) do { } while (0)
#define TRACEB(i) do { } while (0)
#endif

// What the phases of an operation share. The phase functions are inlined: with 227 KB of shared memory in use the
// L1 cache is a few KB, so a stack frame (calls, spills) costs a trip to L2 per access.
struct TokCtx {
    uint8_t *ring, *xfb;
    float *part, *resid, *red, *nwbuf;
    uint4 *sdesc;
    uint64_t *full;
    uint32_t *done;
    volatile uint32_t *s_abort;
    const uint4 *myslots;
    uint32_t *status;
    unsigned long long *trace;
    uint32_t trace_op, my_slots, nslot, G, b, pos, seq, token, h0, hn;
    uint32_t par_cur, par_alt;  // word offsets of this launch's copy of the activation vectors and of the other one
    uint32_t oi;  // current operation (trace builds)
    __device__ __forceinline__ uint32_t *status_word() const { return status; }
    __device__ __forceinline__ volatile uint32_t *abort_flag() const { return s_abort; }
};

// This warp's place in the block's slot list: next list index, its ring slot, that use's phase parity.
struct WarpRing {
    uint32_t kk, rs, rph;
};

// a slot descriptor {address lo, address hi, bytes, part} -> ring[s]
__device__ __forceinline__ void issue_slot(const TokCtx &c, uint4 d, uint32_t s) {
    const uint8_t *src = reinterpret_cast<const uint8_t *>(((unsigned long long)d.y << 32) | d.x);
    uint8_t *dst = c.ring + (size_t)s * SLOT_CAP;
    mbar_expect_tx(&c.full[s], d.z);
    if (d.w == 0) {
        bulk_g2s(dst, src, d.z, &c.full[s]);
        return;
    }
    // half rows: a row's codes and scales of these columns, laid together as a row of that many columns is
    const uint32_t cols = d.w & 0xffffu, n = (d.w >> 16) & 0xffu, half = d.w >> 24, cb = cols / 2, sb = cols / 16;
#pragma unroll 1
    for (uint32_t r = 0; r < n; ++r, src += 2 * (cb + sb), dst += cb + sb) {
        bulk_g2s(dst, src + half * cb, cb, &c.full[s]);
        bulk_g2s(dst + cb, src + 2 * cb + half * sb, sb, &c.full[s]);
    }
}

// ---- GEMV, phase 1: wait for the input, fold the norm weight, convert to fixed point. A thread takes one quad of four
// values at a time (quads t, t + 512, ..), so that the whole block polls at once; the four lanes of a half block share
// its largest magnitude and its integer sum by shuffles and each writes its own words of the record (the record
// x_half_block_to_fixed builds, same arithmetic). Returns the thread's share of sum x^2. (Asking for all of a thread's
// quads at once measured 5 % slower over the token than one quad after the other: polls and weights share the L2.)

// element index of quad qi: the quads of a half block start at +0, +16, +4, +20
__device__ __forceinline__ uint32_t quad_elem(uint32_t qi) {
    const uint32_t hbi = qi >> 2, j = qi & 3;
    return (hbi >> 1) * 32 + 8 * (hbi & 1) + 16 * (j & 1) + 2 * (j & 2);
}

template <int P>
__device__ __forceinline__ void quad_to_fixed(const TokCtx &c, const TokOp &op, uint32_t *xw, uint32_t qi, float4 v, float &ssq) {
    constexpr uint32_t BITS = P == 3 ? 22 : 16;
    const uint32_t hbi = qi >> 2, j = qi & 3, e = quad_elem(qi);
    ssq = fmaf(v.x, v.x, ssq); ssq = fmaf(v.y, v.y, ssq); ssq = fmaf(v.z, v.z, ssq); ssq = fmaf(v.w, v.w, ssq);
    if (op.save_resid) {  // this vector is the residual a later epilogue adds: keep this block's rows
        const uint32_t r = e - c.h0;  // wraps for rows before h0
        if (r + 0 < c.hn) c.resid[r + 0] = v.x;
        if (r + 1 < c.hn) c.resid[r + 1] = v.y;
        if (r + 2 < c.hn) c.resid[r + 2] = v.z;
        if (r + 3 < c.hn) c.resid[r + 3] = v.w;
    }
    if (op.normw) {
        const float4 nw = *reinterpret_cast<const float4 *>(c.nwbuf + e);
        v.x *= nw.x; v.y *= nw.y; v.z *= nw.z; v.w *= nw.w;
    }
    float amax = fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
    // step = 2^(exponent(amax) - (BITS - 2)); zero (or denormal) groups get step 0; infinities travel in the step
    const uint32_t ebits = __float_as_uint(amax) & 0x7F800000u;
    const bool live = ebits > ((BITS - 1) << 23) && ebits < 0x7F800000u;
    const float step = live ? __uint_as_float(ebits - ((BITS - 2) << 23)) : (ebits == 0x7F800000u ? amax : 0.0f);
    const float inv = live ? __uint_as_float((254u << 23) - (ebits - ((BITS - 2) << 23))) : 0.0f;  // 1 / step, exact
    int X[4] = {__float2int_rn(v.x * inv), __float2int_rn(v.y * inv), __float2int_rn(v.z * inv), __float2int_rn(v.w * inv)};
    if (P == 2) {  // a value that rounds up to 2^15 stays inside the signed top byte
#pragma unroll
        for (int k = 0; k < 4; ++k) X[k] = min(X[k], 32767);
    }
    int total = X[0] + X[1] + X[2] + X[3];
    total += __shfl_xor_sync(0xffffffffu, total, 1);
    total += __shfl_xor_sync(0xffffffffu, total, 2);
    // byte planes of the four integers: byte k of every X gathered into one word
    const uint32_t lo01 = __byte_perm(X[0], X[1], 0x5140), lo23 = __byte_perm(X[2], X[3], 0x5140);
    const uint32_t w0 = __byte_perm(lo01, lo23, 0x5410), w1 = __byte_perm(lo01, lo23, 0x7632);
    if (P == 3) {
        const uint32_t hi01 = __byte_perm(X[0], X[1], 0x7362), hi23 = __byte_perm(X[2], X[3], 0x7362);
        const uint32_t w2 = __byte_perm(hi01, hi23, 0x5410);
        const uint32_t sw = (hbi >> 1) & 3;  // record words 3j .. 3j + 2; 16-byte chunk n of a record lies at n ^ sw
        const uint32_t i0 = 3 * j, i1 = 3 * j + 1, i2 = 3 * j + 2;
        xw[(hbi * 4 + ((i0 >> 2) ^ sw)) * 4 + (i0 & 3)] = w0;
        xw[(hbi * 4 + ((i1 >> 2) ^ sw)) * 4 + (i1 & 3)] = w1;
        xw[(hbi * 4 + ((i2 >> 2) ^ sw)) * 4 + (i2 & 3)] = w2;
        if (j == 0) *reinterpret_cast<uint4 *>(xw + (hbi * 4 + (3 ^ sw)) * 4) = make_uint4((uint32_t)total, __float_as_uint(step), 0, 0);
    } else {
        *reinterpret_cast<uint2 *>(xw + hbi * 12 + 2 * j) = make_uint2(w0, w1);
        if (j == 0) *reinterpret_cast<uint4 *>(xw + hbi * 12 + 8) = make_uint4((uint32_t)total, __float_as_uint(step), 0, 0);
    }
}

template <int P>
__device__ __forceinline__ float gemv_input(const TokCtx &c, const TokOp &op, const uint8_t *embed, uint32_t vocab, uint32_t half) {
    const int tid = threadIdx.x;
    const uint32_t cols = op.cols, nq = cols / 4;  // a multiple of 64: a warp is inside or outside as a whole
    uint32_t *xw = reinterpret_cast<uint32_t *>(c.xfb);
    const uint32_t *in = op.in + c.par_cur + half * cols;
    float ssq = 0.0f;
    if (op.in_kind == IN_EMBED) {
#pragma unroll 1
        for (uint32_t qi = tid; qi < nq; qi += TK_THREADS) {
            const uint32_t j = qi & 3;
            float4 q[4];
            if (c.token < vocab) embed_half_block(embed, c.token, cols, qi >> 2, q);
            else q[0] = q[1] = q[2] = q[3] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            quad_to_fixed<P>(c, op, xw, qi, j == 0 ? q[0] : (j == 1 ? q[1] : (j == 2 ? q[2] : q[3])), ssq);
        }
        return ssq;
    }
#pragma unroll 1
    for (uint32_t qi = tid; qi < nq; qi += 2 * TK_THREADS) {  // two quads of the thread in flight: half the round trips
        const uint32_t qj = qi + TK_THREADS;
        const bool two = qj < nq;
        uint4 w0, w1 = make_uint4(0, 0, 0, 0);
        for (uint32_t it = 0;; ++it) {
            w0 = vs_load4(in + quad_elem(qi));
            if (two) w1 = vs_load4(in + quad_elem(qj));
            const bool ok = w0.x != VS_EMPTY && w0.y != VS_EMPTY && w0.z != VS_EMPTY && w0.w != VS_EMPTY &&
                            w1.x != VS_EMPTY && w1.y != VS_EMPTY && w1.z != VS_EMPTY && w1.w != VS_EMPTY;
            if (ok || *c.abort_flag()) break;
            if (it >= POLL_LIMIT) {
                give_up(c, 3);
                break;
            }
        }
        TRACE(2);
        quad_to_fixed<P>(c, op, xw, qi, make_float4(__uint_as_float(w0.x), __uint_as_float(w0.y), __uint_as_float(w0.z), __uint_as_float(w0.w)), ssq);
        if (two) quad_to_fixed<P>(c, op, xw, qj, make_float4(__uint_as_float(w1.x), __uint_as_float(w1.y), __uint_as_float(w1.z), __uint_as_float(w1.w)), ssq);
    }
    return ssq;
}

// ---- GEMV, phase 2: the rows. A slot holds up to RPS rows of one segment; its eight warps (half_w rows x S slices)
// share them; a lane keeps the same half blocks of x for every row.
// NACT > 0: the operation's half blocks per lane are known when the kernel is built and every lane's half blocks but those
// of the last iteration lie inside the row (TokOp::fast): loads at addresses worked out once (row_pair_dot_at).
// NACT = 0: any shape the kernel takes, addresses worked out per half block.
template <int QT, int P, int NACT>
__device__ __forceinline__ WarpRing gemv_rows(const TokCtx &c, const TokOp &op, const uint32_t *bo, uint32_t gslot, uint32_t half, const WarpRing wr) {
    constexpr int NX = NACT > 0 ? NACT : NMAX;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t cols = op.cols, nhb = cols / 16, lS = op.log2S, S = 1u << lS, nact = op.nact;
    const uint32_t lRPS = 4 - lS, RPS = 1u << lRPS, lhw = lRPS - 1, half_w = 1u << lhw;  // rows per slot = warps side by side
    const uint32_t row_bytes = tiled_row_bytes(QT, cols);
    const uint32_t rows0 = bo[1] & 0xffffu, rows1 = bo[1] >> 16, rows2 = bo[2];
    const uint32_t sl0 = (rows0 + RPS - 1) >> lRPS, sl1 = sl0 + ((rows1 + RPS - 1) >> lRPS), total_slots = sl1 + ((rows2 + RPS - 1) >> lRPS);
    const uint4 *xf = reinterpret_cast<const uint4 *>(c.xfb);
    const uint32_t slice = warp & (S - 1), rwl = (warp >> lS) & (half_w - 1);
    const uint32_t lP = lS + op.halves - 1, sum = slice + (half << lS);  // this warp's place among a row's partial sums
    XFixed<P> xr[NX];
#pragma unroll
    for (int i = 0; i < NX; ++i) {
        const uint32_t want = (slice * nact + i) * 32 + lane;
        const uint32_t hbi = min(want, nhb - 1);
        xr[i] = x_fixed_load<P>(xf, hbi);
        if (want >= nhb || (uint32_t)i >= nact) xr[i].step = 0.0f;  // lanes past the end of the row, unused registers
        if (NACT > 0) xr[i].total *= -(QT == BRASA_Q4_0 ? 8 : 32);  // the bias term of half_block_idot_pre
    }
    const uint32_t hi_off = tiled_hi_off(cols), sc_off = tiled_scale_off(QT, cols);
    RowLaneOffsets lo{};
    if (NACT > 0) lo = row_lane_offsets<QT, NX>(cols, slice, lane);
    const uint32_t ring32 = smem_u32(c.ring);
    uint32_t kk = wr.kk, rs = wr.rs, rph = wr.rph;
    bool first_slot = true;
    TRACE(5);
#pragma unroll 1
    for (uint32_t j = kk - gslot; j < total_slots; j += 2) {
        const uint32_t sgi = (j >= sl0) + (j >= sl1);
        const uint32_t ks = j - (sgi == 0 ? 0u : (sgi == 1 ? sl0 : sl1));
        const uint32_t sg_rows = sgi == 0 ? rows0 : (sgi == 1 ? rows1 : rows2), sg_before = sgi == 0 ? 0u : (sgi == 1 ? rows0 : rows0 + rows1);
#ifdef BRASA_TRACE_BUILD
        const long long tw0 = clock64();
#endif
        if (!slot_wait(c, &c.full[rs], rph) && lane == 0) give_up(c, 2);
#ifdef BRASA_TRACE_BUILD
        if (c.trace && c.b == 0 && (threadIdx.x == 0 || threadIdx.x == 256) && c.oi >= c.trace_op && c.oi < c.trace_op + 16) {
            const uint32_t rnd = (j - (kk - gslot - (kk - gslot) % 2)) ;  // unused
            (void)rnd;
            const uint32_t round = (j >> 1) & 7;
            c.trace[4096 + ((c.oi - c.trace_op) * 2 + (threadIdx.x >> 8)) * 16 + round * 2] = (unsigned long long)(clock64() - tw0);
            c.trace[4096 + ((c.oi - c.trace_op) * 2 + (threadIdx.x >> 8)) * 16 + round * 2 + 1] = (unsigned long long)tw0;
        }
#endif
        if (first_slot) {
            TRACE(6);
            first_slot = false;
        }
        const uint32_t n_slot = min(RPS, sg_rows - (ks << lRPS));
        const uint32_t qn = (n_slot + half_w - 1) >> lhw, in_slot = rwl * qn;
        const uint32_t nv = in_slot < n_slot ? min(qn, n_slot - in_slot) : 0u;
        const uint8_t *row0 = c.ring + (size_t)rs * SLOT_CAP + (size_t)in_slot * row_bytes;
        const uint32_t row0_32 = ring32 + rs * SLOT_CAP + in_slot * row_bytes;
        uint32_t r = 0;
#pragma unroll 1
        for (; r + 1 < nv; r += 2) {
            float z;
            if (NACT > 0) {
                z = row_pair_dot_at<QT, NX, P>(row0_32 + r * row_bytes, row0_32 + (r + 1) * row_bytes, lo, xr, lane);
            } else {
                const uint8_t *row_a = row0 + (size_t)r * row_bytes;
                z = row_pair_dot<QT, NX>(row_a, row_a + row_bytes, xr, slice, nhb, hi_off, sc_off, lane, (int)nact);
            }
            if ((lane & 23) == 0) c.part[((sg_before + (ks << lRPS) + in_slot + r + (lane >> 3)) << lP) + sum] = z;
        }
        if (r < nv) {  // an odd row on its own: half the work of a pair (short last slots are shared out one row per warp)
            float z;
            if (NACT > 0) z = row_single_dot_at<QT, NX, P>(row0_32 + r * row_bytes, lo, xr);
            else z = row_single_dot<QT, NX>(row0 + (size_t)r * row_bytes, xr, slice, nhb, hi_off, sc_off, lane, (int)nact);
            if (lane == 0) c.part[((sg_before + (ks << lRPS) + in_slot + r) << lP) + sum] = z;
        }
        __syncwarp();
        if (lane == 0 && kk + c.nslot < c.my_slots) {
            // (the warp's reads of the slot are complete: their values went into the sums stored above)
            // last of the eight: the slot is free, refill it (not after a wait that gave up: the slot's last copy may be on its way still)
            if ((atomicAdd(&c.done[rs], 1u) & ~DONE_PARITY) == TK_WARPS / 2 - 1 && !*c.abort_flag()) {
                c.done[rs] = (c.done[rs] & DONE_PARITY) ^ DONE_PARITY;
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                issue_slot(c, c.sdesc[j], rs);
            }
        }
        kk += 2;
        rs += 2;
        if (rs >= c.nslot) {
            rs -= c.nslot;
            rph ^= 1;
        }
    }
    return WarpRing{kk, rs, rph};
}

// ---- GEMV, phase 3: one thread per output row of this block; the result goes out as activation words.
__device__ __forceinline__ void gemv_epilogue(const TokCtx &c, const TokOp &op, const uint32_t *bo, float scale, uint32_t epoch, float *logits,
                                           unsigned long long *cand, const TokParams &p) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t lS = op.log2S + op.halves - 1, S = 1u << lS;
    const bool swiglu = op.epilogue == EPI_SWIGLU;
    const uint32_t r0 = bo[0], rows0 = bo[1] & 0xffffu, rows1 = bo[1] >> 16, rows2 = bo[2];
    const uint32_t nr = swiglu ? rows0 : rows0 + rows1 + rows2;  // segments follow one another in part[] and in the output
    const float *part = c.part;
    Best bst{-INFINITY, 0xffffffffu};
#ifdef BRASA_TRACE_BUILD
    {
        TRACE(13);
        volatile float dummy = *reinterpret_cast<volatile float *>(c.part);
        if (dummy == 1.2345e-33f) c.part[0] = 0.0f;
        TRACE(14);
        volatile uint32_t d2 = *reinterpret_cast<volatile uint32_t *>(&c.red[40]);
        if (d2 == 0x12345678u) c.part[0] = 0.0f;
        TRACE(15);
    }
#endif
#pragma unroll 1
    for (uint32_t j = tid; j < nr; j += TK_THREADS) {
        float v = 0.0f;
#pragma unroll 1
        for (uint32_t sl = 0; sl < S; ++sl) v += part[(j << lS) + sl];
        v *= scale;
        if (swiglu) {
            float u = 0.0f;
#pragma unroll 1
            for (uint32_t sl = 0; sl < S; ++sl) u += part[((nr + j) << lS) + sl];
            u *= scale;
            v = (v / (1.0f + expf(-v))) * u;
        }
        if (op.epilogue == EPI_RESID && op.xchg) {
            // Tensor parallel: v is this rank's share of the sum over the split columns. It goes into slot [this rank] of
            // every rank's exchange area (parity of the exchange: a slot is rewritten two exchanges later, when its
            // reader has long passed); the owner of the row on every rank then adds the slots in rank order, so all
            // ranks hold the same bits.
            const size_t base = (size_t)((op.xchg - 1) & 1) * p.tp_world * p.tp_stride + r0 + j;
            for (uint32_t q = 0; q < p.tp_world; ++q) xg_store(p.tp_peer[q] + base + (size_t)p.tp_rank * p.tp_stride, __float_as_uint(v), epoch);
            // all ranks' slots are asked for together and only the missing ones again: one round trip once they are there
            const unsigned long long *mine = p.tp_peer[p.tp_rank] + base;
            unsigned long long w[BRASA_TP_MAX_RANKS];
#pragma unroll
            for (int q = 0; q < BRASA_TP_MAX_RANKS; ++q) w[q] = 0;  // epoch 0 is never a launch's
            for (uint32_t it = 0;; ++it) {
                bool ok = true;
#pragma unroll
                for (int q = 0; q < BRASA_TP_MAX_RANKS; ++q) {
                    if ((uint32_t)q < p.tp_world && (uint32_t)(w[q] >> 32) != epoch) {
                        w[q] = xg_load(mine + (size_t)q * p.tp_stride);
                        ok = ok && (uint32_t)(w[q] >> 32) == epoch;
                    }
                }
                if (ok || *c.abort_flag()) break;
                if (it >= p.tp_poll_limit) {
                    give_up(c, 6);
                    break;
                }
            }
            float sum = __uint_as_float((uint32_t)w[0]);
#pragma unroll
            for (int q = 1; q < BRASA_TP_MAX_RANKS; ++q)
                if ((uint32_t)q < p.tp_world) sum += __uint_as_float((uint32_t)w[q]);
            v = sum;
        }
        if (op.epilogue == EPI_RESID) v += c.resid[j];
        if (op.epilogue == EPI_LOGITS) {
            logits[r0 + j] = v;
            if (v > bst.v) bst = Best{v, r0 + j};
        } else {
            TRACE(9);
            vs_store(op.out + c.par_cur + r0 + j, op.out + c.par_alt + r0 + j, __float_as_uint(v));
            TRACE(10);
        }
    }
    if (op.epilogue == EPI_LOGITS) {  // this block's best logit for the greedy choice
        for (int o = 16; o > 0; o >>= 1) {
            Best other{__shfl_xor_sync(0xffffffffu, bst.v, o), __shfl_xor_sync(0xffffffffu, bst.i, o)};
            bst = better(bst, other);
        }
        if (lane == 0) { c.red[RED_BEST + warp] = bst.v; c.red[RED_INDEX + warp] = __uint_as_float(bst.i); }
        __syncthreads();
        if (tid == 0) {
#pragma unroll 1
            for (int w = 1; w < TK_WARPS; ++w) bst = better(bst, Best{c.red[RED_BEST + w], __float_as_uint(c.red[RED_INDEX + w])});
            ll_store(cand + 2 * c.b, __float_as_uint(bst.v), epoch);
            ll_store(cand + 2 * c.b + 1, bst.i, epoch);
        }
    }
}

// PLANES: byte planes of the fixed-point input of the GEMVs (gemv_device.cuh). An f32 cache keeps the f32 accuracy class of the kernel-
// per-operation path; f16 and q8_0 caches, whose own rounding is orders of magnitude larger, take two. Models whose feed-forward goes in
// halves keep three for every cache: they had the 22 bits of the kernel-per-operation path before they came here.
template <int KV, int PLANES>
__global__ void __maxnreg__(128) decode_token_kernel(TokParams p) {
    extern __shared__ __align__(128) uint8_t smem[];
    TokCtx c;
    c.ring = smem;
    c.xfb = c.ring + (size_t)p.nslot * SLOT_CAP;
    c.part = reinterpret_cast<float *>(c.xfb + p.xf_bytes);
    c.resid = c.part + p.part_floats;
    c.nwbuf = c.resid + p.resid_floats;                              // norm weight of the current operation
    c.sdesc = reinterpret_cast<uint4 *>(c.nwbuf + p.nw_floats);      // descriptors of the slots this operation refills
    c.full = reinterpret_cast<uint64_t *>(c.sdesc + p.sdesc_n);
    c.done = reinterpret_cast<uint32_t *>(c.full + p.nslot);
    c.red = reinterpret_cast<float *>(c.done + p.nslot);             // [RED_WORDS]
    uint32_t *ops_s = reinterpret_cast<uint32_t *>(c.red + RED_WORDS);      // [2][OPS_WORDS]: operation, then this block's rows
    c.s_abort = ops_s + 2 * OPS_WORDS;
    c.status = p.status;
    c.trace = p.trace;
    c.trace_op = p.trace_op;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t G = gridDim.x, b = blockIdx.x;
    c.G = G;
    c.b = b;
    c.pos = p.state[0];
    c.seq = p.state[2];
    c.par_cur = (c.seq & 1) * p.par_words;
    c.par_alt = p.par_words - c.par_cur;
    c.token = p.ids[0];
    c.nslot = p.nslot;
    const uint32_t slot_lo = p.slot_begin[b];
    c.my_slots = p.slot_begin[b + 1] - slot_lo;
    c.myslots = reinterpret_cast<const uint4 *>(p.slots + slot_lo);
    c.h0 = p.hidden * b / G;  // this block's rows of a hidden-size vector
    c.hn = p.hidden * (b + 1) / G - c.h0;

    // operation oi and this block's row counts for it -> ops_s[oi & 1]
    // (by the last threads of the block: the first ones are the busiest in the input phase)
    auto fetch_op = [&](uint32_t oi) {
        const int t = TK_THREADS - 1 - tid;
        if (t < (int)OP_WORDS) ops_s[(oi & 1) * OPS_WORDS + t] = reinterpret_cast<const uint32_t *>(p.ops + oi)[t];
        else if (t < (int)OPS_WORDS) ops_s[(oi & 1) * OPS_WORDS + t] = reinterpret_cast<const uint32_t *>(p.block_ops + (size_t)oi * G + b)[t - OP_WORDS];
    };
    if (tid == 0) {
        for (uint32_t s = 0; s < p.nslot; ++s) {
            mbar_init(&c.full[s], 1);
            c.done[s] = 0;
        }
        *c.s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    fetch_op(0);
    __syncthreads();
    {   // the first operation's norm weight (later ones are staged one operation ahead)
        const TokOp &op0 = *reinterpret_cast<const TokOp *>(ops_s);
        if (op0.normw)
            for (uint32_t i = tid; i < op0.cols / 4; i += TK_THREADS) cp_async16(c.nwbuf + 4 * i, op0.normw + 4 * i);
        asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
    }
    if (tid == 0) {
        uint32_t k = 0;
        for (; k < c.my_slots && k < p.nslot; ++k) issue_slot(c, c.myslots[k], k);
    }

    // This warp's slots are the list entries kk = sub, sub + 2, ..: warps 0-7 take the even ones, warps 8-15 the odd
    // ones, and with an even ring a ring slot always serves the same eight warps, which all wait for every use of it.
    WarpRing wr{(uint32_t)warp >> 3, (uint32_t)warp >> 3, 0u};
    uint32_t gslot = 0;  // list index of the current operation's first slot

#pragma unroll 1
    for (uint32_t oi = 0; oi < p.nops; ++oi) {
        const TokOp &op = *reinterpret_cast<const TokOp *>(ops_s + (oi & 1) * OPS_WORDS);
        const uint32_t *bo = ops_s + (oi & 1) * OPS_WORDS + OP_WORDS;  // r0, rows of segments 0 and 1 (16 bits each), rows of segment 2
        if (oi + 1 < p.nops) fetch_op(oi + 1);
        const uint32_t epoch = c.seq * EPOCH_SPAN + oi + 1;

        c.oi = oi;
        TRACE(0);
        TRACEB(0);
        if (op.next_normw) {  // the next operation's norm weight, copied while this one runs (the idle end of the block first)
            for (uint32_t i = TK_THREADS - 1 - tid; i < op.next_cols / 4; i += TK_THREADS) cp_async16(c.nwbuf + 4 * i, op.next_normw + 4 * i);
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
        if (op.type == OP_GEMV) {
            const uint32_t lRPS = 4 - op.log2S, RPS = 1u << lRPS;
            const uint32_t total_slots = (((bo[1] & 0xffffu) + RPS - 1) >> lRPS) + (((bo[1] >> 16) + RPS - 1) >> lRPS) + ((bo[2] + RPS - 1) >> lRPS);
#pragma unroll 1
            for (uint32_t half = 0; half < op.halves; ++half) {
                // the descriptors this operation's refills and L2 requests will need, fetched by the threads that poll least
                for (uint32_t i = TK_THREADS - 1 - tid; i < total_slots; i += TK_THREADS) {
                    const uint32_t k = gslot + p.nslot + i;
                    c.sdesc[i] = k < c.my_slots ? c.myslots[k] : make_uint4(0, 0, 0, 0);
                }
                TRACE(1);
                float ssq = gemv_input<PLANES>(c, op, p.embed, p.vocab, half);
                TRACE(3);
                TRACEB(1);
                for (int o = 16; o > 0; o >>= 1) ssq += __shfl_xor_sync(0xffffffffu, ssq, o);
                if (lane == 0) c.red[warp] = ssq;
                __syncthreads();
                TRACE(4);
                if (warp == TK_WARPS - 1) {  // 1 / rms of the whole input from the warps' sums, parked for the epilogue
                    float tot = c.red[lane & (TK_WARPS - 1)];
                    for (int o = TK_WARPS / 2; o > 0; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
                    if (lane == 0) c.red[RED_SCALE] = op.scaled ? 1.0f / sqrtf(tot / (float)op.cols + op.eps) : 1.0f;
                }
                if (op.qtype == BRASA_Q4_0) {
                    if (op.fast && op.nact == 5) wr = gemv_rows<BRASA_Q4_0, PLANES, 5>(c, op, bo, gslot, half, wr);
                    else if (op.fast && op.nact == 4) wr = gemv_rows<BRASA_Q4_0, PLANES, 4>(c, op, bo, gslot, half, wr);
                    else wr = gemv_rows<BRASA_Q4_0, PLANES, 0>(c, op, bo, gslot, half, wr);
                } else {
                    if (op.fast && op.nact == 5) wr = gemv_rows<BRASA_Q6_0, PLANES, 5>(c, op, bo, gslot, half, wr);
                    else wr = gemv_rows<BRASA_Q6_0, PLANES, 0>(c, op, bo, gslot, half, wr);
                }
                TRACE(7);
                TRACEB(2);
                gslot += total_slots;
                __syncthreads();
                TRACE(8);
            }
            gemv_epilogue(c, op, bo, c.red[RED_SCALE], epoch, p.logits, p.cand, p);
        } else {
            attention_op<KV>(AttnCtx{c.xfb, c.s_abort, c.status, c.G, c.b, c.pos, c.par_cur, c.par_alt}, op, oi, epoch, p.heads, p.kv_heads, p.max_chunks, p.cos_t, p.sin_t, p.partials, p.attn_scale);
        }
        TRACE(11);
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        TRACE(12);
        TRACEB(3);
    }

    // a block that has given up waits (again with a limit) for its copies before it leaves
    if (*c.s_abort) {
        uint32_t s;  // worked out anew: what is kept for here from before the loop over the operations is spilled in it
        asm volatile("mov.u32 %0, %%tid.x;" : "=r"(s));
        if (s < min(p.nslot, p.slot_begin[b + 1] - p.slot_begin[b])) mbar_wait(&c.full[s], c.done[s] >> 31);
    }

    // ---- greedy choice and the step's bookkeeping: block 0 gathers every block's best logit ----
    if (b == 0) {
        const uint32_t epoch = c.seq * EPOCH_SPAN + p.nops;  // of the lm_head, the last operation
        Best bst{-INFINITY, 0xffffffffu};
#pragma unroll 1
        for (uint32_t i = tid; i < G; i += TK_THREADS) {
            uint32_t raw[4];
            ll_wait4(c, p.cand + 2 * i, p.cand + 2 * i + 1, p.cand + 2 * i, p.cand + 2 * i + 1, epoch, raw);
            bst = better(bst, Best{__uint_as_float(raw[0]), raw[1]});
        }
        for (int o = 16; o > 0; o >>= 1) {
            Best other{__shfl_xor_sync(0xffffffffu, bst.v, o), __shfl_xor_sync(0xffffffffu, bst.i, o)};
            bst = better(bst, other);
        }
        if (lane == 0) { c.red[RED_BEST + warp] = bst.v; c.red[RED_INDEX + warp] = __uint_as_float(bst.i); }
        __syncthreads();
        if (tid == 0) {
#pragma unroll 1
            for (int w = 1; w < TK_WARPS; ++w) bst = better(bst, Best{c.red[RED_BEST + w], __float_as_uint(c.red[RED_INDEX + w])});
            if (p.tp_world > 1) {
                // this rank's best (logit, vocabulary row) to every rank, then the best of all: largest logit, lowest row
                // among equals (NaN never wins: it never became a candidate)
                const size_t abase = 2 * (size_t)p.tp_world * p.tp_stride + (size_t)(c.seq & 1) * p.tp_world * 2;
                const uint32_t mine = bst.i == 0xffffffffu ? 0xffffffffu : bst.i + p.tp_row0;
                for (uint32_t q = 0; q < p.tp_world; ++q) {
                    xg_store(p.tp_peer[q] + abase + 2 * p.tp_rank, __float_as_uint(bst.v), epoch);
                    xg_store(p.tp_peer[q] + abase + 2 * p.tp_rank + 1, mine, epoch);
                }
                Best all{-INFINITY, 0xffffffffu};
                for (uint32_t q = 0; q < p.tp_world; ++q) {
                    const unsigned long long *src = p.tp_peer[p.tp_rank] + abase + 2 * q;
                    unsigned long long w0 = 0, w1 = 0;
                    for (uint32_t it = 0;; ++it) {
                        w0 = xg_load(src);
                        w1 = xg_load(src + 1);
                        if (((uint32_t)(w0 >> 32) == epoch && (uint32_t)(w1 >> 32) == epoch) || *c.abort_flag()) break;
                        if (it >= p.tp_poll_limit) {
                            give_up(c, 6);
                            break;
                        }
                    }
                    if ((uint32_t)(w0 >> 32) == epoch && (uint32_t)(w1 >> 32) == epoch)
                        all = better(all, Best{__uint_as_float((uint32_t)w0), (uint32_t)w1});
                }
                bst = all;
            }
            const uint32_t tok = (bst.v == -INFINITY || bst.i == 0xffffffffu) ? 0u : bst.i;
            *p.next_id = tok;
            p.ids[0] = tok;
            const uint32_t n = p.state[1];
            if (n < p.out_cap) p.out_ids[n] = tok;
            p.state[1] = n + 1;
            p.state[0] = c.pos + 1;
            p.state[2] = c.seq + 1;
        }
    }
}

typedef void (*TokenKernel)(TokParams);
TokenKernel token_kernel(int32_t kv, int planes) {
    if (kv == BRASA_KV_F32) return decode_token_kernel<BRASA_KV_F32, 3>;
    if (kv == BRASA_KV_F16) return planes == 3 ? decode_token_kernel<BRASA_KV_F16, 3> : decode_token_kernel<BRASA_KV_F16, 2>;
    return planes == 3 ? decode_token_kernel<BRASA_KV_Q8_0, 3> : decode_token_kernel<BRASA_KV_Q8_0, 2>;
}

// Column slices and active half blocks per lane for a GEMV of this width; false when the kernel does not take it.
bool gemv_shape(int qtype, uint32_t cols, uint32_t *S_out, uint32_t *nact_out) {
    if (cols == 0 || cols % 256 != 0) return false;
    const uint32_t nhb = cols / 16, row_bytes = tiled_row_bytes(qtype, cols);
    for (uint32_t S = 1; S <= 8; S *= 2) {
        uint32_t N = (nhb + 32 * S - 1) / (32 * S);
        uint32_t RPS = TK_WARPS / S * R / 2;
        if (N <= NMAX && (uint64_t)RPS * row_bytes <= SLOT_CAP) {
            *S_out = S;
            *nact_out = N;
            return true;
        }
    }
    return false;
}

// How many pieces a q4_0 row of `cols` columns is taken in: one where the kernel takes it whole, two where it takes half of it (20 481 to
// 40 960 columns: the 32B architecture's 25 600 on one GPU), 0 where neither.
uint32_t gemv_halves(uint32_t cols) {
    uint32_t S, n;
    if (gemv_shape(BRASA_Q4_0, cols, &S, &n)) return 1;
    return cols % 512 == 0 && cols / 2 < 65536 && gemv_shape(BRASA_Q4_0, cols / 2, &S, &n) ? 2 : 0;
}

}  // namespace

struct brasa_token_program {
    brasa_ctx *ctx = nullptr;
    TokParams params{};
    size_t smem = 0;
    int32_t kv = 0;
    int planes = 2;
    uint32_t grid = 0;
    std::vector<void *> device;  // allocations owned by the program
    void *vectors = nullptr;     // both copies of the activation vectors
    size_t vector_bytes = 0;
    uint32_t timeouts_seen = 0;  // the context's count of abandoned waits when the vectors were last known clean
    brasa_token_mma *mma = nullptr;  // the token runs there instead (decode_token_mma.cu)
};

bool brasa_token_program_supported(brasa_ctx *ctx, const brasa_token_model &m) {
    if (m.head_dim != 128 || m.kv_heads == 0 || m.heads % m.kv_heads != 0 || m.heads / m.kv_heads > 8) return false;
    if (m.layers.empty() || m.layers.size() * 5 + 3 >= EPOCH_SPAN) return false;
    if (m.embed.layout != BRASA_LAYOUT_TILED || m.embed.qtype != BRASA_Q6_0 || m.embed.cols != m.hidden) return false;
    if (m.head.layout != BRASA_LAYOUT_TILED || (m.head.qtype != BRASA_Q4_0 && m.head.qtype != BRASA_Q6_0)) return false;
    uint32_t S, n;
    if (!gemv_shape(m.head.qtype, m.hidden, &S, &n) || !gemv_shape(BRASA_Q4_0, m.hidden, &S, &n) ||
        !gemv_shape(BRASA_Q4_0, m.heads * 128, &S, &n) || !gemv_halves(m.ffn))
        return false;
    for (const brasa_token_layer &l : m.layers)
        for (const brasa_qmatrix *w : {&l.wq, &l.wk, &l.wv, &l.wo, &l.gate, &l.up, &l.down})
            if (w->layout != BRASA_LAYOUT_TILED || w->qtype != BRASA_Q4_0) return false;
    int coop = 0;
    if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, ctx->device) != cudaSuccess || !coop) return false;
    return true;
}

void brasa_token_program_free(brasa_token_program *p) {
    if (!p) return;
    brasa_token_mma_free(p->mma);
    for (void *d : p->device) cudaFree(d);
    delete p;
}

int32_t brasa_token_program_create(brasa_ctx *ctx, const brasa_token_model &m, brasa_token_program **out) {
    BRASA_REQUIRE(ctx, out && brasa_token_program_supported(ctx, m), "token program: model shape not supported");
    std::unique_ptr<brasa_token_program, void (*)(brasa_token_program *)> prog(new brasa_token_program, brasa_token_program_free);
    prog->ctx = ctx;
    if (brasa_token_mma_takes(m)) {
        BRASA_TRY(brasa_token_mma_create(ctx, m, &prog->mma));
        if (prog->mma) {
            *out = prog.release();
            return BRASA_OK;
        }
    }
    prog->kv = m.kv;
    prog->planes = m.kv == BRASA_KV_F32 || gemv_halves(m.ffn) == 2 ? 3 : 2;
    const uint32_t G = (uint32_t)ctx->sm_count;
    prog->grid = G;
    const uint32_t H = m.hidden, QD = m.heads * 128, KD = m.kv_heads * 128, F = m.ffn;
    const uint32_t C = attn_chunk(m.kv), max_chunks = (m.cache_positions + C - 1) / C;

    auto dev_alloc = [&](size_t bytes, void **ptr) -> int32_t {
        BRASA_CUDA(ctx, cudaMalloc(ptr, bytes));
        prog->device.push_back(*ptr);
        return brasa_check_cuda(ctx, cudaMemset(*ptr, 0, bytes), "cudaMemset");
    };
    // attention partials and argmax candidates as {value, epoch} words
    unsigned long long *partials, *cand;
    const size_t ll_words = (size_t)m.heads * max_chunks * 130 + 2 * G;
    void *ll_base;
    BRASA_TRY(dev_alloc(ll_words * 8, &ll_base));
    partials = (unsigned long long *)ll_base;
    cand = partials + (size_t)m.heads * max_chunks * 130;
    // every operation's output vector: two copies of par_words 4-byte words, all empty at first
    const size_t per_layer = (size_t)(QD + 2 * KD) + QD + H + F + H;
    const size_t par_words = (per_layer * m.layers.size() + 31) / 32 * 32;
    BRASA_REQUIRE(ctx, par_words < (1u << 31), "token program: activation vectors too large");
    void *vs_base;
    BRASA_TRY(dev_alloc(par_words * 8, &vs_base));
    BRASA_CUDA(ctx, cudaMemset(vs_base, 0xff, par_words * 8));
    prog->vectors = vs_base;
    prog->vector_bytes = par_words * 8;
    prog->timeouts_seen = ctx->timeouts;
    uint32_t *vs_next = (uint32_t *)vs_base;
    auto vec_alloc = [&](size_t n) { uint32_t *r = vs_next; vs_next += n; return r; };

    // ---- the operations ----
    std::vector<TokOp> ops;
    auto gemv_op = [&](uint32_t nmat, const brasa_qmatrix *w, uint32_t epilogue, bool scaled, const float *normw, int in_op, bool save_resid) {
        TokOp o{};
        o.type = OP_GEMV;
        o.qtype = (uint32_t)w[0].qtype;
        o.halves = w[0].qtype == BRASA_Q4_0 && gemv_halves(w[0].cols) == 2 ? 2 : 1;
        o.cols = w[0].cols / o.halves;
        o.nmat = nmat;
        o.total_rows = 0;
        for (uint32_t i = 0; i < nmat; ++i) {
            o.rows[i] = w[i].rows;
            o.w[i] = arg_ptr(w[i].data);
            o.total_rows += w[i].rows;
        }
        if (epilogue == EPI_SWIGLU) o.total_rows = w[0].rows;
        o.epilogue = epilogue;
        o.scaled = scaled ? 1 : 0;
        uint32_t S = 1;
        gemv_shape(w[0].qtype, o.cols, &S, &o.nact);
        for (o.log2S = 0; (1u << o.log2S) < S; ++o.log2S) {}
        o.fast = o.nact >= 2 ? ((S * o.nact - 2) * 32 + 31 < o.cols / 16) : 1;
        o.in_kind = in_op < 0 ? IN_EMBED : IN_LL;
        o.in_op = in_op < 0 ? 0 : (uint32_t)in_op;
        o.save_resid = save_resid ? 1 : 0;
        o.eps = m.eps;
        o.normw = normw;
        o.in = in_op < 0 ? nullptr : ops[in_op].out;
        o.out = epilogue == EPI_LOGITS ? nullptr : vec_alloc(o.total_rows);
        ops.push_back(o);
        return (int)ops.size() - 1;
    };
    int x_op = -1;  // operation that produced the current residual stream (-1: the embedding row)
    const bool tp_on = m.tp.world > 1;
    BRASA_REQUIRE(ctx, !tp_on || (m.tp.world <= BRASA_TP_MAX_RANKS && m.tp.rank < m.tp.world && m.tp.stride >= H),
                  "token program: the exchange area is smaller than the hidden size");
    uint32_t nxchg = 0;
    for (const brasa_token_layer &l : m.layers) {
        brasa_qmatrix wqkv[3] = {l.wq, l.wk, l.wv};
        BRASA_REQUIRE(ctx, l.wq.rows == QD && l.wk.rows == KD && l.wv.rows == KD && l.wq.cols == H && l.wo.rows == H && l.wo.cols == QD &&
                               l.gate.rows == F && l.up.rows == F && l.gate.cols == H && l.down.rows == H && l.down.cols == F,
                      "token program: unexpected matrix shape");
        int qkv_op = gemv_op(3, wqkv, EPI_SCALE, true, l.attn_norm, x_op, true);
        TokOp a{};
        a.type = OP_ATTN;
        a.in_op = (uint32_t)qkv_op;
        a.eps = m.eps;
        a.in = ops[qkv_op].out;
        a.out = vec_alloc(QD);
        a.q_norm = l.q_norm;
        a.k_norm = l.k_norm;
        a.kc = l.kc;
        a.vc = l.vc;
        ops.push_back(a);
        int attn_op = (int)ops.size() - 1;
        int o_op = gemv_op(1, &l.wo, EPI_RESID, false, nullptr, attn_op, false);
        if (tp_on) ops[o_op].xchg = ++nxchg;
        brasa_qmatrix wgu[2] = {l.gate, l.up};
        int gu_op = gemv_op(2, wgu, EPI_SWIGLU, true, l.ffn_norm, o_op, true);
        x_op = gemv_op(1, &l.down, EPI_RESID, false, nullptr, gu_op, false);
        if (tp_on) ops[x_op].xchg = ++nxchg;
    }
    BRASA_REQUIRE(ctx, (tp_on ? m.head.rows + m.head_row0 <= m.vocab : m.head.rows == m.vocab) && m.head.cols == H, "token program: unexpected lm_head shape");
    gemv_op(1, &m.head, EPI_LOGITS, true, m.final_norm, x_op, false);
    BRASA_REQUIRE(ctx, (size_t)(vs_next - (uint32_t *)vs_base) <= par_words, "token program: activation vectors overran their area");
    BRASA_REQUIRE(ctx, ops.size() + 2 < EPOCH_SPAN, "token program: too many operations");
    uint32_t nw_floats = 0;
    for (size_t i = 0; i < ops.size(); ++i) {
        if (ops[i].normw) nw_floats = std::max(nw_floats, ops[i].cols);
        if (i + 1 < ops.size() && ops[i + 1].normw) {
            BRASA_REQUIRE(ctx, !ops[i].normw, "token program: two operations in a row with a norm weight");
            ops[i].next_normw = ops[i + 1].normw;
            ops[i].next_cols = ops[i + 1].cols;
        }
    }

    // ---- every block's slot list, in the order the kernel consumes it, and its rows of every operation ----
    std::vector<SlotDesc> slots;
    std::vector<uint32_t> slot_begin(G + 1, 0);
    std::vector<uint4> block_ops(ops.size() * G, make_uint4(0, 0, 0, 0));
    uint32_t part_floats = 0, max_cols = 0, max_op_slots = 0;
    for (uint32_t b = 0; b < G; ++b) {
        slot_begin[b] = (uint32_t)slots.size();
        for (size_t oi = 0; oi < ops.size(); ++oi) {
            const TokOp &o = ops[oi];
            if (o.type != OP_GEMV) continue;
            const bool swiglu = o.epilogue == EPI_SWIGLU;
            uint32_t r0, r1, first[3], nrows[3];
            block_rows(o.total_rows, o.nmat, o.rows, swiglu, b, G, r0, r1, first, nrows);
            BRASA_REQUIRE(ctx, nrows[0] < 65536 && nrows[1] < 65536, "token program: too many rows per block");
            block_ops[oi * G + b] = make_uint4(r0, nrows[0] | (nrows[1] << 16), nrows[2], 0);
            const uint32_t S = 1u << o.log2S, RPS = TK_WARPS / S * R / 2, row_bytes = tiled_row_bytes((int)o.qtype, o.cols);
            uint32_t items = 0, op_slots = 0;
            for (uint32_t half = 0; half < o.halves; ++half) {
                op_slots = 0;
                items = 0;
                for (int i = 0; i < 3; ++i) {
                    for (uint32_t f = 0; f < nrows[i]; f += RPS) {
                        const uint32_t n = std::min(RPS, nrows[i] - f);
                        slots.push_back(SlotDesc{o.w[i] + (size_t)(first[i] + f) * row_bytes * o.halves, n * row_bytes,
                                                 o.halves == 2 ? o.cols | (n << 16) | (half << 24) : 0u});
                        ++op_slots;
                    }
                    items += nrows[i];
                }
            }
            part_floats = std::max(part_floats, items * S * o.halves);
            max_cols = std::max(max_cols, o.cols);
            max_op_slots = std::max(max_op_slots, op_slots);
        }
    }
    slot_begin[G] = (uint32_t)slots.size();

    TokParams &p = prog->params;
    void *d_ops, *d_slots, *d_begin, *d_bops;
    BRASA_TRY(dev_alloc(block_ops.size() * sizeof(uint4), &d_bops));
    BRASA_CUDA(ctx, cudaMemcpy(d_bops, block_ops.data(), block_ops.size() * sizeof(uint4), cudaMemcpyHostToDevice));
    BRASA_TRY(dev_alloc(ops.size() * sizeof(TokOp), &d_ops));
    BRASA_TRY(dev_alloc(std::max<size_t>(slots.size(), 1) * sizeof(SlotDesc), &d_slots));
    BRASA_TRY(dev_alloc(slot_begin.size() * 4, &d_begin));
    BRASA_CUDA(ctx, cudaMemcpy(d_ops, ops.data(), ops.size() * sizeof(TokOp), cudaMemcpyHostToDevice));
    BRASA_CUDA(ctx, cudaMemcpy(d_slots, slots.data(), slots.size() * sizeof(SlotDesc), cudaMemcpyHostToDevice));
    BRASA_CUDA(ctx, cudaMemcpy(d_begin, slot_begin.data(), slot_begin.size() * 4, cudaMemcpyHostToDevice));
    p.ops = (const TokOp *)d_ops;
    p.nops = (uint32_t)ops.size();
    p.slots = (const SlotDesc *)d_slots;
    p.slot_begin = (const uint32_t *)d_begin;
    p.block_ops = (const uint4 *)d_bops;

    // ---- shared memory ----
    const size_t attn_bytes = ATTN_AREA_BYTES;
    p.xf_bytes = (uint32_t)((std::max<size_t>((size_t)max_cols / 16 * 16 * (prog->planes == 3 ? XRec<3>::CHUNKS : XRec<2>::CHUNKS), attn_bytes) + 127) / 128 * 128);
    p.part_floats = (part_floats + 3) & ~3u;
    p.resid_floats = ((H + G - 1) / G + 4) & ~3u;
    p.sdesc_n = max_op_slots;
    p.nw_floats = (nw_floats + 3) & ~3u;
    const size_t fixed = p.xf_bytes + (size_t)(p.part_floats + p.resid_floats + p.nw_floats) * 4 + (size_t)p.sdesc_n * 16 + RED_WORDS * 4 + 2 * OPS_WORDS * 4 + 16;
    BRASA_REQUIRE(ctx, fixed + 2 * (SLOT_CAP + 12) + 1024 <= ctx->smem_optin, "token program: the model's vectors do not fit shared memory");
    uint32_t nslot = (uint32_t)((ctx->smem_optin - 1024 - fixed) / (SLOT_CAP + 12));
    nslot &= ~1u;  // even: a ring slot always serves the same half of the warps
    p.nslot = nslot;
    prog->smem = (size_t)nslot * (SLOT_CAP + 12) + fixed;

    p.state = m.state;
    p.ids = m.ids;
    p.next_id = m.next_id;
    p.out_ids = m.out_ids;
    p.out_cap = m.out_cap;
    p.embed = arg_ptr(m.embed.data);
    p.vocab = m.vocab;
    p.hidden = H;
    p.heads = m.heads;
    p.kv_heads = m.kv_heads;
    p.max_chunks = max_chunks;
    p.cos_t = m.cos_t;
    p.sin_t = m.sin_t;
    p.logits = m.logits;
    p.cand = cand;
    p.par_words = (uint32_t)par_words;
    p.partials = partials;
    p.attn_scale = 1.0f / sqrtf(128.0f);
    p.status = ctx->status;
    p.tp_world = tp_on ? m.tp.world : 1;
    p.tp_rank = tp_on ? m.tp.rank : 0;
    p.tp_row0 = m.head_row0;
    p.tp_stride = m.tp.stride;
    p.tp_poll_limit = m.tp.poll_limit ? m.tp.poll_limit : POLL_LIMIT;
    for (uint32_t r = 0; r < BRASA_TP_MAX_RANKS; ++r) p.tp_peer[r] = tp_on && r < m.tp.world ? m.tp.peer[r] : nullptr;
    p.trace = ctx->gemv_trace;
    {
        const char *env = getenv("BRASA_TRACE_OP");
        p.trace_op = env ? (uint32_t)atoi(env) : 5;
    }

    const TokenKernel fn = token_kernel(m.kv, prog->planes);
    BRASA_TRY(brasa_smem_optin(ctx, (const void *)fn, prog->smem));
    int per_sm = 0;
    BRASA_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, TK_THREADS, prog->smem));
    BRASA_REQUIRE(ctx, per_sm >= 1, "token program: the kernel does not fit an SM");
    *out = prog.release();
    return BRASA_OK;
}

int32_t brasa_token_program_launch(brasa_cmd *cmd, brasa_token_program *prog) {
    brasa_ctx *ctx = cmd->ctx;
    if (prog->mma) return brasa_token_mma_launch(cmd, prog->mma);
    if (prog->timeouts_seen != ctx->timeouts) {
        // a launch that gave up may have left words of either copy unwritten or not emptied: start from all empty
        BRASA_CUDA(ctx, cudaMemsetAsync(prog->vectors, 0xff, prog->vector_bytes, ctx->stream));
        prog->timeouts_seen = ctx->timeouts;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(prog->grid);
    cfg.blockDim = dim3(TK_THREADS);
    cfg.dynamicSmemBytes = prog->smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;  // every block resident at once: blocks wait for one another's outputs
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    BRASA_CUDA(ctx, cudaLaunchKernelEx(&cfg, token_kernel(prog->kv, prog->planes), prog->params));
    return brasa_post_launch(cmd, "decode_token");
}
