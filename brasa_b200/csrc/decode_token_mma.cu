// The whole-token kernel of decode_token.cu with its GEMVs on integer tensor products (gemv_mma.cuh): one cooperative launch, one block per
// SM, the weights of all operations streaming through a shared-memory ring, the activations through words in L2 that carry their own
// arrival. It takes models whose input vectors are two byte planes (f16 and q8_0 caches, one GPU) and whose operations have enough to
// multiply (brasa_token_mma_takes). What is different here:
//   * The rows phase takes tiles of up to sixteen rows; a block's rows of all an operation's matrices stand in one list, a ring slot is
//     a run of that list. dp4a needs 8 instructions for 16 weights and plane pair beside the loads; here it is one for 512 weights.
//   * What a warp has to work out for its rows, and the wait for their slots, come before the wait for the input (tile_begin): behind
//     it every one of those instructions is on the path of the whole token, 900 cycles of an operation's 6 000.
//   * What an operation needs beside its input (itself, its slots' descriptors, its norm weight) is copied asynchronously.
// Bound: the exchanges and, in the rows phase, shared-memory bandwidth (a unit of 16 rows x 128 columns takes 22 wavefronts, 8 of
// them the codes). Each operation ends with a block barrier although nothing there needs one: without it the warps that have no
// rows to store poll for the next input beside those that do, and hold up their stores (1.24 against 1.10 ms a token).
// us a token, one B200, decode_token.cu's in brackets: 4B architecture at 512 positions, f16 992 (1 118); at 16 384, q8_0 1 698 (1 845).
#include <memory>

#include "decode_token_mma.h"
#include "gemv_mma.cuh"
#include "token_device.cuh"

using namespace brasa_dev;

namespace {

constexpr uint32_t SLOT_CAP = 23040;  // bytes of one ring slot: sixteen rows of 2 560 columns, eight of 5 120, four of 10 240
constexpr uint32_t TILE = 16;         // rows of a warp's products
constexpr uint32_t MAX_COLS = 10240;  // (wider rows are fewer than four to a slot: a tile would hold most of the ring)
// Hidden sizes this kernel takes; us a token against decode_token.cu's (4 layers, f16, 100 positions): 512 55.6 (57.4), but a short chat of
// it 1 052 (1 023); 768 73.5 (75.4), 1 024 77.7 (83.8), 1 536 83.7 (90.3), 2 048 161 (167), 2 560 173 (201), 4 096 193 (182): rows of 4 096
// columns all begin in the same shared-memory bank and fill four fifths of a slot.
constexpr uint32_t MIN_HIDDEN = 768, MAX_HIDDEN = 3072;

struct SlotDesc {
    const uint8_t *src[2];  // the rows of one matrix, and of the next one where the slot reaches into it
    uint32_t bytes[2];
    uint32_t pad[2];
};
static_assert(sizeof(SlotDesc) == 32, "SlotDesc is copied as two 16-byte words");

struct TokOp {
    uint32_t type, qtype, cols, lrps;       // lrps: log2 of the rows of a slot
    uint32_t tile, step, slices, swap;      // rows of a tile (its slots are held together while it is worked on), from a warp's tile to its next; swap: see tile_row
    uint32_t epilogue, scaled, in_kind, save_resid;
    uint32_t meta_off, part_off, nw_use, next_cols;  // where x's bias terms and steps lie in shared memory, where the partial sums; how many
                                                     // norm weights have been staged when this one is there; length of next_normw
    float eps;
    uint32_t nmat, rows[3], total_rows;     // (host)
    const uint8_t *w[3];                    // (host)
    const float *normw, *next_normw;        // next_normw: of the operation after this one (null: none)
    const uint32_t *in;                     // first copy; the second one lies TokParams::par_words further
    uint32_t *out;
    const float *q_norm, *k_norm;
    uint8_t *kc, *vc;
};
// What a warp has to do with an operation: the first row of its first tile (NO_ROWS: none), its slice, its groups of 128 columns.
struct WarpPlan {
    uint32_t row, slice, g0, g1;
};
constexpr uint32_t NO_ROWS = 0x7fffffffu;
// An operation as the blocks fetch it: the operation, the warps' plans, and (per block) the block's rows.
struct OpRecord {
    TokOp op;
    WarpPlan plan[TK_WARPS];
};
struct BlockRows {
    uint32_t r0, nout, nrows, slots;  // first output row, output rows, rows of the list over the matrices, ring slots
};
static_assert(sizeof(TokOp) % 16 == 0 && sizeof(OpRecord) % 16 == 0 && sizeof(BlockRows) == 16, "records are copied in 16-byte words");
constexpr uint32_t REC_WORDS = sizeof(OpRecord) / 16, OP_BUFFERS = 2;
struct OpBuffer {
    OpRecord rec;
    BlockRows rows;
};

struct TokParams {
    const OpRecord *ops;
    uint32_t nops;
    const SlotDesc *slots;
    const uint32_t *slot_begin;  // [grid + 1]
    const BlockRows *block_ops;  // [nops][grid]
    uint32_t nslot, nslot_mul;   // nslot_mul: 2^32 / nslot, rounded up
    // where things lie in shared memory behind the ring (TokCtx)
    uint32_t off_xf, off_resid, off_nw, off_sdesc, off_full, off_done, off_red, off_ops, off_zeros;
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
#ifdef BRASA_TRACE_BUILD
    unsigned long long *trace;  // block 0 stamps the phases of 16 operations from trace_op on, as in decode_token.cu
    uint32_t trace_op;
#endif
};

#ifdef BRASA_TRACE_BUILD
#define TRACE(i) do { if (p.trace && blockIdx.x == 0 && threadIdx.x == 0 && oi >= p.trace_op && oi < p.trace_op + 16) p.trace[16 + (oi - p.trace_op) * 16 + (i)] = (unsigned long long)clock64(); } while (0)
#else
#define TRACE(i) do { } while (0)
#endif

// Values 4 qi .. 4 qi + 3 of row `row` of a tiled q6_0 table (embed_kernel's arithmetic).
__device__ __forceinline__ float4 embed_quad(const uint8_t *table, uint32_t row, uint32_t cols, uint32_t qi) {
    const uint8_t *r = table + (size_t)row * tiled_row_bytes(BRASA_Q6_0, cols);
    const uint32_t blk = qi >> 3, w = qi & 3, high = (qi >> 2) & 1;  // word w of the block's codes, its low or high nibbles
    const uint32_t codes = *reinterpret_cast<const uint32_t *>(r + blk * 16 + 4 * w);
    const uint32_t hb = *reinterpret_cast<const uint32_t *>(r + tiled_hi_off(cols) + blk * 8 + 4 * (w >> 1));
    const float d = __half2float(*reinterpret_cast<const __half *>(r + tiled_scale_off(BRASA_Q6_0, cols) + blk * 2));
    const uint32_t up = (w & 1) ? (high ? hb << 4 : hb << 2) : (high ? hb >> 2 : hb);
    const uint32_t a = lop_and_or(up, 0x30303030u, (high ? codes >> 4 : codes) & 0x0F0F0F0Fu);
    return make_float4(d * (float)((int)(a & 255u) - 32), d * (float)((int)((a >> 8) & 255u) - 32), d * (float)((int)((a >> 16) & 255u) - 32),
                       d * (float)((int)(a >> 24) - 32));
}

extern __shared__ __align__(128) uint8_t tk_smem[];

// What the phases of an operation share. The phase functions are inlined: with 227 KB of shared memory in use the
// L1 cache is a few KB, so a stack frame (calls, spills) costs a trip to L2 per access. Places in shared memory are worked out
// where they are used, from constants of the launch: held as pointers they would take a quarter of the registers.
struct TokCtx {
    const TokParams &p;
    uint32_t my_slots, G, b, pos, seq, token, h0, hn;
    uint32_t par_cur, par_alt;  // word offsets of this launch's copy of the activation vectors and of the other one
    __device__ __forceinline__ uint8_t *ring() const { return tk_smem; }
    __device__ __forceinline__ uint8_t *xfb() const { return tk_smem + p.off_xf; }
    __device__ __forceinline__ float *part(const TokOp &op) const { return reinterpret_cast<float *>(tk_smem + op.part_off); }
    __device__ __forceinline__ float *resid() const { return reinterpret_cast<float *>(tk_smem + p.off_resid); }  // this block's rows of the residual stream
    __device__ __forceinline__ float *nwbuf() const { return reinterpret_cast<float *>(tk_smem + p.off_nw); }    // norm weight of the current operation
    __device__ __forceinline__ uint4 *sdesc() const { return reinterpret_cast<uint4 *>(tk_smem + p.off_sdesc); }  // descriptors of the slots this operation refills
    __device__ __forceinline__ uint64_t *full(uint32_t s) const { return reinterpret_cast<uint64_t *>(tk_smem + p.off_full) + s; }
    __device__ __forceinline__ uint64_t *nw_full() const { return full(p.nslot); }
    __device__ __forceinline__ uint32_t *done(uint32_t s) const { return reinterpret_cast<uint32_t *>(tk_smem + p.off_done) + s; }  // warps that are done with a slot
    __device__ __forceinline__ uint32_t *gen(uint32_t s) const { return done(p.nslot + s); }                                       // how often it has been reused
    __device__ __forceinline__ float *red() const { return reinterpret_cast<float *>(tk_smem + p.off_red); }                       // [RED_WORDS]
    __device__ __forceinline__ OpBuffer *ops() const { return reinterpret_cast<OpBuffer *>(tk_smem + p.off_ops); }                 // [OP_BUFFERS]
    __device__ __forceinline__ uint32_t *zeros() const { return reinterpret_cast<uint32_t *>(tk_smem + p.off_zeros); }               // [8]
    __device__ __forceinline__ volatile uint32_t *abort_flag() const { return zeros() + 8; }
    __device__ __forceinline__ volatile uint32_t *norms_asked() const { return zeros() + 9; }  // norm weights whose copy has been asked for
    __device__ __forceinline__ uint32_t *status_word() const { return p.status; }
};

// The thread's number, worked out anew where a phase begins: what a phase derives from it is otherwise moved out of the loop over the
// operations and held in (or spilled from) registers that the other phases need.
__device__ __forceinline__ uint32_t phase_tid() {
    uint32_t t;
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
    return t;
}

__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// A slot's descriptor (two 16-byte words: SlotDesc) -> ring[s].
__device__ __forceinline__ void issue_slot(const TokCtx &c, const uint4 *desc, uint32_t s) {
    const uint4 a = desc[0], d = desc[1];
    uint8_t *dst = c.ring() + (size_t)s * SLOT_CAP;
    mbar_expect_tx(c.full(s), d.x + d.y);
    bulk_g2s(dst, reinterpret_cast<const uint8_t *>(((unsigned long long)a.y << 32) | a.x), d.x, c.full(s));
    if (d.y) bulk_g2s(dst + d.x, reinterpret_cast<const uint8_t *>(((unsigned long long)a.w << 32) | a.z), d.y, c.full(s));
}

// ---- GEMV, phase 1: wait for the input, fold the norm weight, convert to fixed point. A thread takes eight values at a
// time (values 4 j .. and 16 + 4 j .. of a block of 32, so that its words of the planes are neighbours), four lanes share a
// block. Up to 4 096 columns, an input with a norm and an embedding row among them, that is one pass of the block, up to MAX_COLS three; the polls of
// all of them are in flight at once. Returns the warp's share of sum x^2.
static_assert(MAX_HIDDEN <= TK_THREADS * 8 && MAX_COLS <= 3 * TK_THREADS * 8, "passes of gemv_input");
__device__ __forceinline__ float gemv_input(const TokCtx &c, const TokOp &op, const uint8_t *embed, uint32_t vocab) {
    const uint32_t cols = op.cols;
    const uint32_t tid = phase_tid(), nu = cols / 8;  // a multiple of 32: a warp is inside or outside as a whole
    const uint32_t *in = op.in + c.par_cur;
    const int bias = op.qtype == BRASA_Q4_0 ? 8 : 32;
    float ssq = 0.0f;
    const bool normed = op.normw != nullptr;
    float4 n0 = make_float4(1.0f, 1.0f, 1.0f, 1.0f), n1 = n0;
    if (normed && tid < nu) {  // the norm weight, a bulk copy asked for one operation ahead: of the thread's values before the input is there
        if (!slot_wait(c, c.nw_full(), (op.nw_use - 1) & 1)) give_up(c, 2);
        const uint32_t e = (tid >> 2) * 32 + 4 * (tid & 3);
        n0 = *reinterpret_cast<const float4 *>(c.nwbuf() + e);
        n1 = *reinterpret_cast<const float4 *>(c.nwbuf() + e + 16);
    }
    const bool save = op.save_resid != 0;
    // (one round for every width taken; written as a branch, a token behind 16 384 keys of an 8-bit cache takes 1 709 us for 1 698)
#pragma unroll 1
    for (uint32_t u0 = tid; u0 < nu; u0 += 3 * TK_THREADS) {
        uint32_t u = u0, e = (u >> 2) * 32 + 4 * (u & 3), passes = (nu - u + TK_THREADS - 1) / TK_THREADS;
        constexpr uint32_t FAR = TK_THREADS * 8;  // elements from a thread's unit to its next
        uint4 a, b, a2 = make_uint4(0, 0, 0, 0), b2 = a2, a3 = a2, b3 = a2;
        if (op.in_kind == IN_EMBED) {
            const bool in_table = c.token < vocab;
            const float4 z = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            const float4 va = in_table ? embed_quad(embed, c.token, cols, e / 4) : z, vb = in_table ? embed_quad(embed, c.token, cols, e / 4 + 4) : z;
            a = make_uint4(__float_as_uint(va.x), __float_as_uint(va.y), __float_as_uint(va.z), __float_as_uint(va.w));
            b = make_uint4(__float_as_uint(vb.x), __float_as_uint(vb.y), __float_as_uint(vb.z), __float_as_uint(vb.w));
        } else {
            const uint32_t *src = in + e;
#pragma unroll 1
            for (uint32_t it = 0;; ++it) {
                a = vs_load4(src);
                b = vs_load4(src + 16);
                if (passes > 1) {
                    a2 = vs_load4(src + FAR);
                    b2 = vs_load4(src + FAR + 16);
                }
                if (passes > 2) {
                    a3 = vs_load4(src + 2 * FAR);
                    b3 = vs_load4(src + 2 * FAR + 16);
                }
                if ((vs_there(a) && vs_there(b) && vs_there(a2) && vs_there(b2) && vs_there(a3) && vs_there(b3)) || *c.abort_flag()) break;
                if (it >= POLL_LIMIT) {
                    give_up(c, 3);
                    break;
                }
            }
            __syncwarp();  // (lanes leave the wait one by one; the conversion's shuffles want the warp together)
        }
#pragma unroll 1
        for (;;) {
            float v[8] = {__uint_as_float(a.x), __uint_as_float(a.y), __uint_as_float(a.z), __uint_as_float(a.w),
                          __uint_as_float(b.x), __uint_as_float(b.y), __uint_as_float(b.z), __uint_as_float(b.w)};
            float sq = v[0] * v[0];
#pragma unroll
            for (int k = 1; k < 8; ++k) sq = fmaf(v[k], v[k], sq);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);  // (beside the conversion, whose chain is longer)
            ssq += sq;
            if (save) {  // this vector is the residual a later epilogue adds: keep this block's rows
                const uint32_t r = e - c.h0;  // wraps for rows before h0
#pragma unroll
                for (uint32_t k = 0; k < 4; ++k) {
                    if (r + k < c.hn) c.resid()[r + k] = v[k];
                    if (r + 16 + k < c.hn) c.resid()[r + 16 + k] = v[4 + k];
                }
            }
            if (normed) {
                v[0] *= n0.x; v[1] *= n0.y; v[2] *= n0.z; v[3] *= n0.w;
                v[4] *= n1.x; v[5] *= n1.y; v[6] *= n1.z; v[7] *= n1.w;
            }
            x_eighth_to_planes(c.xfb(), tk_smem + op.meta_off, u >> 2, u & 3, v, bias);
            if (--passes == 0) break;
            a = a2;
            b = b2;
            a2 = a3;
            b2 = b3;
            u += TK_THREADS;
            e += FAR;
        }
    }
    return ssq;
}

// ---- GEMV, phase 2: the rows, in tiles of sixteen (gemv_mma.cuh). The block's rows of the operation's matrices stand in one list; a
// ring slot holds 2^lrps of them, so a tile is one slot or several. Warp (slice, place) multiplies tiles place, place + row_warps, ..
// by its slice of the columns.
// Row m of a tile that lane group m (and m + 8) takes: sixteen bytes of two neighbouring groups meet in one shared-memory access, and rows
// that lie 64 bytes apart modulo 128 do not share its banks. swap: two bits of m that change places to bring such rows together.
__device__ __forceinline__ uint32_t tile_row(uint32_t g, uint32_t swap) {
    return swap == 1 ? ((g & 4) | ((g & 1) << 1) | ((g >> 1) & 1)) : (swap == 2 ? ((g & 2) | ((g & 1) << 2) | (g >> 2)) : g);
}

// A warp's work on an operation, set up before the input is waited for: its slice of x, its rows, and its first tile, whose slots have
// arrived by then (the set-up is some hundred dependent instructions, which behind the input's barrier the whole token waits for).
struct RowsJob {
    uint32_t row, last, m, g0, ng, j0, nj, k, use, rs;
    const uint8_t *ra, *rb;
};

// The tile from `row` on: wait for its slots (lane i for the i-th), find this lane's two rows.
__device__ __forceinline__ void tile_begin(const TokCtx &c, const TokOp &op, RowsJob &t, uint32_t nrows, uint32_t gslot, uint32_t row_bytes, uint32_t lane) {
    const uint32_t lrps = op.lrps;
    t.last = min(t.row + op.tile, nrows) - 1;  // (lanes past it repeat it)
    t.j0 = t.row >> lrps;
    t.nj = (t.last >> lrps) - t.j0 + 1;
    t.k = gslot + t.j0 + lane;
    t.use = __umulhi(t.k, c.p.nslot_mul);
    t.rs = t.k - t.use * c.p.nslot;
    if (lane < t.nj) {
        // A slot used twice within the operation: a warp that had no part in its earlier use could take that use's absence for this
        // one's arrival (the barrier knows two phases), so it waits until this use has been asked for.
        if (t.j0 + lane >= c.p.nslot) {
#pragma unroll 1
            for (uint32_t it = 0; *(volatile uint32_t *)c.gen(t.rs) < t.use; ++it) {
                if (*c.abort_flag()) break;
                if (it >= POLL_LIMIT) {
                    give_up(c, 2);
                    break;
                }
            }
        }
        if (!slot_wait(c, c.full(t.rs), t.use & 1)) give_up(c, 2);
    }
    __syncwarp();
    const uint32_t ia = min(t.row + t.m, t.last), ib = min(t.row + 8 + t.m, t.last), in = (1u << lrps) - 1;
    t.ra = c.ring() + __shfl_sync(0xffffffffu, t.rs, (ia >> lrps) - t.j0) * SLOT_CAP + (ia & in) * row_bytes;
    t.rb = c.ring() + __shfl_sync(0xffffffffu, t.rs, (ib >> lrps) - t.j0) * SLOT_CAP + (ib & in) * row_bytes;
}

__device__ __forceinline__ RowsJob rows_begin(const TokCtx &c, const TokOp &op, const WarpPlan &plan, uint32_t nrows, uint32_t gslot, uint32_t row_bytes) {
    RowsJob t{};
    const uint32_t lane = phase_tid() & 31;
    t.row = plan.row;
    t.g0 = plan.g0;
    t.ng = plan.g1 - plan.g0;
    t.m = tile_row(lane >> 2, op.swap);
    if (t.row < nrows) tile_begin(c, op, t, nrows, gslot, row_bytes, lane);
    return t;
}

template <int QT>
__device__ __forceinline__ void gemv_rows(const TokCtx &c, const TokOp &op, RowsJob &t, const WarpPlan &plan, uint32_t nrows, uint32_t gslot) {
    if (t.row >= nrows) return;
    const uint32_t lane = phase_tid() & 31, row_bytes = tiled_row_bytes(QT, op.cols);
    const XLane x = x_lane(c.xfb(), tk_smem + op.meta_off, reinterpret_cast<const uint8_t *>(c.zeros()), lane, t.g0);
    TileRows<QT> tr;
    tr.set(op.cols, t.g0, lane);
    float *part = c.part(op) + plan.slice;
    const uint32_t pitch = op.slices;
#pragma unroll 1
    for (;;) {
        const bool both = t.last >= t.row + 8;
        float acc_a = 0.0f, acc_b = 0.0f;
#pragma unroll 2
        for (uint32_t i = 0; i < t.ng; ++i) tr.group(t.ra, t.rb, both, x, i, acc_a, acc_b);
        // the four lanes of a row meet: lane t = 0 ends with row m, lane t = 1 with row m + 8
        float z = (lane & 1) ? acc_b : acc_a;
        z += __shfl_xor_sync(0xffffffffu, (lane & 1) ? acc_a : acc_b, 1);
        z += __shfl_xor_sync(0xffffffffu, z, 2);
        const uint32_t row = t.row + t.m + 8 * (lane & 1);
        if ((lane & 2) == 0 && row <= t.last) part[row * pitch] = z;
        __syncwarp();
        // (the warp's reads of the slots are complete: their values went into the sums stored above)
        // the last slice refills them (not after a wait that gave up: the slot's last copy may be on its way still)
        if (lane < t.nj && t.k + c.p.nslot < c.my_slots && atomicAdd(c.done(t.rs), 1u) == op.slices - 1 && !*c.abort_flag()) {
            *c.done(t.rs) = 0;
            __threadfence_block();
            *(volatile uint32_t *)c.gen(t.rs) = t.use + 1;
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            issue_slot(c, c.sdesc() + 2 * (t.j0 + lane), t.rs);
        }
        t.row += op.step;
        if (t.row >= nrows) break;
        tile_begin(c, op, t, nrows, gslot, row_bytes, lane);
    }
}

// The partial sums of a row, all loads in flight before the first addition.
__device__ __forceinline__ float sum_slices(const float *p, uint32_t n) {
    float v = 0.0f;
#pragma unroll 1
    for (uint32_t i = 0; i < n; i += 8) {
        float a[8];
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) a[k] = i + k < n ? p[i + k] : 0.0f;
        v += ((a[0] + a[1]) + (a[2] + a[3])) + ((a[4] + a[5]) + (a[6] + a[7]));
    }
    return v;
}

// ---- GEMV, phase 3: one thread per output row of this block; the result goes out as activation words.
__device__ __forceinline__ void gemv_epilogue(const TokCtx &c, const TokOp &op, const BlockRows &bo, float scale, uint32_t epoch, float *logits,
                                              unsigned long long *cand) {
    const int tid = phase_tid(), warp = tid >> 5, lane = tid & 31;
    const uint32_t S = op.slices;
    const bool swiglu = op.epilogue == EPI_SWIGLU;
    const uint32_t r0 = bo.r0, nr = bo.nout;  // segments follow one another in part[] and in the output
    const float *part = c.part(op);
    Best bst{-INFINITY, 0xffffffffu};
#pragma unroll 1
    for (uint32_t j = tid; j < nr; j += TK_THREADS) {
        float v = sum_slices(part + j * S, S) * scale;
        if (swiglu) {
            const float u = sum_slices(part + (nr + j) * S, S) * scale;
            v = (v / (1.0f + expf(-v))) * u;
        }
        if (op.epilogue == EPI_RESID) v += c.resid()[j];
        if (op.epilogue == EPI_LOGITS) {
            logits[r0 + j] = v;
            if (v > bst.v) bst = Best{v, r0 + j};
        } else {
            vs_store(op.out + c.par_cur + r0 + j, op.out + c.par_alt + r0 + j, __float_as_uint(v));
        }
    }
    if (op.epilogue == EPI_LOGITS) {  // this block's best logit for the greedy choice
        for (int o = 16; o > 0; o >>= 1) {
            Best other{__shfl_xor_sync(0xffffffffu, bst.v, o), __shfl_xor_sync(0xffffffffu, bst.i, o)};
            bst = better(bst, other);
        }
        if (lane == 0) { c.red()[RED_BEST + warp] = bst.v; c.red()[RED_INDEX + warp] = __uint_as_float(bst.i); }
        __syncthreads();
        if (tid == 0) {
#pragma unroll 1
            for (int w = 1; w < TK_WARPS; ++w) bst = better(bst, Best{c.red()[RED_BEST + w], __float_as_uint(c.red()[RED_INDEX + w])});
            ll_store(cand + 2 * c.b, __float_as_uint(bst.v), epoch);
            ll_store(cand + 2 * c.b + 1, bst.i, epoch);
        }
    }
}

template <int KV>
__global__ void __maxnreg__(128) decode_token_mma_kernel(const __grid_constant__ TokParams p) {
    TokCtx c{p};
    OpBuffer *ops_s = c.ops();

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t G = gridDim.x, b = blockIdx.x;
    c.G = G;
    c.b = b;
    c.pos = p.state[0];
    c.seq = p.state[2];
    c.par_cur = (c.seq & 1) * p.par_words;
    c.par_alt = p.par_words - c.par_cur;
    c.token = p.ids[0];
    const uint32_t slot_lo = p.slot_begin[b];
    c.my_slots = p.slot_begin[b + 1] - slot_lo;
    const uint4 *myslots = reinterpret_cast<const uint4 *>(p.slots + slot_lo);
    c.h0 = p.hidden * b / G;  // this block's rows of a hidden-size vector
    c.hn = p.hidden * (b + 1) / G - c.h0;

    // Operation oi, its warps' plans and this block's rows -> buffer oi % 2, by one warp while the operation before runs.
    auto fetch_op = [&](uint32_t oi, uint32_t buf) {
        uint4 *dst = reinterpret_cast<uint4 *>(ops_s + buf);
#pragma unroll 1
        for (uint32_t i = lane; i <= REC_WORDS; i += 32)
            cp_async16(dst + i, i < REC_WORDS ? reinterpret_cast<const uint4 *>(p.ops + oi) + i : reinterpret_cast<const uint4 *>(p.block_ops + (size_t)oi * G + b));
    };
    // (not after a wait that gave up: the norm weight before this one may be on its way still, and its barrier must not be armed anew)
    auto stage_norm = [&](const float *w, uint32_t cols) {
        if (*c.abort_flag()) return;
        *c.norms_asked() = *c.norms_asked() + 1;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        mbar_expect_tx(c.nw_full(), cols * 4);
        bulk_g2s(c.nwbuf(), w, cols * 4, c.nw_full());
    };
    if (tid == 0) {
#pragma unroll 1
        for (uint32_t s = 0; s < p.nslot; ++s) {
            mbar_init(c.full(s), 1);
            *c.done(s) = 0;
            *c.gen(s) = 0;
        }
        mbar_init(c.nw_full(), 1);
        *c.abort_flag() = 0;
        *c.norms_asked() = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (tid < 8) c.zeros()[tid] = 0;
    if (warp == 0) {
        fetch_op(0, 0);
        cp_async_wait();
    }
    __syncthreads();
    if (tid == 0) {
        uint32_t k = 0;
#pragma unroll 1
        for (; k < c.my_slots && k < p.nslot; ++k) issue_slot(c, myslots + 2 * k, k);
        if (ops_s[0].rec.op.normw) stage_norm(ops_s[0].rec.op.normw, ops_s[0].rec.op.cols);  // (later ones are staged one operation ahead)
    }

    uint32_t gslot = 0;  // list index of the current operation's first slot

#pragma unroll 1
    for (uint32_t oi = 0, buf = 0; oi < p.nops; ++oi) {
        const OpRecord &rec = ops_s[buf].rec;
        const TokOp &op = rec.op;
        const BlockRows &bo = ops_s[buf].rows;
        buf = buf + 1 == OP_BUFFERS ? 0 : buf + 1;
        if (warp == TK_WARPS - 2 && oi + 1 < p.nops) fetch_op(oi + 1, buf);
        const uint32_t epoch = c.seq * EPOCH_SPAN + oi + 1;

        TRACE(0);
        if (tid == TK_THREADS - 1 && op.next_normw) stage_norm(op.next_normw, op.next_cols);
        if (op.type == OP_GEMV) {
            const uint32_t nrows = bo.nrows, total_slots = bo.slots;
            // the descriptors this operation's refills will need, fetched by the last warp
            if (warp == TK_WARPS - 1) {
#pragma unroll 1
                for (uint32_t i = lane; i < 2 * total_slots; i += 32) {
                    const uint32_t k = 2 * (gslot + p.nslot) + i;
                    if (k < 2 * c.my_slots) cp_async16(c.sdesc() + i, myslots + k);
                }
            }
            RowsJob job = rows_begin(c, op, rec.plan[warp], nrows, gslot, tiled_row_bytes((int)op.qtype, op.cols));
            TRACE(1);
            const float ssq = gemv_input(c, op, p.embed, p.vocab);
            TRACE(3);
            if (lane == 0) c.red()[warp] = ssq;
            if (warp >= TK_WARPS - 2) cp_async_wait();  // the descriptors, the next operation: asked for before the input was waited for
            __syncthreads();
            TRACE(4);
            if (warp == TK_WARPS - 1) {  // 1 / rms of the whole input from the warps' sums, parked for the epilogue
                float tot = c.red()[lane & (TK_WARPS - 1)];
                for (int o = TK_WARPS / 2; o > 0; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
                if (lane == 0) c.red()[RED_SCALE] = op.scaled ? 1.0f / sqrtf(tot / (float)op.cols + op.eps) : 1.0f;
            }
            if (op.qtype == BRASA_Q4_0) gemv_rows<BRASA_Q4_0>(c, op, job, rec.plan[warp], nrows, gslot);
            else gemv_rows<BRASA_Q6_0>(c, op, job, rec.plan[warp], nrows, gslot);
            TRACE(7);
            gslot += total_slots;
            __syncthreads();
            TRACE(8);
            gemv_epilogue(c, op, bo, c.red()[RED_SCALE], epoch, p.logits, p.cand);
        } else {
            if (warp == TK_WARPS - 2) cp_async_wait();
            attention_op<KV>(AttnCtx{c.xfb(), c.abort_flag(), p.status, c.G, c.b, c.pos, c.par_cur, c.par_alt}, op, oi, epoch, p.heads, p.kv_heads, p.max_chunks, p.cos_t, p.sin_t, p.partials, p.attn_scale);
        }
        TRACE(11);
        __syncthreads();
        TRACE(12);
    }

    // a block that has given up waits (again with a limit) for its copies before it leaves
    if (*c.abort_flag()) {
        if (tid < (int)min(p.nslot, c.my_slots)) mbar_wait(c.full(tid), *c.gen(tid) & 1);
        if (tid == TK_THREADS - 1 && *c.norms_asked()) mbar_wait(c.nw_full(), (*c.norms_asked() - 1) & 1);
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
        if (lane == 0) { c.red()[RED_BEST + warp] = bst.v; c.red()[RED_INDEX + warp] = __uint_as_float(bst.i); }
        __syncthreads();
        if (tid == 0) {
#pragma unroll 1
            for (int w = 1; w < TK_WARPS; ++w) bst = better(bst, Best{c.red()[RED_BEST + w], __float_as_uint(c.red()[RED_INDEX + w])});
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
TokenKernel token_kernel(int32_t kv) { return kv == BRASA_KV_F16 ? decode_token_mma_kernel<BRASA_KV_F16> : decode_token_mma_kernel<BRASA_KV_Q8_0>; }

// log2 of the rows a ring slot takes: as many as fit, a tile at most. False when not one row of this width does.
bool slot_rows(int qtype, uint32_t cols, uint32_t *lrps) {
    if (cols == 0 || cols % 256 != 0) return false;
    const uint32_t row_bytes = tiled_row_bytes(qtype, cols);
    for (uint32_t l = 4;; --l) {
        if (((uint64_t)row_bytes << l) <= SLOT_CAP) {
            *lrps = l;
            return true;
        }
        if (l == 0) return false;
    }
}

// How the sixteen warps share the `rows` rows of `cols` columns that a block has: tiles of `tile` rows, row_warps of them side by side, each
// cut into `slices` of its columns. The warps' first tiles are waited for before the input is (tile_begin), so the ring must hold them
// all: row_warps x slots of a tile <= ring; where the block has more slots than the ring, a tile of several takes a third of it at most, so that
// slots are asked for while a tile is worked on. Among what fits, the split whose busiest warp has the least shared-memory traffic (a group of
// 128 columns: 10 wavefronts of x, 12 of sixteen rows), then the one with fewer partial sums. More than one slice asks for at most sum_room
// partial sums; one slice's are as many as the block has rows, however many that is (ring_layout).
constexpr uint32_t SUM_ROOM = 6144;
struct Split {
    uint32_t tile, slices, row_warps;
};
Split gemv_split(uint32_t rows, uint32_t lrps, uint32_t cols, uint32_t ring, uint32_t sum_room) {
    const uint32_t groups = cols / 128, all = (rows + (1u << lrps) - 1) >> lrps;
    Split best{1u << lrps, 1, 1};
    uint64_t least = ~0ull;
    for (uint32_t tile = TILE; tile >= 1u << lrps && tile >= 1; tile /= 2) {
        const uint32_t slots = tile >> lrps, most = slots > 1 && all > ring && 3 * slots > ring ? 0 : ring / slots, tiles = (rows + tile - 1) / tile;
        for (uint32_t s = 1; most > 0 && s <= TK_WARPS && s <= groups && (s == 1 || (uint64_t)rows * s <= sum_room); ++s) {
            const uint32_t w = std::min(most, TK_WARPS / s);
            const uint64_t cost = (uint64_t)((tiles + w - 1) / w) * ((groups + s - 1) / s) * (10 + 12 * std::max(tile, 8u) / TILE);
            if (cost < least) {
                least = cost;
                best = Split{tile, s, w};
            }
        }
    }
    return best;
}

// Splits for a ring of `ring` slots and where things lie in shared memory then; bytes of it. op_rows: the most rows a block has of an
// operation. Beside the ring lie x in fixed point from the bottom of one area, partial sums at its top, and the norm weight, over whose place
// the attention's area goes on: it is staged during o_proj and down only.
size_t ring_layout(std::vector<OpRecord> &ops, const std::vector<uint32_t> &op_rows, uint32_t G, uint32_t hidden, uint32_t ring, TokParams &p) {
    uint32_t sums = 0, last_sums = 0, max_cols = 0, max_op_slots = 0;  // sums: of the layers' operations, of the lm_head
    for (size_t i = 0; i < ops.size(); ++i) {
        TokOp &o = ops[i].op;
        if (o.type != OP_GEMV) continue;
        const Split split = gemv_split(op_rows[i], o.lrps, o.cols, ring, SUM_ROOM);
        o.tile = split.tile;
        o.slices = split.slices;
        o.step = split.row_warps * split.tile;
        uint32_t &most = o.epilogue == EPI_LOGITS ? last_sums : sums;
        most = std::max(most, op_rows[i] * o.slices);
        max_cols = std::max(max_cols, o.cols);
        max_op_slots = std::max(max_op_slots, (op_rows[i] + (1u << o.lrps) - 1) >> o.lrps);
        const uint32_t groups = o.cols / 128;
        for (uint32_t w = 0; w < TK_WARPS; ++w) {
            const uint32_t place = w / o.slices, slice = w % o.slices;
            ops[i].plan[w] = WarpPlan{place < split.row_warps ? place * o.tile : NO_ROWS, slice, groups * slice / o.slices, groups * (slice + 1) / o.slices};
        }
    }
    const size_t nw_bytes = (size_t)hidden * 4;
    size_t at = (size_t)ring * SLOT_CAP;
    auto take = [&](size_t bytes) {
        const size_t o = at;
        at = (at + bytes + 15) / 16 * 16;
        return (uint32_t)o;
    };
    const size_t x_bytes = (size_t)max_cols / 32 * X_BLOCK_BYTES, last_x = (size_t)hidden / 32 * X_BLOCK_BYTES;
    const size_t area = std::max(x_bytes + (size_t)sums * 4, last_x + (size_t)last_sums * 4) + 16;
    const size_t xf_bytes = (std::max(area, ATTN_AREA_BYTES > nw_bytes ? ATTN_AREA_BYTES - nw_bytes : 0) + 127) / 128 * 128;
    p.nslot = ring;
    p.nslot_mul = (uint32_t)(((1ull << 32) + ring - 1) / ring);
    p.off_xf = take(xf_bytes);
    p.off_nw = take(nw_bytes);
    p.off_resid = take(((size_t)(hidden + G - 1) / G + 1) * 4);
    p.off_sdesc = take((size_t)max_op_slots * sizeof(SlotDesc));
    p.off_full = take(((size_t)ring + 1) * 8);
    p.off_done = take((size_t)ring * 8);
    p.off_red = take(RED_WORDS * 4);
    p.off_ops = take(OP_BUFFERS * sizeof(OpBuffer));
    // zeros, two words; off the banks that the lanes with a share of x read at the same time (its words begin at 32 bytes)
    p.off_zeros = take(16 + 32 + 8) / 32 * 32 + 16;
    for (OpRecord &r : ops) {
        r.op.meta_off = p.off_xf + r.op.cols / 32 * X_PLANE_BYTES;
        r.op.part_off = (uint32_t)(p.off_xf + xf_bytes - (size_t)(r.op.epilogue == EPI_LOGITS ? last_sums : sums) * 4) & ~15u;
    }
    return at;
}
// The ring's length and the operations' splits want each other: the longest ring that the splits it allows leave room for (p and smem are its
// layout), 0 where there is none. A ring of one slot counts as none: 2^32 / 1 does not fit nslot_mul, and a block that waits for its
// only slot's next rows keeps no weights coming. An lm_head of millions of rows, whose partial sums lie beside the ring, shortens it that far.
uint32_t fit_ring(std::vector<OpRecord> &ops, const std::vector<uint32_t> &op_rows, uint32_t G, uint32_t hidden, uint32_t smem_optin, TokParams &p, size_t &smem) {
    for (uint32_t ring = smem_optin / SLOT_CAP; ring >= 2; --ring) {
        smem = ring_layout(ops, op_rows, G, hidden, ring, p);
        if (smem <= smem_optin) return ring;
    }
    return 0;
}
// The most rows that one of G blocks has of an operation, over its matrices.
uint32_t most_rows(const TokOp &o, uint32_t G) {
    uint32_t most = 0;
    for (uint32_t b = 0; b < G; ++b) {
        uint32_t r0, r1, first[3], nrows[3];
        block_rows(o.total_rows, o.nmat, o.rows, o.epilogue == EPI_SWIGLU, b, G, r0, r1, first, nrows);
        most = std::max(most, nrows[0] + nrows[1] + nrows[2]);
    }
    return most;
}

}  // namespace

struct brasa_token_mma {
    TokParams params{};
    size_t smem = 0;
    int32_t kv = 0;
    uint32_t grid = 0;
    std::vector<void *> device;  // allocations owned by the program
    void *vectors = nullptr;     // both copies of the activation vectors
    size_t vector_bytes = 0;
    uint32_t timeouts_seen = 0;  // the context's count of abandoned waits when the vectors were last known clean
};

extern "C" uint32_t brasa_token_ring_slots(uint32_t sm_count, uint32_t smem_bytes, uint32_t hidden, uint32_t heads, uint32_t kv_heads, uint32_t ffn, uint32_t vocab,
                                           int32_t head_qtype, int32_t kv) {
    brasa_token_model m{};
    m.hidden = hidden;
    m.heads = heads;
    m.ffn = ffn;
    m.kv = kv;
    if (sm_count == 0 || heads == 0 || kv_heads == 0 || vocab == 0 || (head_qtype != BRASA_Q4_0 && head_qtype != BRASA_Q6_0) || !brasa_token_mma_takes(m)) return 0;
    std::vector<OpRecord> ops;
    std::vector<uint32_t> op_rows;
    auto add = [&](int32_t qtype, uint32_t cols, std::initializer_list<uint32_t> rows, uint32_t epilogue) {
        OpRecord r{};
        r.op.type = OP_GEMV;
        r.op.cols = cols;
        r.op.epilogue = epilogue;
        for (uint32_t n : rows) r.op.total_rows += r.op.rows[r.op.nmat++] = n;
        if (epilogue == EPI_SWIGLU) r.op.total_rows = r.op.rows[0];
        if (!slot_rows(qtype, cols, &r.op.lrps)) return false;
        op_rows.push_back(most_rows(r.op, sm_count));
        ops.push_back(r);
        return true;
    };
    if (!add(BRASA_Q4_0, hidden, {heads * 128, kv_heads * 128, kv_heads * 128}, EPI_SCALE) || !add(BRASA_Q4_0, heads * 128, {hidden}, EPI_RESID) ||
        !add(BRASA_Q4_0, hidden, {ffn, ffn}, EPI_SWIGLU) || !add(BRASA_Q4_0, ffn, {hidden}, EPI_RESID) || !add(head_qtype, hidden, {vocab}, EPI_LOGITS))
        return 0;
    TokParams p{};
    size_t smem = 0;
    return fit_ring(ops, op_rows, sm_count, hidden, smem_bytes, p, smem);
}

bool brasa_token_mma_takes(const brasa_token_model &m) {
    if (m.kv == BRASA_KV_F32 || m.tp.world > 1 || m.hidden < MIN_HIDDEN || m.hidden > MAX_HIDDEN) return false;
    for (uint32_t cols : {m.hidden, m.heads * 128, m.ffn})
        if (cols == 0 || cols % 256 != 0 || cols > MAX_COLS) return false;
    return true;
}

void brasa_token_mma_free(brasa_token_mma *p) {
    if (!p) return;
    for (void *d : p->device) cudaFree(d);
    delete p;
}

int32_t brasa_token_mma_create(brasa_ctx *ctx, const brasa_token_model &m, brasa_token_mma **out) {
    *out = nullptr;
    std::unique_ptr<brasa_token_mma, void (*)(brasa_token_mma *)> prog(new brasa_token_mma, brasa_token_mma_free);
    prog->kv = m.kv;
    const uint32_t G = (uint32_t)ctx->sm_count;
    prog->grid = G;
    const uint32_t H = m.hidden, QD = m.heads * 128, KD = m.kv_heads * 128, F = m.ffn;
    const uint32_t C = attn_chunk(m.kv), max_chunks = (m.cache_positions + C - 1) / C;

    auto dev_alloc = [&](size_t bytes, void **ptr) -> int32_t {
        BRASA_CUDA(ctx, cudaMalloc(ptr, bytes));
        prog->device.push_back(*ptr);
        return brasa_check_cuda(ctx, cudaMemset(*ptr, 0, bytes), "cudaMemset");
    };
    auto upload = [&](const void *src, size_t bytes, void **ptr) -> int32_t {
        BRASA_TRY(dev_alloc(std::max<size_t>(bytes, 16), ptr));
        return brasa_check_cuda(ctx, cudaMemcpy(*ptr, src, bytes, cudaMemcpyHostToDevice), "cudaMemcpy");
    };
    // attention partials and argmax candidates as {value, epoch} words; every operation's output vector: two copies of par_words 4-byte
    // words, all empty at first
    void *ll_base, *vs_base;
    BRASA_TRY(dev_alloc(((size_t)m.heads * max_chunks * 130 + 2 * G) * 8, &ll_base));
    const size_t par_words = ((size_t)(QD + 2 * KD + QD + H + F + H) * m.layers.size() + 31) / 32 * 32;
    BRASA_REQUIRE(ctx, par_words < (1u << 31), "token program: activation vectors too large");
    BRASA_TRY(dev_alloc(par_words * 8, &vs_base));
    BRASA_CUDA(ctx, cudaMemset(vs_base, 0xff, par_words * 8));
    prog->vectors = vs_base;
    prog->vector_bytes = par_words * 8;
    prog->timeouts_seen = ctx->timeouts;
    uint32_t *vs_next = (uint32_t *)vs_base;
    auto vec_alloc = [&](size_t n) { uint32_t *r = vs_next; vs_next += n; return r; };

    // ---- the operations ----
    std::vector<OpRecord> ops;
    auto add_op = [&](const TokOp &o) {
        OpRecord r{};
        r.op = o;
        ops.push_back(r);
        return (int)ops.size() - 1;
    };
    auto gemv_op = [&](uint32_t nmat, const brasa_qmatrix *w, uint32_t epilogue, bool scaled, const float *normw, int in_op, bool save_resid) {
        TokOp o{};
        o.type = OP_GEMV;
        o.qtype = (uint32_t)w[0].qtype;
        o.cols = w[0].cols;
        o.nmat = nmat;
        for (uint32_t i = 0; i < nmat; ++i) {
            o.rows[i] = w[i].rows;
            o.w[i] = arg_ptr(w[i].data);
            o.total_rows += w[i].rows;
        }
        if (epilogue == EPI_SWIGLU) o.total_rows = w[0].rows;
        o.epilogue = epilogue;
        o.scaled = scaled ? 1 : 0;
        slot_rows(w[0].qtype, o.cols, &o.lrps);
        const uint32_t apart = tiled_row_bytes(w[0].qtype, o.cols) % 128;  // rows that are 64 bytes apart modulo 128: see tile_row
        o.swap = 2 * apart % 128 == 64 ? 1 : (4 * apart % 128 == 64 ? 2 : 0);
        o.in_kind = in_op < 0 ? IN_EMBED : IN_LL;
        o.save_resid = save_resid ? 1 : 0;
        o.eps = m.eps;
        o.normw = normw;
        o.in = in_op < 0 ? nullptr : ops[in_op].op.out;
        o.out = epilogue == EPI_LOGITS ? nullptr : vec_alloc(o.total_rows);
        return add_op(o);
    };
    int x_op = -1;  // operation that produced the current residual stream (-1: the embedding row)
    for (const brasa_token_layer &l : m.layers) {
        brasa_qmatrix wqkv[3] = {l.wq, l.wk, l.wv}, wgu[2] = {l.gate, l.up};
        BRASA_REQUIRE(ctx, l.wq.rows == QD && l.wk.rows == KD && l.wv.rows == KD && l.wq.cols == H && l.wo.rows == H && l.wo.cols == QD &&
                               l.gate.rows == F && l.up.rows == F && l.gate.cols == H && l.down.rows == H && l.down.cols == F,
                      "token program: unexpected matrix shape");
        TokOp a{};
        a.type = OP_ATTN;
        a.eps = m.eps;
        a.in = ops[gemv_op(3, wqkv, EPI_SCALE, true, l.attn_norm, x_op, true)].op.out;
        a.out = vec_alloc(QD);
        a.q_norm = l.q_norm;
        a.k_norm = l.k_norm;
        a.kc = l.kc;
        a.vc = l.vc;
        const int attn_op = add_op(a), o_op = gemv_op(1, &l.wo, EPI_RESID, false, nullptr, attn_op, false);
        x_op = gemv_op(1, &l.down, EPI_RESID, false, nullptr, gemv_op(2, wgu, EPI_SWIGLU, true, l.ffn_norm, o_op, true), false);
    }
    BRASA_REQUIRE(ctx, m.head.rows == m.vocab && m.head.cols == H, "token program: unexpected lm_head shape");
    gemv_op(1, &m.head, EPI_LOGITS, true, m.final_norm, x_op, false);
    BRASA_REQUIRE(ctx, (size_t)(vs_next - (uint32_t *)vs_base) <= par_words, "token program: activation vectors overran their area");
    BRASA_REQUIRE(ctx, ops.size() + 2 < EPOCH_SPAN, "token program: too many operations");
    uint32_t staged = 0;
    for (size_t i = 0; i < ops.size(); ++i) {
        TokOp &o = ops[i].op;
        if (o.normw) o.nw_use = ++staged;
        if (i + 1 < ops.size() && ops[i + 1].op.normw) {
            BRASA_REQUIRE(ctx, !o.normw, "token program: two operations in a row with a norm weight");
            o.next_normw = ops[i + 1].op.normw;
            o.next_cols = ops[i + 1].op.cols;
        }
    }

    // ---- every block's slot list, in the order the kernel consumes it, and its rows of every operation ----
    std::vector<SlotDesc> slots;
    std::vector<uint32_t> slot_begin(G + 1, 0), op_rows(ops.size(), 0);  // op_rows: the most rows a block has of an operation
    std::vector<BlockRows> block_ops(ops.size() * G, BlockRows{});
    for (uint32_t b = 0; b < G; ++b) {
        slot_begin[b] = (uint32_t)slots.size();
        for (size_t oi = 0; oi < ops.size(); ++oi) {
            const TokOp &o = ops[oi].op;
            if (o.type != OP_GEMV) continue;
            const bool swiglu = o.epilogue == EPI_SWIGLU;
            uint32_t r0, r1, first[3], nrows[3];
            block_rows(o.total_rows, o.nmat, o.rows, swiglu, b, G, r0, r1, first, nrows);
            const uint32_t rps = 1u << o.lrps, row_bytes = tiled_row_bytes((int)o.qtype, o.cols), items = nrows[0] + nrows[1] + nrows[2];
            block_ops[oi * G + b] = BlockRows{r0, swiglu ? nrows[0] : items, items, (items + rps - 1) / rps};
            for (uint32_t f = 0; f < items; f += rps) {  // rows [f, f + n) of the block's list over the matrices
                const uint32_t n = std::min(rps, items - f);
                SlotDesc d{};
                uint32_t base = 0, srcs = 0;
                for (int i = 0; i < 3; ++i) {
                    const uint32_t lo = std::max(f, base), hi = std::min(f + n, base + nrows[i]);
                    if (hi > lo) {
                        BRASA_REQUIRE(ctx, srcs < 2, "token program: a slot reaches into three matrices");
                        d.src[srcs] = o.w[i] + (size_t)(first[i] + lo - base) * row_bytes;
                        d.bytes[srcs++] = (hi - lo) * row_bytes;
                    }
                    base += nrows[i];
                }
                slots.push_back(d);
            }
            op_rows[oi] = std::max(op_rows[oi], items);
        }
    }
    slot_begin[G] = (uint32_t)slots.size();

    TokParams &p = prog->params;
    const uint32_t ring = fit_ring(ops, op_rows, G, H, (uint32_t)ctx->smem_optin, p, prog->smem);
    if (ring == 0) return BRASA_OK;  // (the vectors leave no room for weights)

    void *d_ops, *d_slots, *d_begin, *d_bops;
    BRASA_TRY(upload(ops.data(), ops.size() * sizeof(OpRecord), &d_ops));
    BRASA_TRY(upload(slots.data(), slots.size() * sizeof(SlotDesc), &d_slots));
    BRASA_TRY(upload(slot_begin.data(), slot_begin.size() * 4, &d_begin));
    BRASA_TRY(upload(block_ops.data(), block_ops.size() * sizeof(BlockRows), &d_bops));
    p.ops = (const OpRecord *)d_ops;
    p.nops = (uint32_t)ops.size();
    p.slots = (const SlotDesc *)d_slots;
    p.slot_begin = (const uint32_t *)d_begin;
    p.block_ops = (const BlockRows *)d_bops;
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
    p.partials = (unsigned long long *)ll_base;
    p.cand = p.partials + (size_t)m.heads * max_chunks * 130;
    p.par_words = (uint32_t)par_words;
    p.attn_scale = 1.0f / sqrtf(128.0f);
    p.status = ctx->status;
#ifdef BRASA_TRACE_BUILD
    p.trace = ctx->gemv_trace;
    const char *env = getenv("BRASA_TRACE_OP");
    p.trace_op = env ? (uint32_t)atoi(env) : 5;
#endif

    const TokenKernel fn = token_kernel(m.kv);
    BRASA_TRY(brasa_smem_optin(ctx, (const void *)fn, prog->smem));
    int per_sm = 0;
    BRASA_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, TK_THREADS, prog->smem));
    BRASA_REQUIRE(ctx, per_sm >= 1, "token program: the kernel does not fit an SM");
    *out = prog.release();
    return BRASA_OK;
}

int32_t brasa_token_mma_launch(brasa_cmd *cmd, brasa_token_mma *prog) {
    brasa_ctx *ctx = cmd->ctx;
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
    BRASA_CUDA(ctx, cudaLaunchKernelEx(&cfg, token_kernel(prog->kv), prog->params));
    return brasa_post_launch(cmd, "decode_token_mma");
}
