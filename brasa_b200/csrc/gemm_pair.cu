// Prefill GEMM over CTA pairs (more than 64 tokens; those up to 128 that the few-token kernel leaves): Y[t, :] = W X[t, :],
// W q4_0 in the tiled layout, X f16, f32 accumulation
// (crates/kernels/src/lib.rs:842-970 and matmul_tiled.metal:35-53: each dequantised weight is rounded to f16 before it meets X).
//
// What bounds it: the tensor cores, once both operands reach them. A 128 x 256 product out of two shared-memory operands asks
// for all 128 bytes per clock that shared memory has, and a converted weight tile has to be written there first. So
//   * the weights are the M operand, out of TENSOR memory: a lane is a weight row, a conversion thread turns its 32 codes into 16
//     registers of f16 pairs and stores them with one tcgen05.st (exact: 0x6400 | q is the half 1024 + q; minus 1032; times d in
//     f16 rounds the product once), as in the few-token kernel of gemm_tc.cu;
//   * two CTAs share one product (cta_group::2, M = 256 weight rows, N = up to 256 tokens): each holds 128 weight rows and half of
//     the tokens' X, so a CTA fetches 16 KB of X per K stage of 64 and the tensor core reads 32 bytes per clock of it;
//   * the launch is persistent and, where that is shorter, cut evenly: the (weight tile, token tile, K chunk of 256) units, in that order,
//     are split into one run per pair. 152 tiles over 74 pairs are 2.05 waves, and 20 tiles (a 2 560-row matrix at 512 tokens) not even one. A
//     run that holds a tile's whole K range stores Y; any other leaves a partial tile, at most two per run, and a dependent
//     kernel adds each shared tile's parts in K order;
//   * a thread converts the first chunk of the next tile before it drains the finished one, and frees the accumulator as soon
//     as the last of it is in registers: the tensor core goes on while results are still being stored.
// Roles: warp 0 raw weights by TMA (128 rows x (128 code + 16 scale) bytes a chunk), warp 2 X by TMA, warp 1 of the first CTA the
// products, warps 4-11 conversion and epilogue. Gate and up share a tile (64 rows of each per CTA, lanes 0-15 of a warp gate, 16-31
// the same rows of up): silu(gate) * up is formed with one shuffle per value.
// Measured (4B layer: qkv, o + residual, gate / up, down + residual; us, gemm_tc.cu's kernel in brackets): 3 584 tokens 99 (139), 70 (113),
// 322 (377), 141 (185), 1 143 (889) TFLOP/s together; 1 024 tokens 45 (52), 39 (80), 108 (145), 51 (132), 850 (505) TFLOP/s; 512 tokens 29
// (42), 30 (47), 66 (99), 38 (66). Tensor pipe active 78 % of the cycles in down; 55 % in gate / up, whose SwiGLU keeps the conversion
// threads from the next tile's chunks.
// Every wait is bounded: one that runs out raises the context's status word and a CTA-wide flag, every role leaves its loop, both
// CTAs meet at the cluster barrier, tensor memory is freed and the kernel returns.
#include <cuda.h>

#include <string.h>

#include <algorithm>
#include <type_traits>

#include "brasa_internal.h"
#include "tc_device.cuh"

using namespace brasa_dev;

namespace {

constexpr uint32_t GP_STAGE = 64, GP_CHUNK = 256;                    // K per product stage, per chunk (8 quantisation blocks)
constexpr uint32_t GP_X_STAGE = 128 * GP_STAGE * 2, GP_X_SLOT = 2 * GP_X_STAGE, GP_X_SLOTS = 4;  // a CTA's X: 128 tokens; a slot is half a chunk
constexpr uint32_t GP_CODES = 128 * 128, GP_RAW = GP_CODES + 128 * 16, GP_RAW_SLOTS = 5;
constexpr uint32_t GP_ACOL = 256, GP_TMEM = 512;                     // accumulator [0, 256), two chunks of A behind it
constexpr uint32_t GP_WAIT_LIMIT = 1u << 22;
constexpr size_t GP_SMEM = (size_t)GP_X_SLOTS * GP_X_SLOT + GP_RAW_SLOTS * GP_RAW + 1024;

struct PairMaps {
    CUtensorMap codes[3], scales[3];
};

struct PairParams {
    float *y[3];
    uint32_t rows[3];
    uint32_t tile_end[3];  // weight tiles of matrices 0..i, cumulative (256 rows each; gate and up together: 128 of each)
    uint32_t cols, tokens;
    uint32_t n, ntok;      // tokens per tile (a multiple of 32, at most 256), token tiles
    uint32_t units, gran;  // tiles x chunks; a run begins and ends at a multiple of gran units
    uint32_t *status;
    uint32_t settled;      // the weights may be asked for ahead of the dependency wait (SettledOperands)
    const float *resid;
    float *part;           // [2 x pairs][n tokens][256 rows]: slot 2 b is run b's tile that began before it, 2 b + 1 the one it leaves open
    __half *glu;
};

__host__ __device__ inline uint32_t pair_begin(uint32_t b, uint32_t pairs, uint32_t units, uint32_t gran) {
    return (uint32_t)((uint64_t)b * (units / gran) / pairs) * gran;
}

__device__ __forceinline__ uint32_t in_first_cta(const void *p) {  // the same shared-memory word of the pair's first CTA
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(smem_u32(p)));
    return r;
}
__device__ __forceinline__ void arrive_first_cta(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void commit_both(uint64_t *bar) {  // arrives at this barrier of both CTAs once the products so far are done
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)), "h"((unsigned short)3)
                 : "memory");
}
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// (A branch-free quotient, rcp.approx refined and corrected in fma, costs more than it saves: 367 us against 317 for gate / up at 3 584 tokens.)
__device__ __forceinline__ float swiglu(float g, float u) { return (g / (1.0f + expf(-g))) * u; }

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(384, 1)
    gemm_pair_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ PairMaps maps, const __grid_constant__ PairParams p) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);  // (the same offset in both CTAs)
    __shared__ uint64_t x_full[GP_X_SLOTS], x_empty[GP_X_SLOTS], a_full[2], a_empty[2], raw_full[GP_RAW_SLOTS], raw_empty[GP_RAW_SLOTS], acc_full, acc_empty;
    __shared__ uint32_t tmem_base_s, abort_s;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = blockIdx.x & 1, b = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    const uint32_t cpt = p.cols / GP_CHUNK;
    const uint32_t u_beg = pair_begin(b, pairs, p.units, p.gran), u_end = pair_begin(b + 1, pairs, p.units, p.gran), nc = u_end - u_beg;
    uint8_t *raw_base = smem + (size_t)GP_X_SLOTS * GP_X_SLOT;
    const bool glu = p.glu != nullptr;

    if (tid == 0) {
        for (uint32_t s = 0; s < GP_X_SLOTS; ++s) {
            mbar_init(&x_full[s], 1);
            mbar_init(&x_empty[s], 1);
        }
        for (uint32_t s = 0; s < 2; ++s) {
            mbar_init(&a_full[s], 16);  // one arrival per conversion warp of both CTAs
            mbar_init(&a_empty[s], 1);
        }
        for (uint32_t s = 0; s < GP_RAW_SLOTS; ++s) {
            mbar_init(&raw_full[s], 1);
            mbar_init(&raw_empty[s], 8);
        }
        mbar_init(&acc_full, 1);
        mbar_init(&acc_empty, 16);
        abort_s = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        const uint32_t ncols = GP_TMEM;
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)), "r"(ncols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_barrier();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

    auto tile_matrix = [&](uint32_t rt) { return (uint32_t)(rt >= p.tile_end[0]) + (uint32_t)(rt >= p.tile_end[1]); };
    auto tile_first = [&](uint32_t mi) { return mi == 0 ? 0u : (mi == 1 ? p.tile_end[0] : p.tile_end[1]); };
    auto issue_raw = [&](uint32_t ci) {  // codes and scales of the run's chunk ci for this CTA's 128 rows, as two boxes of 64
        const uint32_t u = u_beg + ci, t = u / cpt, kc = u - t * cpt, rt = t / p.ntok, r = ci % GP_RAW_SLOTS;
        const uint32_t mi = glu ? 0u : tile_matrix(rt);
        uint8_t *dst = raw_base + (size_t)r * GP_RAW;
        mbar_expect_tx(&raw_full[r], GP_RAW);
        const int sx = (int)(tiled_scale_off(BRASA_Q4_0, p.cols) + kc * 16);
#pragma unroll
        for (uint32_t h = 0; h < 2; ++h) {
            const uint32_t m = glu ? h : mi;
            const int row = (int)(glu ? rt * 128 + rank * 64 : (rt - tile_first(mi)) * 256 + rank * 128 + h * 64);
            tma_load_2d(dst + h * (GP_CODES / 2), &maps.codes[m], (int)(kc * 128), row, &raw_full[r]);
            tma_load_2d(dst + GP_CODES + h * 1024, &maps.scales[m], sx, row, &raw_full[r]);
        }
    };
    // Launched as a programmatic dependent: the set-up above and a model's first chunks of weights overlap the end of the kernel before
    // this one; what that kernel wrote (X, the residual, the workspace) is touched after the wait.
    const uint32_t early = p.settled ? min(GP_RAW_SLOTS, nc) : 0u;
    if (tid == 0) {
        for (uint32_t ci = 0; ci < early; ++ci) issue_raw(ci);
    }
    pdl_wait();
    pdl_launch();
    const uint32_t tmem = tmem_base_s;
    volatile uint32_t *abort_flag = &abort_s;
    auto wait = [&](uint64_t *bar, uint32_t parity) -> bool {  // bounded; false when it gave up (or another role did)
        for (uint32_t it = 0; it < GP_WAIT_LIMIT; ++it) {
            if (tc_mbar_try(bar, parity)) return true;
            if (*abort_flag) return false;
        }
        atomicExch(p.status, 4u);
        *abort_flag = 1;
        return false;
    };

    if (warp == 0) {
        if (lane == 0) {  // ---- raw weight chunks ----
            uint32_t issued = early;
            for (uint32_t ci = early; ci < nc; ++ci) {
                if (ci >= GP_RAW_SLOTS && !wait(&raw_empty[ci % GP_RAW_SLOTS], ((ci / GP_RAW_SLOTS) - 1) & 1)) break;
                issue_raw(ci);
                issued = ci + 1;
            }
            if (*abort_flag) {  // leaving early: let the copies in flight land before the block exits
                for (uint32_t ci = issued > GP_RAW_SLOTS ? issued - GP_RAW_SLOTS : 0; ci < issued; ++ci)
                    for (uint32_t it = 0; it < GP_WAIT_LIMIT && !tc_mbar_try(&raw_full[ci % GP_RAW_SLOTS], (ci / GP_RAW_SLOTS) & 1); ++it) {}
            }
        }
    } else if (warp == 2) {
        if (lane == 0) {  // ---- X: this CTA's half of the tile's tokens; both halves complete on the first CTA's barrier ----
            uint32_t kc = u_beg % cpt, tt = (u_beg / cpt) % p.ntok, issued = 0;
            const uint32_t nx = 2 * nc;
            bool ok = true;
            for (uint32_t xi = 0; xi < nx; ++xi) {
                const uint32_t s = xi % GP_X_SLOTS;
                if (xi >= GP_X_SLOTS && !(ok = wait(&x_empty[s], ((xi / GP_X_SLOTS) - 1) & 1))) break;
                if (rank == 0) mbar_expect_tx(&x_full[s], p.n * 256);  // two CTAs x two stages x n / 2 tokens x 128 bytes
                const uint32_t bar = in_first_cta(&x_full[s]);
#pragma unroll
                for (uint32_t j = 0; j < 2; ++j)
                    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                                     smem_u32(smem + (size_t)s * GP_X_SLOT + j * GP_X_STAGE)),
                                 "l"(&tmap_x), "r"((int)(kc * GP_CHUNK + ((xi & 1) * 2 + j) * GP_STAGE)), "r"((int)(tt * p.n + rank * (p.n / 2))), "r"(bar)
                                 : "memory");
                issued = xi + 1;
                if (xi & 1) {
                    if (++kc == cpt) {
                        kc = 0;
                        if (++tt == p.ntok) tt = 0;
                    }
                }
            }
            // the products that read these slots (and the arrivals that say so) are over before the CTA leaves
            for (uint32_t xi = issued > GP_X_SLOTS ? issued - GP_X_SLOTS : 0; xi < issued && ok; ++xi) ok = wait(&x_empty[xi % GP_X_SLOTS], (xi / GP_X_SLOTS) & 1);
            if (*abort_flag && rank == 0) {
                for (uint32_t xi = issued > GP_X_SLOTS ? issued - GP_X_SLOTS : 0; xi < issued; ++xi)
                    for (uint32_t it = 0; it < GP_WAIT_LIMIT && !tc_mbar_try(&x_full[xi % GP_X_SLOTS], (xi / GP_X_SLOTS) & 1); ++it) {}
            }
        }
    } else if (warp == 1) {
        if (rank == 0) {  // ---- the products of both CTAs: the warp walks the chunks and waits, one lane issues ----
            // instruction descriptor: D f32, A and B f16, both K-major, M = 256 weight rows, N = n tokens
            const uint32_t idesc = (1u << 4) | ((p.n >> 3) << 17) | ((256u >> 4) << 24);
            const uint64_t db0 = tc_desc_kmajor(smem_u32(smem));
            uint32_t kc = u_beg % cpt, seg = 0;
            bool first = true, ok = true;
            for (uint32_t c = 0; c < nc && ok; ++c) {
                const uint32_t slot = c & 1;
                const bool last = kc + 1 == cpt || c + 1 == nc;
                if (first && seg > 0) ok = wait(&acc_empty, (seg - 1) & 1);
                ok = ok && wait(&a_full[slot], (c >> 1) & 1);
                ok = __all_sync(0xffffffffu, ok);
#pragma unroll
                for (uint32_t h = 0; h < 2; ++h) {
                    const uint32_t xi = 2 * c + h, xs = xi % GP_X_SLOTS;
                    ok = ok && wait(&x_full[xs], (xi / GP_X_SLOTS) & 1);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    if (tc_elect_one()) {
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                        for (uint32_t j = 0; j < 2; ++j) {
                            const uint64_t db = db0 + (uint64_t)((xs * GP_X_SLOT + j * GP_X_STAGE) >> 4);
                            const uint32_t a0 = tmem + GP_ACOL + 128 * slot + 32 * (2 * h + j);
#pragma unroll
                            for (uint32_t ks = 0; ks < 4; ++ks) {  // A: 16 halves of K = 8 columns of tensor memory; B: 32 bytes further along K
                                const uint32_t acc = (!first || h > 0 || j > 0 || ks > 0) ? 1u : 0u;
                                asm volatile(
                                    "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                                    "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem),
                                    "r"(a0 + ks * 8), "l"(db + (uint64_t)(ks * 2)), "r"(idesc), "r"(acc)
                                    : "memory");
                            }
                        }
                        commit_both(&x_empty[xs]);
                        if (h == 1) {
                            commit_both(&a_empty[slot]);
                            if (last) commit_both(&acc_full);
                        }
                    }
                    __syncwarp();
                }
                seg += last;
                first = last;
                if (++kc == cpt) kc = 0;
            }
        }
    } else if (warp >= 4) {
        // ---- conversion and epilogue ----
        const uint32_t q = warp & 3, th = (warp - 4) >> 2;  // lane quarter of tensor memory; block of the stage, half of the tokens
        const uint32_t wr = glu ? (lane >> 4) * 64 + q * 16 + (lane & 15) : 32 * q + lane, r8 = wr & 7;  // the lane's row among the CTA's 128
        const uint32_t coff = wr * 128, soff = GP_CODES + wr * 16 + th * 2;
        const uint32_t t_lane = tmem + ((q * 32u) << 16), a_lane = t_lane + GP_ACOL + 16 * th, half = p.n / 2;
        const uint32_t a_full_at = in_first_cta(&a_full[0]), acc_empty_at = in_first_cta(&acc_empty);
        bool ok = true;
        // reads tile t's accumulator (lane = weight row, column = token): Y when the run held all of its chunks, else a partial tile
        auto epilogue = [&](uint32_t t, uint32_t k0, uint32_t len, uint32_t seg) {
            ok = ok && wait(&acc_full, seg & 1);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) return;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t rt = t / p.ntok, tt = t - rt * p.ntok, tok = tt * p.n + th * half;  // the thread's first token
            const uint32_t live = tok < p.tokens ? min(half, p.tokens - tok) : 0u;
            const uint32_t mi = glu ? 0u : tile_matrix(rt), yrows = mi == 0 ? p.rows[0] : (mi == 1 ? p.rows[1] : p.rows[2]);
            float *ymat = mi == 0 ? p.y[0] : (mi == 1 ? p.y[1] : p.y[2]);
            const size_t at = (size_t)tok * yrows + (rt - tile_first(mi)) * 256 + rank * 128 + 32 * q + lane;
            // 64 tokens at a time: the whole half would take 128 registers, and spilled ones come back from L2 (shared memory leaves
            // no first-level cache to speak of)
#pragma unroll 1
            for (uint32_t c0 = 0; c0 < half; c0 += 64) {
                uint32_t v[2][32];
#pragma unroll
                for (uint32_t k = 0; k < 2; ++k)
                    if (c0 + 32 * k < half) tc_ld32(t_lane + th * half + c0 + 32 * k, v[k]);
                if (c0 + 64 >= half) {
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) arrive_first_cta(acc_empty_at);  // the next tile's products may overwrite it
                }
                const uint32_t left = live > c0 ? live - c0 : 0u;
                if (len < cpt) {
                    float *dst = p.part + ((size_t)(2 * b + (k0 == 0)) * p.n + th * half + c0) * 256 + rank * 128 + 32 * q + lane;
#pragma unroll
                    for (uint32_t k = 0; k < 2; ++k)
#pragma unroll
                        for (uint32_t i = 0; i < 32; ++i)
                            if (32 * k + i < left) dst[(32 * k + i) * 256] = __uint_as_float(v[k][i]);
                } else if (glu) {
                    __half *dst = p.glu + (size_t)(tok + c0 + (lane >> 4)) * p.rows[0] + rt * 128 + rank * 64 + q * 16 + (lane & 15);
                    // (a column without a token holds zeros or what was left there, and a quotient of those takes the division's slow path:
                    // 256 x 256 at 65 tokens 11.9 us with them, 10.2 without; 9 728 x 2 560 at 100 28.5, 27.5)
                    auto emit = [&](auto partial) {
#pragma unroll
                        for (uint32_t k = 0; k < 2; ++k) {
                            if (partial && 32 * k >= left) break;
#pragma unroll
                            for (uint32_t i = 0; i < 32; i += 2) {  // lanes 0-15: gate of these rows, and token i's result; 16-31: up, token i + 1's
                                const float lo = !partial || 32 * k + i < left ? __uint_as_float(v[k][i]) : 1.0f;
                                const float hi = !partial || 32 * k + i + 1 < left ? __uint_as_float(v[k][i + 1]) : 1.0f;
                                const float got = __shfl_xor_sync(0xffffffffu, lane < 16 ? hi : lo, 16);
                                const float o = lane < 16 ? swiglu(lo, got) : swiglu(got, hi);
                                if (!partial || 32 * k + i + (lane >> 4) < left) dst[(size_t)(32 * k + i) * p.rows[0]] = __float2half_rn(o);
                            }
                        }
                    };
                    if (left >= 64) emit(std::false_type{});
                    else emit(std::true_type{});
                } else {
                    float *dst = ymat + at + (size_t)c0 * yrows;
                    const float *src = p.resid ? p.resid + at + (size_t)c0 * yrows : nullptr;
#pragma unroll
                    for (uint32_t k = 0; k < 2; ++k)
#pragma unroll
                        for (uint32_t i0 = 0; i0 < 32; i0 += 16) {
                            float r[16];
                            if (src) {
#pragma unroll
                                for (uint32_t i = 0; i < 16; ++i) r[i] = 32 * k + i0 + i < left ? src[(size_t)(32 * k + i0 + i) * yrows] : 0.0f;
                            }
#pragma unroll
                            for (uint32_t i = 0; i < 16; ++i)
                                if (32 * k + i0 + i < left) dst[(size_t)(32 * k + i0 + i) * yrows] = src ? r[i] + __uint_as_float(v[k][i0 + i]) : __uint_as_float(v[k][i0 + i]);
                        }
                }
            }
        };
        uint32_t t = u_beg / cpt, kc = u_beg - t * cpt, k0 = kc, seg = 0, rslot = 0, rph = 0;
        const __half2 bias = __half2half2(__ushort_as_half((unsigned short)0x6408));  // 1024 + 8
        for (uint32_t c = 0; c < nc && ok; ++c) {
            const uint32_t slot = c & 1;
            ok = wait(&raw_full[rslot], rph);
            if (c >= 2) ok = ok && wait(&a_empty[slot], ((c >> 1) - 1) & 1);
            ok = __all_sync(0xffffffffu, ok);  // the tensor-memory stores need the whole warp
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint8_t *raw = raw_base + (size_t)rslot * GP_RAW;
            uint4 cws[4];  // (all the loads first: a tensor-memory store orders what follows it behind it)
            unsigned short scs[4];
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) {
                cws[j] = *reinterpret_cast<const uint4 *>(raw + coff + (((2 * j + th) ^ r8) << 4));
                scs[j] = *reinterpret_cast<const unsigned short *>(raw + soff + j * 4);
            }
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) {
                const __half2 d2 = __half2half2(__ushort_as_half(scs[j]));
                const uint32_t words[4] = {cws[j].x, cws[j].y, cws[j].z, cws[j].w};
                uint32_t e[16];  // pairs of consecutive columns: elements 0..15 are the low nibbles of bytes 0..15, 16..31 the high nibbles
#pragma unroll
                for (int w4 = 0; w4 < 4; ++w4) {
                    const uint32_t wv = words[w4] & 0x0F0F0F0Fu, wh = (words[w4] >> 4) & 0x0F0F0F0Fu;
                    auto deq = [&](uint32_t two) {  // 1024 + q in each half -> f16(d (q - 8))
                        const __half2 h = __hmul2(__hsub2(*reinterpret_cast<__half2 *>(&two), bias), d2);
                        return *reinterpret_cast<const uint32_t *>(&h);
                    };
                    e[2 * w4] = deq(__byte_perm(wv, 0x64646464u, 0x4140));
                    e[2 * w4 + 1] = deq(__byte_perm(wv, 0x64646464u, 0x4342));
                    e[8 + 2 * w4] = deq(__byte_perm(wh, 0x64646464u, 0x4140));
                    e[8 + 2 * w4 + 1] = deq(__byte_perm(wh, 0x64646464u, 0x4342));
                }
                asm volatile(
                    "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(
                        a_lane + 128 * slot + 32 * j),
                    "r"(e[0]), "r"(e[1]), "r"(e[2]), "r"(e[3]), "r"(e[4]), "r"(e[5]), "r"(e[6]), "r"(e[7]), "r"(e[8]), "r"(e[9]), "r"(e[10]), "r"(e[11]),
                    "r"(e[12]), "r"(e[13]), "r"(e[14]), "r"(e[15])
                    : "memory");
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                arrive_first_cta(a_full_at + 8 * slot);
                tc_mbar_arrive(&raw_empty[rslot]);
            }
            rslot = rslot + 1 == GP_RAW_SLOTS ? 0 : rslot + 1;
            rph ^= (rslot == 0);
            if (kc == 0 && c > 0) {  // this chunk opened a tile: now the one before it
                epilogue(t - 1, k0, cpt - k0, seg);
                ++seg;
                k0 = 0;
            }
            if (++kc == cpt) {
                kc = 0;
                ++t;
            }
        }
        if (nc > 0) {
            const uint32_t t_last = (u_end - 1) / cpt, k_end = u_end - t_last * cpt;
            epilogue(t_last, k0, k_end - k0, seg);
            for (uint32_t c = nc > 2 ? nc - 2 : 0; c < nc && ok; ++c) ok = wait(&a_empty[c & 1], (c >> 1) & 1);  // (the last arrivals have landed)
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_barrier();  // neither CTA leaves while the other may still read its shared memory or signal it
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t ncols = GP_TMEM;
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncols) : "memory");
    }
}

// Y (or silu(gate) * up) of every tile that several runs worked on: block (i, y) takes the tile that run i + 1 goes on with, when that
// run is the first to do so, and every grid.y-th part of it. Parts are added in K order.
__global__ void __launch_bounds__(256) gemm_pair_sum_kernel(const __grid_constant__ PairParams p, uint32_t pairs) {
    pdl_wait();
    pdl_launch();
    const uint32_t b = blockIdx.x + 1, cpt = p.cols / GP_CHUNK, u = pair_begin(b, pairs, p.units, p.gran);
    const uint32_t t = u / cpt;
    if (u % cpt == 0 || u >= p.units || pair_begin(b - 1, pairs, p.units, p.gran) > t * cpt) return;
    uint32_t end = b + 1;
    while (end < pairs && pair_begin(end, pairs, p.units, p.gran) < (t + 1) * cpt) ++end;
    const uint32_t rt = t / p.ntok, tok0 = (t - rt * p.ntok) * p.n, live = min(p.n, p.tokens - tok0);
    const size_t tile = (size_t)p.n * 256;
    auto sum = [&](size_t at) {
        float4 a = __ldcg(reinterpret_cast<const float4 *>(p.part + (size_t)(2 * (b - 1) + 1) * tile + at));
#pragma unroll 4
        for (uint32_t z = b; z < end; ++z) {
            const float4 v = __ldcg(reinterpret_cast<const float4 *>(p.part + (size_t)(2 * z) * tile + at));
            a.x += v.x;
            a.y += v.y;
            a.z += v.z;
            a.w += v.w;
        }
        return a;
    };
    if (p.glu) {
        for (uint32_t i = blockIdx.y * 256 + threadIdx.x; i < live * 32; i += gridDim.y * 256) {
            const uint32_t n = i >> 5, g = (i & 31) * 4;  // four rows of the tile's 128 of gate
            const size_t at = (size_t)n * 256 + (g >> 6) * 128 + ((g >> 4) & 3) * 32 + (g & 15);
            const float4 a = sum(at), c = sum(at + 16);
            const __half2 lo = __floats2half2_rn(swiglu(a.x, c.x), swiglu(a.y, c.y)), hi = __floats2half2_rn(swiglu(a.z, c.z), swiglu(a.w, c.w));
            *reinterpret_cast<uint2 *>(p.glu + (size_t)(tok0 + n) * p.rows[0] + rt * 128 + g) =
                make_uint2(*reinterpret_cast<const uint32_t *>(&lo), *reinterpret_cast<const uint32_t *>(&hi));
        }
        return;
    }
    const uint32_t mi = (uint32_t)(rt >= p.tile_end[0]) + (uint32_t)(rt >= p.tile_end[1]);
    const uint32_t first = mi == 0 ? 0u : (mi == 1 ? p.tile_end[0] : p.tile_end[1]), yrows = mi == 0 ? p.rows[0] : (mi == 1 ? p.rows[1] : p.rows[2]);
    float *ymat = mi == 0 ? p.y[0] : (mi == 1 ? p.y[1] : p.y[2]);
    for (uint32_t i = blockIdx.y * 256 + threadIdx.x; i < live * 64; i += gridDim.y * 256) {
        const uint32_t n = i >> 6, r = (i & 63) * 4;
        float4 a = sum((size_t)n * 256 + r);
        const size_t at = (size_t)(tok0 + n) * yrows + (rt - first) * 256 + r;
        if (p.resid) {
            const float4 x = *reinterpret_cast<const float4 *>(p.resid + at);
            a = make_float4(x.x + a.x, x.y + a.y, x.z + a.z, x.w + a.w);
        }
        *reinterpret_cast<float4 *>(ymat + at) = a;
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                  const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);
EncodeTiledFn encode_tiled() {
    static EncodeTiledFn fn = [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) f = nullptr;
        return (EncodeTiledFn)f;
    }();
    return fn;
}

}  // namespace

// How a product is cut: token tiles of equal size (as few of up to `most` as hold the tokens), runs of whole tiles or even ones.
struct PairPlan {
    uint32_t n, ntok, units, pairs, gran;
    double cost;
};
static PairPlan pair_plan(uint32_t sm_pairs, uint32_t tiles, uint32_t cpt, uint32_t tokens, uint32_t most, bool glu) {
    PairPlan p{};
    p.ntok = (tokens + most - 1) / most;
    p.n = ((tokens + p.ntok - 1) / p.ntok + 31) / 32 * 32;
    p.units = tiles * p.ntok * cpt;
    p.pairs = std::min(sm_pairs, p.units);  // no run is empty
    p.gran = 1;
    // Runs of whole tiles, or even ones that cut tiles: which is shorter, in chunks. Cut tiles cost their parts' way through memory and the
    // kernel behind: 10 chunks' time for 256 tokens a tile, 7 for 128; 4 where that kernel also takes SwiGLU off the blocks. 3 584 tokens: qkv 99 us
    // whole, 109 cut; o 70, 83; down 141, 156; gate / up 322, 320. 512 tokens: qkv 29, 35; gate / up 73, 66.
    uint32_t chunks = (p.units + p.pairs - 1) / p.pairs;
    const uint32_t whole = (tiles * p.ntok + p.pairs - 1) / p.pairs * cpt;
    const bool cut = whole > chunks + 4 + (glu ? 0 : p.n / 42);
    if (!cut) {
        chunks = whole;
        p.gran = cpt;
        p.pairs = std::min(sm_pairs, p.units / cpt);
    }
    p.cost = chunks * (1.0 + p.n / 1100.0) + p.n / 140.0 + (cut ? p.n / 20.0 : 0.0);
    return p;
}

// Token tiles of the width, 256 down to 64, that ends soonest. The costs are in chunks and follow 670 products of 14 matrices, of whose best width
// they miss 0.3 % on average: a chunk takes a little longer the more tokens there are (the conversion of its weights takes the most of it), and
// so does the last tile's way out, the more so through a workspace. A product of few tiles, whose runs are a handful of chunks, is its way in
// and out, and more tiles cost it nothing while pairs are idle; one of little more than a wave of tiles gets by with a chunk less. us with 256,
// 128 and 64: 256 x 256, 256 tokens 12.0, 9.1, 8.4; 1 024 x 2 560 22.0, 16.6, 14.5; 2 560 x 2 560, 512 tokens 22.6, 18.7, 25.4; 1 000 tokens
// 25.0, 27.9, 38.4; 2 560 x 9 728, 256 tokens 30.0, 25.9, 33.4; 512 tokens 34.2, 36.3, 55.4; 2 560 x 512, 2 000 tokens 22.1, 20.7, 27.7, with
// 160 19.4. Up to 96 tokens one tile holds them all (two of 64 cost 3 to 13 % more).
static PairPlan pair_plan(uint32_t sm_pairs, uint32_t tiles, uint32_t cpt, uint32_t tokens, bool glu) {
    PairPlan best = pair_plan(sm_pairs, tiles, cpt, tokens, 256, glu);
    for (uint32_t most = 224; most >= 64 && tokens > 96; most -= 32) {
        const PairPlan p = pair_plan(sm_pairs, tiles, cpt, tokens, most, glu);
        if (p.cost < best.cost) best = p;
    }
    return best;
}

// True when brasa_gemm_pair_launch takes the product (every matrix q4_0 tiled and 16-byte aligned): rows in whole tiles (256; gate
// and up 128 each) and more tokens than the few-token kernel's tile of 64; up to 128 tokens that kernel has the first choice
// (brasa_gemm_tc_few_tokens). gemm_tc_kernel keeps the shapes whose rows are an odd number of 128: a 4B layer's products at 200 tokens take
// 159 us here and 174 there, at 1 024 1.6 times as long there.
bool brasa_gemm_pair_takes(const brasa_qmatrix *ws, uint32_t count, uint32_t tokens, bool glu) {
    if (tokens <= 64 || encode_tiled() == nullptr) return false;
    uint64_t tiles = 0;
    for (uint32_t i = 0; i < count; ++i) {
        if (ws[i].qtype != BRASA_Q4_0 || ws[i].layout != BRASA_LAYOUT_TILED || ws[i].cols % GP_CHUNK || ws[i].rows % (glu ? 128 : 256)) return false;
        if ((reinterpret_cast<uintptr_t>(arg_ptr(ws[i].data)) & 15) != 0) return false;
        tiles += ws[i].rows / (glu ? 128 : 256);
    }
    return tiles * ((tokens + 63ull) / 64) * (ws[0].cols / GP_CHUNK) < (1ull << 31);
}

// True when gemm_tc_kernel is ahead on a product that the pairs take: more than a wave of tiles of few K chunks. The conversion threads drain
// a tile themselves, and behind a handful of chunks the products wait for that; gemm_tc_kernel has twice the blocks, each with a tile of its
// own. Both sides in us by waves (of pairs, of SMs) and chunks a tile, plain and SwiGLU, from 250 products of 256 to 1 536 columns. us, pairs
// and gemm_tc: SwiGLU of 4 096 x 256 at 1 024 tokens 25.6, 18.9; x 512 29.5, 22.9; x 1 024 34.2, 30.0; at 8 192 tokens 200, 193; 2 560 x 512 at
// 3 584 52.2, 42.6; plain 4 096 x 256 at 2 048 18.8, 16.4; x 512 22.8, 20.3. A product with a residual is the pairs' everywhere (0.74 at most).
bool brasa_gemm_pair_behind(const brasa_ctx *ctx, const brasa_qmatrix *ws, uint32_t count, uint32_t tokens, bool resid, bool glu) {
    const uint32_t sms = (uint32_t)ctx->sm_count, cpt = ws[0].cols / GP_CHUNK;
    if (resid || (!glu && cpt > 3)) return false;
    uint32_t tiles = 0;
    for (uint32_t i = 0; i < (glu ? 1 : count); ++i) tiles += ws[i].rows / (glu ? 128 : 256);
    const uint32_t units = tiles * ((tokens + 255) / 256), pair_waves = (units + sms / 2 - 1) / (sms / 2), sm_waves = (units + sms - 1) / sms;
    if (pair_waves < 2) return false;
    const double pairs = glu ? 6.6 + pair_waves * (8.4 + 1.3 * cpt) : 4.7 + 1.35 * cpt + pair_waves * (5.15 + 1.25 * cpt);
    const double tc = glu ? 3.2 + sm_waves * (12.0 + 3.6 * cpt) : 3.7 + sm_waves * (9.05 + 3.7 * cpt);
    return 1.05 * tc < pairs;
}

// Y_i = W_i X (+ resid, one matrix), or out = f16(silu(W_0 X) * (W_1 X)): the arguments of brasa_gemm_tc_launch.
int32_t brasa_gemm_pair_launch(brasa_cmd *cmd, uint32_t count, const brasa_qmatrix *ws, const __half *x, float *const *ys, uint32_t tokens, const float *resid,
                               __half *glu) {
    brasa_ctx *ctx = cmd->ctx;
    PairParams p{};
    PairMaps maps;
    memset(&maps, 0, sizeof maps);
    const uint32_t cols = ws[0].cols, cpt = cols / GP_CHUNK, sm_pairs = (uint32_t)ctx->sm_count / 2;
    uint32_t tiles = 0;
    for (uint32_t i = 0; i < 3; ++i) {
        if (i < count) {
            p.y[i] = ys ? ys[i] : nullptr;
            p.rows[i] = ws[i].rows;
            if (!glu) tiles += ws[i].rows / 256;
        }
        if (glu) tiles = ws[0].rows / 128;
        p.tile_end[i] = tiles;
    }
    const PairPlan plan = pair_plan(sm_pairs, tiles, cpt, tokens, glu != nullptr);
    uint32_t pairs = plan.pairs;
    p.n = plan.n;
    p.ntok = plan.ntok;
    p.units = plan.units;
    p.gran = plan.gran;
    p.cols = cols;
    p.tokens = tokens;
    p.status = ctx->status;
    p.settled = ctx->settled;
    p.resid = resid;
    p.glu = glu;
    BRASA_REQUIRE(ctx, (reinterpret_cast<uintptr_t>(x) & 15) == 0, "gemm: misaligned x");
    bool shared = false;  // some run begins inside a tile
    for (uint32_t b = 1; b < pairs; ++b) shared = shared || pair_begin(b, pairs, p.units, p.gran) % cpt != 0;
    if (shared) {
        // the most that any product asks for (38.8 MB on 148 SMs), so that prompts of growing length allocate and synchronise once
        const size_t need = (size_t)2 * pairs * p.n * 256 * sizeof(float);
        if (ctx->gemm_part_bytes < need && !ctx->capturing) brasa_workspace_had(ctx, (void **)&ctx->gemm_part, &ctx->gemm_part_bytes, brasa_gemm_part_most(ctx));
        if (ctx->gemm_part_bytes >= need) p.part = ctx->gemm_part;
        else {  // no workspace (a graph is being recorded, or no memory is left): runs of whole tiles
            p.gran = cpt;
            pairs = std::min(sm_pairs, p.units / cpt);
            shared = false;
        }
    }
    CUtensorMap tmap;
    const cuuint32_t estr[2] = {1, 1};
    {
        const cuuint64_t dims[2] = {cols, tokens}, strides[1] = {(cuuint64_t)cols * 2};
        const cuuint32_t box[2] = {GP_STAGE, p.n / 2};
        const CUresult r = encode_tiled()(&tmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<__half *>(x), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                          CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return brasa_fail(ctx, BRASA_ECUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
    }
    const uint32_t rb = tiled_row_bytes(BRASA_Q4_0, cols);
    for (uint32_t i = 0; i < count; ++i) {
        const cuuint64_t dims[2] = {rb, ws[i].rows}, strides[1] = {rb};
        const cuuint32_t cbox[2] = {128, 64}, sbox[2] = {16, 64};
        CUresult r = encode_tiled()(&maps.codes[i], CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, arg_ptr(ws[i].data), dims, strides, cbox, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r == CUDA_SUCCESS)
            r = encode_tiled()(&maps.scales[i], CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, arg_ptr(ws[i].data), dims, strides, sbox, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                               CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return brasa_fail(ctx, BRASA_ECUDA, "cuTensorMapEncodeTiled failed for the weights (%d)", (int)r);
    }
    BRASA_TRY(brasa_smem_optin(ctx, (const void *)gemm_pair_kernel, GP_SMEM));
    BRASA_CUDA(ctx, brasa_launch_dependent(ctx, gemm_pair_kernel, dim3(2 * pairs), dim3(384), GP_SMEM, tmap, maps, p));
    BRASA_TRY(brasa_post_launch(cmd, "gemm_pair"));
    if (!shared) return BRASA_OK;
    BRASA_CUDA(ctx, brasa_launch_dependent(ctx, gemm_pair_sum_kernel, dim3(pairs - 1, 16), dim3(256), 0, p, pairs));
    return brasa_post_launch(cmd, "gemm_pair_sum");
}
