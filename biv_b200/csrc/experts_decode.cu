// Grouped expert products for decode-sized groups with float weights: gate+up with the
// SwiGLU (and, for a quantised down type, the Q8 re-quantisation of its output) fused, then down.
// Reference: dense_ffn (engine/src/model.rs:1119-1126) over matmul
// (engine/src/ops.rs:84-127) and the per-type dots (engine/src/quant.rs:
// 599-686 scalar, 1369-1533 AVX2), for each expert's token list
// (model.rs:875-889) and for the shared expert (model.rs:890-896).
//
// This file holds the float weight types (BF16, F16, F32 weights meeting f32 activations,
// quant.rs:483-521, 1229-1281) and the choice of kernel per product; the quantised types'
// kernel is experts_quant.cu.  No atomics on data: results are run-to-run identical.
#include <cuda_fp16.h>

#include <algorithm>
#include <cstdlib>

#include "common.cuh"
#include "formats.cuh"
#include "tcgen05.cuh"
#include "launch.cuh"

namespace bivmoe {

constexpr int EX_TT = 8;                       // tokens per tile
constexpr uint32_t EX_WAIT_LIMIT = 1u << 16;   // bounded mbarrier wait: tries that may sleep wait_hint_ns each

enum { MODE_GATEUP = 0, MODE_DOWN = 1 };

struct ExpertArgs {
    DevTiles w, sh;        // the routed experts' and the shared expert's tiles for this product
    // activations by position, slice-major (common.cuh): rows of h for GATEUP, of mid for DOWN
    const float* x_f32;
    int act_rows;          // R
    float* out;            // GATEUP: mid f32, slice-major; DOWN: pair_out [R][rows]
    uint8_t* out_t;        // GATEUP with a quantised down type: the Q8 records of mid
    const int4* tile_desc;    // {expert (n_expert: shared), first position, tokens, 0}
    const int32_t* n_tiles;   // [0] all tiles, [1] tiles of the shared group (they come first)
    int32_t* status;
    int n_expert;
    int tiles_mode;        // 0: every tile, 1: skip the shared group's, 2: only the shared group's
    int chunks;            // row chunks per group in this launch
    uint32_t wait_hint_ns; // how long one mbarrier try may sleep
};

// ---------------------------------------------------------------------------
// PTX helpers: mbarrier, bulk copy (TMA, untiled form)
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity, uint32_t hint_ns) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity), "r"(hint_ns)   // may sleep up to hint_ns per try
        : "memory");
    return ok != 0;
}
// One look, without blocking: has the phase of parity `parity` completed?
__device__ __forceinline__ bool mbar_test_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Waits for a phase with an iteration limit; false when it gave up.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, uint32_t hint_ns) {
    for (uint32_t i = 0; i < EX_WAIT_LIMIT; i++)
        if (mbar_try_wait(bar, parity, hint_ns)) return true;
    return false;
}
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
            "r"(smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ void fence_proxy_async() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
template <int TY> struct Fmt;

// ---- BF16, F16 and F32 weights meet f32 activations (quant.rs:483-521, 1229-1281):
//      f32 multiply-adds, a lane per weight row, activations read as broadcasts ----
template <int TY> struct FmtFloat {
    static constexpr int ELEMS = 64, SL = TY == BIVMOE_F32 ? 256 : 128, MINB = TY == BIVMOE_F32 ? 3 : 4;
    static constexpr int PER_UNIT = TY == BIVMOE_F32 ? 4 : 8;   // values in a 16-byte unit
    __device__ static void widen(const uint4& v, float (&w)[8]) {
        if (TY == BIVMOE_BF16) {
            w[0] = __uint_as_float(v.x << 16); w[1] = __uint_as_float(v.x & 0xFFFF0000u);
            w[2] = __uint_as_float(v.y << 16); w[3] = __uint_as_float(v.y & 0xFFFF0000u);
            w[4] = __uint_as_float(v.z << 16); w[5] = __uint_as_float(v.z & 0xFFFF0000u);
            w[6] = __uint_as_float(v.w << 16); w[7] = __uint_as_float(v.w & 0xFFFF0000u);
        } else if (TY == BIVMOE_F16) {
            const uint32_t p[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float2 f = __half22float2(*(const __half2*)&p[i]);
                w[2 * i] = f.x;
                w[2 * i + 1] = f.y;
            }
        } else {
            w[0] = __uint_as_float(v.x); w[1] = __uint_as_float(v.y);
            w[2] = __uint_as_float(v.z); w[3] = __uint_as_float(v.w);
            w[4] = w[5] = w[6] = w[7] = 0.0f;
        }
    }
    // `wrow`: this lane's row (tile + row*16); acc[t] += dot(row slice, token t)
    __device__ static void compute_f32(const uint8_t* wrow, const float* xf, int cnt,
                                       float (&acc)[EX_TT]) {
#pragma unroll 2
        for (int u = 0; u < SL / 16; u++) {
            float w[8];
            widen(*(const uint4*)(wrow + 2048 * u), w);
#pragma unroll
            for (int t = 0; t < EX_TT; t++) {
                if (t < cnt) {
                    const float4* xp = (const float4*)(xf + t * ELEMS + PER_UNIT * u);
                    const float4 x0 = xp[0];
                    float s = acc[t];
                    s = fmaf(w[0], x0.x, s); s = fmaf(w[1], x0.y, s); s = fmaf(w[2], x0.z, s);
                    s = fmaf(w[3], x0.w, s);
                    if (PER_UNIT == 8) {
                        const float4 x1 = xp[1];
                        s = fmaf(w[4], x1.x, s); s = fmaf(w[5], x1.y, s);
                        s = fmaf(w[6], x1.z, s); s = fmaf(w[7], x1.w, s);
                    }
                    acc[t] = s;
                }
            }
        }
    }
};
template <> struct Fmt<BIVMOE_BF16> : FmtFloat<BIVMOE_BF16> {};
template <> struct Fmt<BIVMOE_F16> : FmtFloat<BIVMOE_F16> {};
template <> struct Fmt<BIVMOE_F32> : FmtFloat<BIVMOE_F32> {};

// ---------------------------------------------------------------------------
// The kernel.  One block per SM: G consumer groups of four warps and one producer
// warp.  A group works on its own items - a tile of up to 8 tokens times one chunk
// (gate+up) or two chunks (down) - and owns a two-slot ring of stages (one K-slice of a
// chunk's 128 rows plus the tile's activation record) that lane g of the producer warp
// keeps full: the lane takes the group's next item from the block's own list - item i of
// a launch belongs to block i mod gridDim.x, so every SM gets the same number of (equal)
// items give or take one, and the groups of a block share its list through a counter in
// shared memory - and issues its stages as slots come free.  (Claiming from one global
// counter instead left the SMs unevenly loaded at the end: measured 33 k to 69 k active
// cycles per SM, because an SM's groups share its issue slots and an SM that happened to
// claim four late items took twice as long over them as one that claimed two.)  A consumer warp waits for a slot,
// computes its 32 rows of the stage, and hands the slot back with one mbarrier arrive:
// the consumer warps never meet per stage and carry no pipeline state - everything a
// stage needs to know (tile, chunk, whether it opens or closes an accumulation) comes in
// a small descriptor the producer writes beside it.  The groups of a block share nothing
// but the producer warp, so one group's epilogue overlaps the others' products.
// The producer lanes never block: they stay together and poll their groups' slots in turn,
// so no lane's wait holds up the lanes of the other groups.
// Every wait is bounded; a wait that gives up records BIVMOE_ERR_TIMEOUT (and which wait
// it was) in the status words and raises a block-wide flag on which every role leaves its
// loop (the producer first waits, bounded again, for its copies still in flight).
template <int TY>
__host__ __device__ constexpr int act_stage_bytes() {
    return EX_TT * Fmt<TY>::ELEMS * 4;
}
template <int TY>
__host__ __device__ constexpr int stage_bytes() {
    return kChunkRows * Fmt<TY>::SL + act_stage_bytes<TY>();
}
constexpr int EX_SLOTS = 2;               // ring slots per group
constexpr int EX_HEAD = 1024;             // barriers, abort flag, stage descriptors
constexpr int EX_SMEM_MAX = 227 * 1024;
template <int TY>
__host__ __device__ constexpr int smem_bytes() {
    constexpr int G = Fmt<TY>::MINB;
    return EX_HEAD + G * EX_TT * 64 * 4 + G * EX_SLOTS * stage_bytes<TY>();
}

struct StageDesc {      // what the producer tells a group about a stage
    int pos0, tc;       // the tile: first position, tokens
    int chunk, slice;   // the weights: chunk of the expert's matrix, K-slice
    int expert;         // expert id (n_expert: the shared expert)
    int rows;           // rows of the expert's matrix (down: the stride of the output rows)
    int flags;          // SD_*
    int pad;
};
enum { SD_FIRST = 1, SD_LAST = 2, SD_END = 4 };
// which bounded wait gave up (status word 2, for the error text)
enum { SITE_PRODUCER_SLOT = 1, SITE_CONSUMER_STAGE = 2 };

struct Item {           // a decoded work item: a token tile x a run of chunks
    int shared;         // the shared expert's group
    int expert;
    int chunk0;         // first chunk
    int nch;            // chunks of the item present in this matrix
    int nsl;            // K-slices per chunk
    int pos0;           // first position of the tile
    int tc;             // tokens in the tile
    int rows;
    const uint8_t* src; // K-slice 0 of chunk0; slice s of chunk chunk0 + j is (j * nsl + s) * 128 * SL further
};

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void group_sync(int grp) {   // the 128 threads of one consumer group
    asm volatile("bar.sync %0, 128;" ::"r"(grp + 1) : "memory");
}
// A consumer warp that gave up arrives at its group's meetings for the others, which leave at their next
// wait: for some 65 ms.  (Counting those that have left took 1 to 5 % of passes of a few tokens.)
__device__ __forceinline__ void group_abandon(int grp) { arrive_until_all_left(PfMeetingForAWhile{grp + 1, 128}, 1u << 16); }
template <int TY, int MODE>
__global__ void __launch_bounds__(32 * (4 * Fmt<TY>::MINB + 1), 1)
experts_kernel(const ExpertArgs A) {
    using F = Fmt<TY>;
    constexpr int G = F::MINB;
    constexpr int SB = stage_bytes<TY>();
    constexpr uint32_t W_BYTES = kChunkRows * F::SL, ACT_BYTES = act_stage_bytes<TY>();
    constexpr int CH = MODE == MODE_GATEUP ? 64 : 128;   // output rows per chunk
    pdl_launch_dependents();
    extern __shared__ __align__(128) uint8_t smem[];
    uint64_t* full = (uint64_t*)smem;                 // [G][2] a stage has landed
    uint64_t* empty = full + G * EX_SLOTS;            // [G][2] its four warps are done with it
    int* s_abort = (int*)(smem + 256);
    int* s_next = (int*)(smem + 260);                 // the block's next unclaimed item (index in its list)
    StageDesc* s_desc = (StageDesc*)(smem + 512);     // [G][2]
    float* s_mid_all = (float*)(smem + EX_HEAD);      // [G][EX_TT][64] SwiGLU staging
    uint8_t* ring = (uint8_t*)(s_mid_all + G * EX_TT * 64);   // [G][2][SB]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t hint = A.wait_hint_ns;

    if (tid == 0) {
        for (int i = 0; i < G * EX_SLOTS; i++) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 4);
        }
        *s_abort = 0;
        *s_next = G;   // the first G items of the list are the groups' first items
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    pdl_wait();   // the tile lists and the activation records are the previous kernels'

    // bounded wait that also gives up when another role has
    auto wait = [&](uint64_t* bar, uint32_t parity) -> bool {
        for (uint32_t i = 0; i < EX_WAIT_LIMIT; i++) {
            if (mbar_try_wait(bar, parity, hint)) return true;
            if ((i & 31) == 31 && *(volatile int*)s_abort) return false;
        }
        return false;
    };
    auto give_up = [&](int site) {
        if (atomicExch(A.status, BIVMOE_ERR_TIMEOUT) == 0) atomicExch(A.status + 2, site);
        atomicExch(s_abort, 1);
    };

    if (warp == 4 * G) {
        // ------------------------------------------------------------ producer warp
        // lane g feeds group g
        if (lane >= G) return;
        const int tiles_all = A.n_tiles[0], tiles_sh = A.n_tiles[1];
        const int tile_lo = A.tiles_mode == 1 ? tiles_sh : 0;
        const int tile_hi = A.tiles_mode == 2 ? tiles_sh : tiles_all;
        // an item is a tile times one chunk: 8 stages (gate+up), 2 stages (down) at the qwen35moe shapes
        const int units = (tile_hi - tile_lo) * A.chunks;
        // The lanes stay together: every turn of the loop each lane looks once (without
        // blocking) whether its group has a free slot and, if so, issues its next stage, so
        // no group waits for another lane's wait to end.  A turn without progress in any
        // lane sleeps 64 ns; 2^20 such turns in a row (about 70 ms) end the kernel.
        constexpr uint32_t LANES = (1u << G) - 1u;
        uint32_t issued = 0;      // stages this lane has given its group
        Item it;
        it.nsl = 0;
        int slice = 0, s1 = 0;    // next K-slice of the lane's item, and its end
        int first = 1, ending = 0, done = 0;
        uint32_t idle = 0;
        while (true) {
            int progressed = 0;
            if (!done && !ending && slice >= s1) {
                // the block's list: items blockIdx.x, blockIdx.x + gridDim.x, ...; group g
                // starts with entry g, later entries go to whichever group is ready first
                const int entry = first ? lane : atomicAdd(s_next, 1);
                first = 0;
                const int idx = (int)blockIdx.x + entry * (int)gridDim.x;
                if (idx >= units) {
                    ending = 1;
                } else {
                    const int tile = tile_lo + idx / A.chunks;
                    it.chunk0 = idx % A.chunks;
                    const int4 td = A.tile_desc[tile];
                    it.expert = td.x;
                    it.shared = it.expert == A.n_expert;
                    it.pos0 = td.y;
                    it.tc = td.z;
                    const DevTiles& m = it.shared ? A.sh : A.w;
                    it.nsl = m.nslices;
                    it.nch = it.chunk0 < m.chunks ? 1 : 0;
                    it.rows = m.rows;
                    it.src = m.stage(it.shared ? 0 : it.expert, min(it.chunk0, max(m.chunks - 1, 0)), 0);
                    slice = 0;
                    s1 = it.nch ? it.nsl : 0;
                }
                progressed = 1;
            }
            if (!done && (ending || slice < s1)) {
                const int bi = lane * EX_SLOTS + (int)(issued & 1);
                if (mbar_test_wait(&empty[bi], ((issued >> 1) & 1) ^ 1)) {
                    if (ending) {   // the end marker: a stage without data
                        StageDesc d{};
                        d.flags = SD_END;
                        s_desc[bi] = d;
                        mbar_arrive(&full[bi]);
                        done = 1;
                    } else {
                        StageDesc d;
                        d.pos0 = it.pos0; d.tc = it.tc; d.chunk = it.chunk0; d.slice = slice;
                        d.expert = it.shared ? A.n_expert : it.expert; d.rows = it.rows;
                        d.flags = (slice == 0 ? SD_FIRST : 0) | (slice == s1 - 1 ? SD_LAST : 0);
                        d.pad = 0;
                        s_desc[bi] = d;
                        uint8_t* dst = ring + (size_t)bi * SB;
                        fence_proxy_async();   // the slot was last read through the generic proxy
                        mbar_expect_tx(&full[bi], W_BYTES + ACT_BYTES);
                        bulk_g2s(dst, it.src + (size_t)slice * W_BYTES, W_BYTES, &full[bi]);
                        uint8_t* adst = dst + W_BYTES;
                        const size_t row = (size_t)slice * A.act_rows + it.pos0;
                        bulk_g2s(adst, A.x_f32 + row * F::ELEMS, EX_TT * F::ELEMS * 4, &full[bi]);
                        issued++;
                        slice++;
                    }
                    progressed = 1;
                }
            }
            if (__all_sync(LANES, done)) break;
            if (*(volatile int*)s_abort) break;
            if (__any_sync(LANES, progressed)) {
                idle = 0;
            } else if (++idle > (1u << 20)) {
                if (lane == 0) give_up(SITE_PRODUCER_SLOT);
                break;
            } else {
                __nanosleep(64);
            }
        }
        // leave no copy in flight behind, whoever gave up on it: the last two stages this lane issued, or
        // the last one (the end marker took the other's slot)
        for (uint32_t in_flight = done ? 1 : 2, q = issued > in_flight ? issued - in_flight : 0; q < issued; q++)
            mbar_wait_bounded(&full[lane * EX_SLOTS + (q & 1)], (q >> 1) & 1, hint);
        return;
    }

    // ---------------------------------------------------------------- consumer groups
    const int grp = warp >> 2, wig = warp & 3;
    float* s_mid = s_mid_all + grp * EX_TT * 64;
    // the first chunk row of this warp's two 16-row MMA tiles
    int row_of[2];
    if (MODE == MODE_GATEUP) {   // warp w: gate rows 16w..16w+15 and the same up rows (64 further)
        row_of[0] = 16 * wig;
        row_of[1] = 64 + 16 * wig;
    } else {                     // warp w: down rows 32w..32w+31
        row_of[0] = 32 * wig;
        row_of[1] = 32 * wig + 16;
    }
    float acc[8];   // token t of this lane's row
#pragma unroll
    for (int i = 0; i < 8; i++) acc[i] = 0.0f;
    for (uint32_t q = 0;; q++) {
        const int bi = grp * EX_SLOTS + (int)(q & 1);
        if (!wait(&full[bi], (q >> 1) & 1)) {
            give_up(SITE_CONSUMER_STAGE);
            if (MODE == MODE_GATEUP) group_abandon(grp);   // (down has no meetings)
            return;
        }
        const StageDesc d = s_desc[bi];
        if (d.flags & SD_END) return;
        if (d.flags & SD_FIRST) {
#pragma unroll
            for (int i = 0; i < 8; i++) acc[i] = 0.0f;
        }
        {   // a lane per weight row: GATEUP lanes 0-15 gate rows, 16-31 up rows
            const uint8_t* st = ring + (size_t)bi * SB;
            const uint8_t* wrow;
            if (MODE == MODE_GATEUP) wrow = st + (row_of[lane >> 4] + (lane & 15)) * 16;
            else wrow = st + (32 * wig + lane) * 16;
            F::compute_f32(wrow, (const float*)(st + W_BYTES), d.tc, acc);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[bi]);   // this warp is done with the slot
        if (!(d.flags & SD_LAST)) continue;

        // ---- the chunk is complete
        if (MODE == MODE_GATEUP) {
            // SwiGLU into the staging tile [token][64 rows of the chunk]
#pragma unroll
            for (int t = 0; t < EX_TT; t++) {
                const float u = __shfl_down_sync(0xffffffffu, acc[t], 16);
                if (lane < 16) {
                    const float gt = acc[t];   // ops.rs:160-167: silu(x) = x * (1 / (1 + exp(-x)))
                    s_mid[t * 64 + 16 * wig + lane] = (gt * __fdiv_rn(1.0f, 1.0f + expf(-gt))) * u;
                }
            }
            group_sync(grp);
            // rows of mid: f32 (slice-major by 64) and, for quantised down types, the
            // Q8Act of each 32-row block (quant.rs:368-394); one warp per (token, block)
            for (int p = wig; p < 2 * d.tc; p += 4) {
                const int t = p >> 1, blk = p & 1;
                const float v = s_mid[t * 64 + 32 * blk + lane];
                const int r = d.chunk * CH + 32 * blk + lane;
                const size_t pos = d.pos0 + t;
                A.out[((size_t)(r / 64) * A.act_rows + pos) * 64 + r % 64] = v;
                if (A.out_t) {
                    float dd, ss;
                    const int qv = q8_quantize_lane(v, dd, ss);
                    uint8_t* rec = A.out_t + ((size_t)(r / 256) * (A.act_rows / 8) + pos / 8) * kActTileBytes;
                    rec[act_q_off((int)(pos % 8), r % 256)] = (uint8_t)(int8_t)qv;
                    if (lane < 4) {
                        float shi, slo;
                        split_tf32(ss, &shi, &slo);
                        const float val = lane == 0 ? dd : lane == 1 ? shi : lane == 2 ? slo : ss;
                        *(float*)(rec + act_scale_off(lane, (r % 256) / 32, (int)(pos % 8))) = val;
                    }
                }
            }
            group_sync(grp);   // the staging tile is free for the group's next chunk
        } else {
#pragma unroll
            for (int t = 0; t < EX_TT; t++)
                if (t < d.tc)
                    A.out[(size_t)(d.pos0 + t) * d.rows + d.chunk * CH + 32 * wig + lane] = acc[t];
        }
    }
}

// ---------------------------------------------------------------------------
// host side

bool experts_supported(int ty, int cols, int rows, bool is_down) {
    // every type the reference has a dot kernel for (quant.rs:80-93)
    if (ty != BIVMOE_Q8_0 && ty != BIVMOE_Q4_K && ty != BIVMOE_Q5_K && ty != BIVMOE_Q6_K &&
        ty != BIVMOE_BF16 && ty != BIVMOE_F16 && ty != BIVMOE_F32 && ty != BIVMOE_Q4_0 &&
        ty != BIVMOE_Q4_1)
        return false;
    return cols > 0 && cols % 256 == 0 && rows > 0 && rows % (is_down ? 128 : 64) == 0;
}

template <int TY, int MODE>
static cudaError_t launch_one(const LaunchCfg& c, ExpertArgs A) {
    A.chunks = std::max(A.w.chunks, A.sh.chunks);
    constexpr int smem = smem_bytes<TY>();
    static_assert(smem <= EX_SMEM_MAX, "the block must fit in shared memory");
    static std::atomic<uint64_t> attr_set{0};
    if (cudaError_t e = ensure_dynamic_smem(experts_kernel<TY, MODE>, smem, attr_set)) return e;
    constexpr int threads = 32 * (4 * Fmt<TY>::MINB + 1);
    cudaError_t e = launch_after(c.stream, experts_kernel<TY, MODE>, dim3(c.sm_count), dim3(threads), smem, A);
    count_launch();
    return e;
}

template <int MODE>
static cudaError_t launch_typed(int ty, const LaunchCfg& c, const ExpertArgs& A) {
    switch (ty) {
        case BIVMOE_BF16: return launch_one<BIVMOE_BF16, MODE>(c, A);
        case BIVMOE_F16: return launch_one<BIVMOE_F16, MODE>(c, A);
        case BIVMOE_F32: return launch_one<BIVMOE_F32, MODE>(c, A);
        default: return cudaErrorInvalidValue;
    }
}

// gate+up then down, for the routed experts and the shared expert.  When the
// shared expert's matrices have the routed experts' types it rides in the same
// launches (its tiles come first in the tile list); otherwise it gets its own.
cudaError_t launch_experts(const LaunchCfg& c, const DevTiles& gate_up, const DevTiles& down,
                           const DevTiles& sh_gate_up, const DevTiles& sh_down, const Workspace& ws, bool down_only) {
    ExpertArgs A{};
    A.tile_desc = ws.tile_desc; A.n_tiles = ws.n_tiles;
    A.status = ws.status;
    A.n_expert = c.n_expert;
    A.act_rows = ws.act_rows;
    {
        // read once; the initialisation of a function-local static is safe between host threads
        static const int hint = [] { const char* e = getenv("BIVMOE_WAIT_HINT"); return e ? atoi(e) : 1000; }();
        A.wait_hint_ns = (uint32_t)hint;
    }
    const bool fused = c.has_shared && sh_gate_up.ty == gate_up.ty && sh_down.ty == down.ty;
    cudaError_t err;
    // ---- gate + up (SwiGLU and the Q8 rows of its output in the epilogue)
    auto gateup = [&](int mode, int ty, int down_ty) {
        const DevTiles none{};
        const DevTiles &w = mode == 2 ? none : gate_up, &sh = mode == 1 ? none : sh_gate_up;
        const bool quant_mid = !type_uses_f32_act(down_ty);
        if (c.wide) return launch_experts_tc(c, false, ty, w, sh, ws, mode);
        if (!type_uses_f32_act(ty) || ws.act_3) return launch_experts_quant(c, false, ty, w, sh, ws, quant_mid, mode);
        ExpertArgs G = A;
        G.w = w; G.sh = sh;
        G.x_f32 = ws.act_f;
        G.out = ws.mid;
        G.out_t = quant_mid ? ws.mid_t : nullptr;
        G.tiles_mode = mode;
        return launch_typed<MODE_GATEUP>(ty, c, G);
    };
    if (down_only) {
        err = cudaSuccess;   // gate and up were multiplied already
    } else if (c.only_shared) {
        err = gateup(2, sh_gate_up.ty, sh_down.ty);
    } else if (fused || !c.has_shared) {
        err = gateup(0, gate_up.ty, down.ty);
    } else {
        err = gateup(1, gate_up.ty, down.ty);
        if (err == cudaSuccess) err = gateup(2, sh_gate_up.ty, sh_down.ty);
    }
    if (err == cudaSuccess && c.gateup_parts > 1) err = launch_swiglu_parts(c, ws);
    if (err != cudaSuccess) return err;
    mark(c, EV_GATEUP);
    // ---- down
    auto downp = [&](int mode, int ty) {
        const DevTiles none{};
        const DevTiles &w = mode == 2 ? none : down, &sh = mode == 1 ? none : sh_down;
        if (c.wide) return launch_experts_tc(c, true, ty, w, sh, ws, mode);
        if (!type_uses_f32_act(ty) || ws.act_3) return launch_experts_quant(c, true, ty, w, sh, ws, false, mode);
        ExpertArgs D = A;
        D.w = w; D.sh = sh;
        D.x_f32 = ws.mid;
        D.out = ws.pair_out;
        D.tiles_mode = mode;
        return launch_typed<MODE_DOWN>(ty, c, D);
    };
    if (c.only_shared) return downp(2, sh_down.ty);
    if (fused || !c.has_shared) return downp(0, down.ty);
    err = downp(1, down.ty);
    return err != cudaSuccess ? err : downp(2, sh_down.ty);
}

}  // namespace bivmoe
