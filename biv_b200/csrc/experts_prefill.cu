// Grouped expert products for prefill-sized groups (Q8_0 weights) on the 5th
// generation tensor cores: tcgen05.mma kind::i8 with the accumulator in tensor
// memory, operands staged in shared memory by bulk copies.
// Reference: the same functions as experts_decode.cu (dense_ffn,
// engine/src/model.rs:1119-1126, over the Q8_0 dot, engine/src/quant.rs:599-607),
// for experts whose token list is long (model.rs:875-889).
//
// Design.  One block per SM: a warp whose elected lane issues the copies,
// a warp whose elected lane issues the MMAs (two lanes of one warp take turns: the MMA
// lane then runs only when the copy lane's waits let the warp switch paths),
// sixteen epilogue warps (four per tensor-memory lane quadrant, up to 32 token columns
// each: a thread's accumulators and one drained block fit in 96 registers, and four
// warps per scheduler hide the tensor-memory load latency better than three) and some output
// warps.  A work item is a tile of 128 tokens of one group times a chunk of 128 weight rows
// (64 gate rows with their 64 up rows, or 128 down rows).  The device layouts of common.cuh are already the tensor core's
// canonical K-major operand layouts, so a stage - one K-slice of 256 columns:
// 128 rows x 272 bytes of weights and of each of the tile's 16 activation records what the products
// read - is seventeen bulk copies (cp.async.bulk) and no shuffling.  The reference scales
// every 32-element block dot by its own pair of scales, so the products cannot
// accumulate across blocks inside the tensor core: each block is one MMA
// (M = 128 rows, N = 128 tokens, K = 32) into tensor memory,
// which the epilogue warps drain (tcgen05.ld), scale by d_w * d_x and add to f32
// accumulators in registers while the next MMAs run.  The int32 values in tensor
// memory are the reference's block dots exactly.  The epilogue is the bottleneck
// by construction - per 32 multiply-adds of the tensor core it converts one
// int32 and does two f32 operations - so everything else is kept out of its way:
// two blocks share a buffer and its pair of barriers, the eight blocks of a stage
// are unrolled, and a buffer is handed back as soon as its second block is in
// registers.  Tensor memory holds two such buffers.  A ragged tile (32 or 64 tokens
// at most) deals its columns out to all four warps of a quadrant, 8 or 16 each.
// A thread gets four rows and two of every eight tokens (tcgen05.ld 16x256b): the d_x
// of its two tokens are one 8-byte load where the 32x32b form, a row per thread,
// loads every token's.  An item's sums go to a tile in shared memory, from where the output warps
// take them while the next item's products are made: SwiGLU, quantiser and their stores (6000 clk
// an item when the epilogue warps did them themselves, all at once, of 45 000), or the rows of down, 512 bytes
// a token by bulk copy (3000 of 13 000).  The block's last item, which nothing would hide, the epilogue warps put out
// themselves.  Where an item's rows lie only the copy lane looks up.
// A 128 x 128 x 32 block takes about 550 clk per SM (a loop that has nothing to wait for 437;
// with the 32x32b form 640, with that and a barrier pair per block and the block index in a
// loop 945).  4096 tokens over 256 skewed experts (2048 / 512) 602 + 269 us with the 32x32b form, 402 + 227
// without output warps and with 4-byte stores, so 378 + 194; a dense pass of 300 tokens
// (4096 / 12288) 263 + 161, 161 + 84, 157 + 88 (163 + 92 in the run that gave 162 + 86 with the last item's
// output at the epilogue warps and their share of the registers).
// (Conversions by adding the bits of 1.5 * 2^23 and subtracting that number measured
// slower, whether the epilogue adds them - the f32 work is what fills a pipe, not the
// conversions - or the MMA accumulates onto a buffer pre-set to them: re-arming it
// with tcgen05.st moves 177 B/clk/SM at most.  Pre-set by an MMA of constants they were free, gate+up 358 us
// instead of 378, but then d_w has to come before d_x, an order of roundings that left more of the re-quantised
// values different from the oracle's.)
// Every wait is bounded; a wait that gives up records BIVMOE_ERR_TIMEOUT, the
// block leaves its loops, frees its tensor memory and returns.
#include <cuda_fp16.h>

#include <algorithm>
#include <cstdlib>
#include <type_traits>

#include "common.cuh"
#include "formats.cuh"
#include "tcgen05.cuh"
#include "launch.cuh"

namespace bivmoe {

constexpr int PF_NT = kPrefillTile;                  // tokens per tile = MMA N
constexpr int PF_EPI_WARPS = 16;                     // four per tensor-memory lane quadrant
constexpr int PF_COLS = PF_NT / (PF_EPI_WARPS / 4);  // token columns per epilogue thread
static_assert(PF_COLS == 32, "an epilogue thread drains one 32-column load per block dot");
constexpr int PF_COPY_WARP = PF_EPI_WARPS, PF_MMA_WARP = PF_COPY_WARP + 1;   // a lane each
constexpr int PF_SL = 272;                           // Q8_0: bytes per row per K-slice
constexpr uint32_t PF_W_BYTES = kChunkRows * PF_SL;                // 34816
constexpr uint32_t PF_X_REC = kActOffSHi;                          // what the products read of a record: q and d_x, 2304
constexpr uint32_t PF_STAGE = PF_W_BYTES + PF_NT / 8 * PF_X_REC;   // 71680
constexpr uint32_t PF_HEAD = 512;
// An item's sums on their way out: [128 tokens][128 rows], the tokens 528 bytes apart, so that the eight
// lanes of a store (two 16-byte pieces, four pairs of tokens) fall into different banks
constexpr int PF_TILE_STRIDE = kChunkRows + 4;
constexpr uint32_t PF_TILE = PF_NT * PF_TILE_STRIDE * 4;           // 67584
constexpr uint32_t PF_SMEM = PF_HEAD + 2 * PF_STAGE + PF_TILE;     // 211456
static_assert(PF_SMEM <= 227 * 1024, "the block must fit in shared memory");
constexpr uint32_t PF_TMEM_COLS = 512;                              // two buffers of two blocks' dots
constexpr uint32_t PF_TBUF = 2;
constexpr uint32_t PF_TSTRIDE = PF_TMEM_COLS / PF_TBUF;
constexpr int PF_BUF_BLOCKS = PF_TSTRIDE / PF_NT;

// PF_DOWN_SHORT: the down product of a mixture's many items of a stage or two (rule: launch_experts_prefill).
enum { PF_GATEUP = 0, PF_DOWN = 1, PF_DOWN_SHORT = 2 };

// Output warps, behind the others: six have SwiGLU and the quantiser done while the next item's products
// are made (two took 437 us for what six take 378), two give the rows of down to the copy engine.  Up to
// twenty warps start with 96 registers a thread, twenty-four with 80; the copy, MMA and output warps (whole
// warpgroups) give the epilogue some of theirs: 512 rows of a dense layer's down (4096 / 12288) 128 us with 112, 133 with 104.
template <int MODE> __host__ __device__ constexpr int pf_out_warps() { return MODE == PF_GATEUP ? 6 : 2; }
template <int MODE> __host__ __device__ constexpr int pf_threads() { return 32 * (PF_EPI_WARPS + 2 + pf_out_warps<MODE>()); }
template <int MODE> __host__ __device__ constexpr int pf_regs() { return MODE == PF_GATEUP ? 80 : 96; }   // at the start
template <int MODE> __host__ __device__ constexpr int pf_epi_regs() { return MODE == PF_GATEUP ? 96 : 112; }
template <int MODE> __host__ __device__ constexpr int pf_other_regs() { return MODE == PF_GATEUP ? 48 : 32; }
template <int MODE> constexpr bool pf_regs_fit() {
    return 32 * PF_EPI_WARPS * pf_epi_regs<MODE>() + (pf_threads<MODE>() - 32 * PF_EPI_WARPS) * pf_other_regs<MODE>() <= pf_threads<MODE>() * pf_regs<MODE>();
}
static_assert(pf_regs_fit<PF_GATEUP>() && pf_regs_fit<PF_DOWN>(), "setmaxnreg would wait for registers that nobody gives");

struct PrefillArgs {
    DevTiles w, sh;
    const uint8_t* x_t;    // Q8 records of the inputs by position, [K/256][R/8]
    int act_rows;          // R
    float* out;            // GATEUP: mid f32 slice-major; DOWN: pair_out [R][rows]
    uint8_t* out_t;        // GATEUP: Q8 records of mid
    const int32_t* grp_expert;
    const int32_t* grp_start;
    const int32_t* grp_count;
    const int32_t* ptile_group;
    const int32_t* ptile_t0;
    const int32_t* n_ptiles;
    int32_t* status;
    int n_expert;
    int tiles_mode;        // 0: every tile, 1: skip the shared group's, 2: only the shared group's
    int chunks;
    int parts, part_rows;  // DOWN of a dense layer: K in parts, their sums to out as [part][part_rows][rows]
};

struct PfItem {            // what the copy thread tells the others about an item
    int nst;               // stages; 0: there are no more items (said only where none was known to be the last)
    int chunk, pos0, tc, part;
    int rows;              // of the matrix (down: the stride of the output rows)
    int last;              // the block's last: every role ends with it
};
constexpr uint32_t PF_ITEM_OFF = 272;
constexpr int PF_ITEMS = 8;   // items that have begun and not ended: at most one on its way out, one being summed and two in flight
static_assert(PF_ITEM_OFF % 16 == 0 && PF_ITEM_OFF + PF_ITEMS * sizeof(PfItem) <= PF_HEAD, "the items lie in front of the stages");

// tokens of a tile rounded up to the MMA's N granularity (ragged last tiles)
__device__ __forceinline__ int pf_mma_n(int tc) { return (tc + 15) & ~15; }

template <int MODE>
__global__ void __launch_bounds__(pf_threads<MODE>(), 1)
experts_prefill_kernel(const PrefillArgs A) {
    pdl_launch_dependents();
    extern __shared__ __align__(1024) uint8_t smem[];
    uint64_t* full = (uint64_t*)smem;            // [2] copies landed
    uint64_t* empty = full + 2;                  // [2] stage free: MMAs done + the epilogue warps
    uint64_t* tfull = full + 16;                 // [4] a block dot is in tensor memory
    uint64_t* tempty = full + 20;                // [2] drained by the epilogue warps
    uint64_t* tile_full = full + 10;             // [1] an item's sums are in the tile
    uint64_t* tile_empty = full + 11;            // [1] and read from there
    uint64_t* mmas = full + 9;                   // [1] everything the MMA thread issued has completed
    uint32_t* s_tmem = (uint32_t*)(smem + 256);
    int* s_abort = (int*)(smem + 260);
    PfItem* s_item = (PfItem*)(smem + PF_ITEM_OFF);   // [PF_ITEMS]
    uint8_t* stages = smem + PF_HEAD;
    float* s_tile = (float*)(smem + PF_HEAD + 2 * PF_STAGE);   // [128 tokens][PF_TILE_STRIDE]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int CH = MODE == PF_GATEUP ? 64 : 128;   // output rows per chunk
    constexpr int OUTS = pf_out_warps<MODE>();
    // Whether a block's last item, whose output no products hide, is left to the epilogue warps: they are faster at it than the
    // output warps (a gate+up item of 128 tokens 2.5 to 3 us, one of down 1.3).  That code and the registers' split, in a
    // pass of many short items, cost 2 to 5 % of down (64 experts, 1000 rows of 2048 / 512 205 -> 215 us); from three stages an item on
    // they win that much (8 experts, 2048 rows: 42.8 -> 43.2 us with two stages, 58.4 -> 55.3 with three, 138 -> 130 with eight).
    constexpr bool LAST = MODE != PF_DOWN_SHORT;

    if (tid == 0) {
        for (int i = 0; i < 2; i++) {
            pf_bar_init(&full[i], 1);
            pf_bar_init(&empty[i], 1 + PF_EPI_WARPS);
        }
        for (int i = 0; i < (int)PF_TBUF; i++) {
            pf_bar_init(&tfull[i], 1);
            pf_bar_init(&tempty[i], PF_EPI_WARPS);
        }
        pf_bar_init(tile_full, PF_EPI_WARPS);
        pf_bar_init(tile_empty, OUTS);
        pf_bar_init(mmas, 1);
        *s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == PF_COPY_WARP) {   // tensor memory: all 512 columns for the whole kernel
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         pf_smem(s_tmem)),
                     "r"(PF_TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    pf_fence_before();
    __syncthreads();
    pf_fence_after();
    const uint32_t tmem = *s_tmem;
    pdl_wait();   // the tile lists and the activation records are the previous kernels'

    const int tiles_all = A.n_ptiles[0], tiles_sh = A.n_ptiles[1];
    const int tile_lo = A.tiles_mode == 1 ? tiles_sh : 0;
    const int tile_hi = A.tiles_mode == 2 ? tiles_sh : tiles_all;
    const int total = (tile_hi - tile_lo) * A.chunks * A.parts;

    auto give_up = [&]() {
        atomicExch(A.status, BIVMOE_ERR_TIMEOUT);
        atomicExch(s_abort, 1);
    };

    // Gate+up, an item's output from the tile, by `warps` warps of which this is number `first`: SwiGLU, the rows of
    // mid in f32 and the Q8Act of each 32-row block (quant.rs:368-394), eight rows a thread, four threads a block, four tokens a warp
    auto swiglu_out = [&](const PfItem& it, int first, int warps) {
        const int u = lane & 7, r = it.chunk * CH + 8 * u;
        float* mid = A.out + ((size_t)(r / 64) * A.act_rows + it.pos0) * 64 + r % 64;
        uint8_t* rec0 = A.out_t + ((size_t)(r / 256) * (A.act_rows / 8) + it.pos0 / 8) * kActTileBytes;
        for (int tb = 4 * first; tb < it.tc; tb += 4 * warps) {
            const int tok = tb + (lane >> 3);   // past the end: what the tile holds, not stored
            const float* gt = s_tile + tok * PF_TILE_STRIDE + 8 * u;
            float v[8];
#pragma unroll
            for (int k = 0; k < 8; k += 4) {
                const float4 a = *(const float4*)(gt + k), b = *(const float4*)(gt + 64 + k);
                // ops.rs:160-167: silu(x) = x * (1 / (1 + exp(-x)))
                v[k] = (a.x * __frcp_rn(1.0f + expf(-a.x))) * b.x;
                v[k + 1] = (a.y * __frcp_rn(1.0f + expf(-a.y))) * b.y;
                v[k + 2] = (a.z * __frcp_rn(1.0f + expf(-a.z))) * b.z;
                v[k + 3] = (a.w * __frcp_rn(1.0f + expf(-a.w))) * b.w;
            }
            uint32_t q0, q1;
            float dd, ss, shi, slo;
            quantize_eight(v, q0, q1, dd, ss);
            if (tok >= it.tc) continue;
            *(float4*)(mid + (size_t)tok * 64) = make_float4(v[0], v[1], v[2], v[3]);
            *(float4*)(mid + (size_t)tok * 64 + 4) = make_float4(v[4], v[5], v[6], v[7]);
            uint8_t* rec = rec0 + (tok >> 3) * kActTileBytes;
            *(uint2*)(rec + act_q_off(tok & 7, r % 256)) = make_uint2(q0, q1);
            split_tf32(ss, &shi, &slo);
            const int which = lane & 3;   // each of the block's four threads stores one of its scales
            *(float*)(rec + act_scale_off(which, (r % 256) / 32, tok & 7)) = which == 0 ? dd : which == 1 ? shi : which == 2 ? slo : ss;
        }
    };

    if (warp >= PF_EPI_WARPS) {
        if constexpr (LAST) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(pf_other_regs<MODE>()));
        if (warp == PF_COPY_WARP) {
            // ---------------- copy thread
            if (pf_elect()) {
                // The items are dealt round-robin.  Only this thread looks them up - two loads, one after the other,
                // from L2, while the stages before are worked on; the others find an item in shared memory with
                // its first stage.
                uint32_t q = 0, n_items = 0;
                auto slot_free = [&]() {
                    if (pf_bar_wait(&empty[q & 1], ((q >> 1) & 1) ^ 1)) return true;
                    give_up();
                    return false;
                };
                bool dead = false, known = false;
                for (int idx = blockIdx.x; idx < total && !dead && !*(volatile int*)s_abort; idx += gridDim.x) {
                    PfItem it;
                    it.part = MODE != PF_GATEUP ? idx % A.parts : 0;
                    const int rest = MODE != PF_GATEUP ? idx / A.parts : idx, tile = tile_lo + rest / A.chunks;
                    it.chunk = rest % A.chunks;
                    const int gi = A.ptile_group[tile], t0 = A.ptile_t0[tile], expert = A.grp_expert[gi];
                    const bool shared = expert == A.n_expert;
                    it.pos0 = A.grp_start[gi] + t0;
                    it.tc = min(PF_NT, A.grp_count[gi] - t0);
                    const DevTiles& m = shared ? A.sh : A.w;
                    it.rows = m.rows;
                    it.last = LAST && idx + (int)gridDim.x >= total;
                    const int all = it.chunk < m.chunks ? m.nslices : 0;
                    const int s0 = MODE != PF_GATEUP ? all * it.part / A.parts : 0;
                    it.nst = (MODE != PF_GATEUP ? all * (it.part + 1) / A.parts : all) - s0;
                    if (it.nst == 0) continue;
                    known = it.last;
                    const uint8_t* wsrc = m.stage(shared ? 0 : expert, it.chunk, s0);
                    const uint8_t* xsrc = A.x_t + ((size_t)s0 * (A.act_rows / 8) + it.pos0 / 8) * kActTileBytes;
                    const int recs = pf_mma_n(it.tc) / 8;
                    for (int s = 0; s < it.nst; s++, q++) {
                        if (!slot_free()) { dead = true; break; }
                        const uint32_t slot = q & 1;
                        if (s == 0) s_item[n_items++ % PF_ITEMS] = it;
                        uint8_t* dst = stages + slot * PF_STAGE;
                        pf_bar_expect_tx(&full[slot], PF_W_BYTES + recs * PF_X_REC);
                        pf_bulk_g2s(dst, wsrc + (size_t)s * PF_W_BYTES, PF_W_BYTES, &full[slot]);
                        const uint8_t* x = xsrc + (size_t)s * (A.act_rows / 8) * kActTileBytes;
                        for (int i = 0; i < recs; i++) pf_bulk_g2s(dst + PF_W_BYTES + i * PF_X_REC, x + i * kActTileBytes, PF_X_REC, &full[slot]);
                    }
                }
                const bool ended = !dead && !known && slot_free();
                if (ended) {   // the end: a stage without data
                    s_item[n_items % PF_ITEMS].nst = 0;
                    pf_bar_arrive(&full[q & 1]);
                }
                // no copy is in flight when the block ends, whoever gave up on it: the last one of either slot
                // has landed, or was waited for
                for (uint32_t last = q + ended, p = last > 2 ? last - 2 : 0; p < q; p++) pf_bar_wait(&full[p & 1], (p >> 1) & 1);
            }
        } else if (warp == PF_MMA_WARP) {
            // ---------------- MMA thread: one MMA per 32-column block, two per buffer.  In a warp of its own:
            // as a second lane of the copy thread's warp it ran only when that lane's waits
            // let the warp switch paths.
            if (pf_elect()) {
                uint32_t q = 0, kb = 0;
                bool dead = false;
                for (uint32_t n_items = 0; !dead && !*(volatile int*)s_abort; n_items++) {
                    if (!pf_bar_wait(&full[q & 1], (q >> 1) & 1)) { give_up(); break; }
                    const PfItem it = s_item[n_items % PF_ITEMS];
                    if (it.nst == 0) break;
                    const uint32_t idesc = pf_idesc(kChunkRows, pf_mma_n(it.tc));
                    for (int s = 0; s < it.nst && !dead; s++, q++) {
                        const uint32_t slot = q & 1;
                        if (s > 0 && !pf_bar_wait(&full[slot], (q >> 1) & 1)) { give_up(); dead = true; break; }
                        const uint32_t wa = pf_smem(stages + slot * PF_STAGE);
                        const uint32_t xa = wa + PF_W_BYTES;
                        for (int b = 0; b < 8 && !dead; b += PF_BUF_BLOCKS, kb++) {
                            const uint32_t buf = kb % PF_TBUF;
                            if (!pf_bar_wait(&tempty[buf], ((kb / PF_TBUF) & 1) ^ 1)) { give_up(); dead = true; break; }
                            pf_fence_after();
                            // A: rows of the chunk, units 2b and 2b+1: 8-row groups 128 B apart,
                            //    K steps 2048 B apart.  B: tokens, units 2b, 2b+1 of each record:
                            //    8-token groups one record apart, K steps 128 B apart.
#pragma unroll
                            for (int i = 0; i < PF_BUF_BLOCKS; i++) {
                                const uint64_t ad = pf_desc(wa + 2 * (b + i) * (kChunkRows * 16), kChunkRows * 16, 128);
                                const uint64_t bd = pf_desc(xa + 2 * (b + i) * 128, 128, PF_X_REC);
                                pf_mma_i8(tmem + buf * PF_TSTRIDE + i * PF_NT, ad, bd, idesc);
                            }
                            pf_commit(&tfull[buf]);
                        }
                        if (!dead) pf_commit(&empty[slot]);   // the stage's operands are no longer read
                    }
                    if (LAST && it.last) break;
                }
                pf_commit(mmas);                              // nor is an MMA
                if (!pf_bar_wait(mmas, 0)) give_up();
            }
        } else {
            // ---------------- output warps: what becomes of an item's sums, while the next item's are made
            for (uint32_t n_items = 0;; n_items++) {
                if (!pf_together(pf_bar_wait_long(tile_full, n_items & 1))) { if (lane == 0) give_up(); break; }
                const PfItem it = s_item[n_items % PF_ITEMS];
                if (it.nst == 0 || (LAST && it.last)) break;
                if (MODE == PF_GATEUP) {
                    swiglu_out(it, warp - PF_MMA_WARP - 1, OUTS);
                } else {
                    // a token's 128 rows at a time
                    float* dst = A.out + ((size_t)it.part * A.part_rows + it.pos0) * it.rows + it.chunk * CH;
                    for (int tok = 32 * (warp - PF_MMA_WARP - 1) + lane; tok < it.tc; tok += 32 * OUTS)
                        pf_bulk_s2g(dst + (size_t)tok * it.rows, s_tile + tok * PF_TILE_STRIDE, kChunkRows * 4);
                    pf_bulk_commit();
                    pf_bulk_wait_read();
                }
                __syncwarp();
                if (lane == 0) pf_bar_arrive(tile_empty);
            }
            if (MODE != PF_GATEUP) pf_bulk_wait();   // before the block ends
        }
    } else {
        if constexpr (LAST) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(pf_epi_regs<MODE>()));
        // ---------------- epilogue warps
        const int quad = warp & 3;               // the tensor-memory lanes this warp may read
        const int cg = warp >> 2;                 // which quarter of the token columns
        const int g = lane >> 2, c = lane & 3;   // places 32 quad + g + 8 i of the chunk, token columns 8 j + 2 c, + 1
        const uint32_t tlane = tmem + ((uint32_t)(32 * quad) << 16);
        uint32_t q = 0, kb = 0, n_items = 0;
        bool last = false;
        for (; pf_together(!*(volatile int*)s_abort); n_items++) {
            bool ok = pf_together(pf_bar_wait(&full[q & 1], (q >> 1) & 1));
            if (!ok) { if (lane == 0) give_up(); break; }
            const PfItem it = s_item[n_items % PF_ITEMS];
            if (it.nst == 0) {   // for the output warps too, once they have the last item
                if (!pf_together(pf_bar_wait(tile_empty, (n_items & 1) ^ 1))) { if (lane == 0) give_up(); break; }
                if (lane == 0) pf_bar_arrive(tile_full);
                break;
            }
            f32x2 acc[4][PF_COLS / 8];   // [i][j]: place g + 8 i, token columns 8 j + 2 c and the next
#pragma unroll
            for (int i = 0; i < PF_COLS / 2; i++) (&acc[0][0])[i] = 0ull;
            // the item's block dots, T token columns per warp: warps of a ragged tile share
            // its columns out instead of leaving them to the first ones.  (The lanes of a warp try, and read
            // the clock, by the same instructions, so a wait ends for all of them or for none; a vote on each
            // made it sure at 3 to 6 % of a pass: 4096 rows 896 -> 921 us, dense 300 rows 254 -> 268.)
            auto products = [&](auto cols) {
                constexpr int T = decltype(cols)::value, J = T / 8;
                const uint32_t tcol = tlane + cg * T;
                for (int s = 0; s < it.nst; s++, q++) {
                    const uint32_t slot = q & 1;
                    if (s > 0 && !pf_bar_wait(&full[slot], (q >> 1) & 1)) { ok = false; return; }
                    const uint8_t* wst = stages + slot * PF_STAGE;
                    const uint8_t* xst = wst + PF_W_BYTES + cg * J * PF_X_REC + kActOffDx + c * 8;
                    const uint8_t* dst = wst + 16 * (kChunkRows * 16) + (32 * quad + g) * 16;   // a row's 8 f16 scales
                    __half2 dh[4];   // rows g + 8 i: the scales of two blocks
#pragma unroll
                    for (int b = 0; b < 8; b++) {
                        const uint32_t buf = kb % PF_TBUF;
                        if (b % PF_BUF_BLOCKS == 0) {
#pragma unroll
                            for (int i = 0; i < 4; i++) dh[i] = *(const __half2*)(dst + i * 128 + b * 2);
                            if (!pf_bar_wait(&tfull[buf], (kb / PF_TBUF) & 1)) { ok = false; return; }
                            pf_fence_after();
                        }
                        // drain this warp's columns; hand the buffer back after its last block
                        int v[2][4 * J];
                        const uint32_t at = tcol + buf * PF_TSTRIDE + (b % PF_BUF_BLOCKS) * PF_NT;
                        pf_tmem_ld_16x8<J>(at, v[0]);
                        pf_tmem_ld_16x8<J>(at + (16u << 16), v[1]);
                        pf_tmem_wait_ld();
                        if (b % PF_BUF_BLOCKS == PF_BUF_BLOCKS - 1) {
                            pf_fence_before();
                            __syncwarp();
                            if (lane == 0) pf_bar_arrive(&tempty[buf]);
                            kb++;
                        }
                        f32x2 dw[4];
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            const float d = b & 1 ? __high2float(dh[i]) : __low2float(dh[i]);
                            dw[i] = pk(d, d);
                        }
#pragma unroll
                        for (int j = 0; j < J; j++) {   // a record: 8 tokens, d_x of block b
                            const f32x2 dx = *(const f32x2*)(xst + j * PF_X_REC + b * 32);
#pragma unroll
                            for (int i = 0; i < 4; i++) {
                                // the int32 block dots, exact as floats (below 2^24)
                                const int* d = &v[i >> 1][4 * j + 2 * (i & 1)];
                                const f32x2 f = pk(__int2float_rn(d[0]), __int2float_rn(d[1]));
                                acc[i][j] = fma2(dw[i], mul2(dx, f), acc[i][j]);
                            }
                        }
                    }
                    __syncwarp();
                    if (lane == 0) pf_bar_arrive(&empty[slot]);   // done with the stage's scales
                }
            };
            // columns per warp (PF_COLS at most): the tile's, in whole records, over four warps
            const int T = it.tc <= 32 ? 8 : it.tc <= 64 ? 16 : 32;
            if (T == 8) products(std::integral_constant<int, 8>{});
            else if (T == 16) products(std::integral_constant<int, 16>{});
            else products(std::integral_constant<int, 32>{});
            if (!ok) { if (lane == 0) give_up(); break; }
            // ---- the item's sums, for the output warps
            if (!pf_together(pf_bar_wait(tile_empty, (n_items & 1) ^ 1))) { if (lane == 0) give_up(); break; }
            const int tok0 = cg * T + 2 * c;
#pragma unroll
            for (int j = 0; j < PF_COLS / 8; j++) {
                if (8 * j >= T) break;
                float* at = s_tile + (tok0 + 8 * j) * PF_TILE_STRIDE + 32 * quad + 4 * g;
                *(float4*)at = make_float4(lo_of(acc[0][j]), lo_of(acc[1][j]), lo_of(acc[2][j]), lo_of(acc[3][j]));
                *(float4*)(at + PF_TILE_STRIDE) = make_float4(hi_of(acc[0][j]), hi_of(acc[1][j]), hi_of(acc[2][j]), hi_of(acc[3][j]));
            }
            if (MODE != PF_GATEUP) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // bulk copies read it
            __syncwarp();
            if (lane == 0) pf_bar_arrive(tile_full);
            if (LAST && (last = it.last)) break;
        }
        // (behind the loop: in it, it took the products' registers, 2 to 4 % of a long pass)
        if (last && !pf_together(pf_bar_wait(tile_full, n_items & 1))) {
            if (lane == 0) give_up();
        } else if (last) {
            const PfItem it = s_item[n_items % PF_ITEMS];
            if (MODE == PF_GATEUP) {
                swiglu_out(it, warp, PF_EPI_WARPS);
            } else {
                float* dst = A.out + ((size_t)it.part * A.part_rows + it.pos0) * it.rows + it.chunk * CH + 4 * lane;
                for (int tok = warp; tok < it.tc; tok += PF_EPI_WARPS)
                    *(float4*)(dst + (size_t)tok * it.rows) = *(const float4*)(s_tile + tok * PF_TILE_STRIDE + 4 * lane);
            }
        }
    }
    pf_fence_before();
    __syncthreads();
    pf_fence_after();
    if (warp == PF_COPY_WARP) {
        __syncwarp();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                     "r"(PF_TMEM_COLS)
                     : "memory");
    }
}

// ---------------------------------------------------------------------------
// host side

bool prefill_supported(int gate_up_ty, int down_ty) {
    return (gate_up_ty == BIVMOE_Q8_0 && down_ty == BIVMOE_Q8_0) ||
           (gate_up_ty == BIVMOE_BF16 && down_ty == BIVMOE_BF16);
}

template <int MODE>
static cudaError_t launch_prefill_one(const LaunchCfg& c, PrefillArgs A) {
    A.chunks = std::max(A.w.chunks, A.sh.chunks);
    static std::atomic<uint64_t> attr_set{0};
    if (cudaError_t e = ensure_dynamic_smem(experts_prefill_kernel<MODE>, (int)PF_SMEM, attr_set)) return e;
    // setmaxnreg deals out the registers of pf_regs<MODE>(): a build that launches with fewer would wait for the rest for ever
    static const bool enough = [] {
        cudaFuncAttributes a{};
        return cudaFuncGetAttributes(&a, experts_prefill_kernel<MODE>) == cudaSuccess && a.numRegs >= pf_regs<MODE>();
    }();
    if (MODE != PF_DOWN_SHORT && !enough) return cudaErrorLaunchOutOfResources;
    count_launch();
    return launch_after(c.stream, experts_prefill_kernel<MODE>, dim3(c.sm_count), dim3(pf_threads<MODE>()), PF_SMEM, A);
}

// gate+up then down for the groups the sort put on the prefill tile list
cudaError_t launch_experts_prefill(const LaunchCfg& c, const DevTiles& gate_up, const DevTiles& down,
                                   const DevTiles& sh_gate_up, const DevTiles& sh_down,
                                   const Workspace& ws) {
    const int ty = c.only_shared ? sh_gate_up.ty : gate_up.ty;
    if (ty == BIVMOE_BF16) return launch_experts_prefill_bf16(c, gate_up, down, sh_gate_up, sh_down, ws);
    PrefillArgs A{};
    A.grp_expert = ws.grp_expert; A.grp_start = ws.grp_start; A.grp_count = ws.grp_count;
    A.ptile_group = ws.ptile_group; A.ptile_t0 = ws.ptile_t0; A.n_ptiles = ws.n_ptiles;
    A.status = ws.status;
    A.n_expert = c.n_expert;
    A.act_rows = ws.act_rows;
    A.tiles_mode = c.only_shared ? 2 : 0;
    A.parts = 1;
    PrefillArgs G = A;
    G.w = gate_up; G.sh = sh_gate_up;
    G.x_t = ws.act_t; G.out = ws.mid; G.out_t = ws.mid_t;
    cudaError_t err = launch_prefill_one<PF_GATEUP>(c, G);
    if (err != cudaSuccess) return err;
    PrefillArgs D = A;
    D.w = down; D.sh = sh_down;
    D.x_t = ws.mid_t; D.out = ws.pair_out; D.out_t = nullptr;
    D.parts = c.down_parts; D.part_rows = c.n;
    if (D.parts > 1) D.out = ws.parts;
    // a stage or two an item, and several items a block (their tiles, at most; the list is on the device)
    const long long tiles = (long long)c.n * c.k / PF_NT + c.n_expert + (c.has_shared ? (c.n + PF_NT - 1) / PF_NT : 0);
    const bool few = tiles * std::max(down.chunks, sh_down.chunks) * D.parts <= 4 * c.sm_count;
    return few || std::max(down.nslices, sh_down.nslices) / D.parts >= 3 ? launch_prefill_one<PF_DOWN>(c, D) : launch_prefill_one<PF_DOWN_SHORT>(c, D);
}

}  // namespace bivmoe

// ---------------------------------------------------------------------------
// The int8 tensor-pipe peak of this GPU, measured: no int8 figure comes with the
// machine's measured peaks, so the Q8_0 kernel's roofline denominator is taken here.
// One block per SM issues back-to-back tcgen05.mma kind::i8 (M 128, N 256, K 32) from
// one thread, alternating between two tensor-memory accumulators, on operands that stay
// in shared memory; nothing is loaded or drained, so this is the pipe alone.
namespace bivmoe {

constexpr uint32_t PEAK_SMEM = 1024 + 128 * 32 + 256 * 32;   // descriptors' operands: A 4 KiB, B 8 KiB

__global__ void __launch_bounds__(128, 1) int8_peak_kernel(int mmas, int32_t* status) {
    extern __shared__ __align__(1024) uint8_t smem[];
    uint64_t* done = (uint64_t*)smem;
    uint32_t* s_tmem = (uint32_t*)(smem + 64);
    const int tid = threadIdx.x, warp = tid >> 5;
    for (uint32_t i = tid; i < (PEAK_SMEM - 1024) / 4; i += blockDim.x) ((uint32_t*)(smem + 1024))[i] = 0x01010101u;
    if (tid == 0) {
        pf_bar_init(done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the operands, for the tensor core
    if (warp == 0) {
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         pf_smem(s_tmem)),
                     "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    pf_fence_before();
    __syncthreads();
    pf_fence_after();
    const uint32_t tmem = *s_tmem;
    if (tid == 0) {
        const uint32_t a = pf_smem(smem + 1024), b = a + 128 * 32;
        // K-major, two 16-byte K units: rows 16 bytes apart inside an 8-row group
        const uint64_t ad = pf_desc(a, 128 * 16, 128), bd = pf_desc(b, 256 * 16, 128);
        const uint32_t idesc = pf_idesc(128, 256);
        for (int i = 0; i < mmas; i++) pf_mma_i8(tmem + (i & 1) * 256, ad, bd, idesc);
        pf_commit(done);
        if (!pf_bar_wait(done, 0)) atomicExch(status, BIVMOE_ERR_TIMEOUT);
    }
    pf_fence_before();
    __syncthreads();
    pf_fence_after();
    if (warp == 0) {
        __syncwarp();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u)
                     : "memory");
    }
}

// tera-operations per second (2 per multiply-add) over all SMs; `status_dev`: a device
// word that a bounded wait flags
cudaError_t measure_int8_peak(int sm_count, int32_t* status_dev, cudaStream_t stream, double* tops) {
    static std::atomic<uint64_t> attr_set{0};
    if (cudaError_t e = ensure_dynamic_smem(int8_peak_kernel, (int)PEAK_SMEM, attr_set)) return e;
    const int mmas = 1 << 15;
    cudaEvent_t e0, e1;
    cudaError_t err = cudaEventCreate(&e0);
    if (err != cudaSuccess) return err;
    err = cudaEventCreate(&e1);
    if (err != cudaSuccess) { cudaEventDestroy(e0); return err; }
    int8_peak_kernel<<<sm_count, 128, PEAK_SMEM, stream>>>(1 << 10, status_dev);   // warm-up
    cudaEventRecord(e0, stream);
    int8_peak_kernel<<<sm_count, 128, PEAK_SMEM, stream>>>(mmas, status_dev);
    cudaEventRecord(e1, stream);
    err = cudaEventSynchronize(e1);
    float ms = 0.0f;
    if (err == cudaSuccess) err = cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (err != cudaSuccess) return err;
    *tops = 2.0 * 128 * 256 * 32 * (double)mmas * sm_count / (ms * 1e-3) / 1e12;
    return cudaGetLastError();
}

}  // namespace bivmoe
