// Grouped expert products for prefill-sized groups (Q8_0 weights) on the 5th
// generation tensor cores: tcgen05.mma kind::i8 with the accumulator in tensor
// memory, operands staged in shared memory by bulk copies.
// Reference: the same functions as experts_decode.cu (dense_ffn,
// engine/src/model.rs:1119-1126, over the Q8_0 dot, engine/src/quant.rs:599-607),
// for experts whose token list is long (model.rs:875-889).
//
// Design.  One block per SM, eighteen warps: a warp whose lane 0 issues the copies,
// a warp whose lane 0 issues the MMAs (two lanes of one warp take turns: the MMA
// lane then runs only when the copy lane's waits let the warp switch paths), and
// sixteen epilogue warps (four per tensor-memory lane quadrant, up to 32 token columns
// each: a thread's accumulators and one drained block fit in 96 registers, and four
// warps per scheduler hide the tensor-memory load latency better than three).  A
// work item is a tile of 128 tokens of one group times a chunk of 128 weight rows
// (64 gate rows with their 64 up rows, or 128 down rows).  The device layouts of common.cuh are already the tensor core's
// canonical K-major operand layouts, so a stage - one K-slice of 256 columns:
// 128 rows x 272 bytes of weights and the 16 activation records of the tile -
// is two bulk copies (cp.async.bulk) and no shuffling.  The reference scales
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
// loads every token's.  A 128 x 128 x 32 block takes about 600 clk per SM (with the
// 32x32b form 640, with that and a barrier pair per block and the block index in a
// loop 945; the SwiGLU tail is 70 of them).  A dense pass of 300 tokens (4096 / 12288)
// went from 263 + 161 to 161 + 84 us, 4096 tokens over 256 skewed experts
// (2048 / 512) from 602 + 269 to 402 + 227 us.  (Copying only the q and d_x of a
// record, a quarter less, changed nothing: L2 is not what it waits for.)
// (Conversions by adding the bits of 1.5 * 2^23 and subtracting that number measured
// slower, whether the epilogue adds them - the f32 work is what fills a pipe, not the
// conversions - or the MMA accumulates onto a buffer pre-set to them: re-arming it
// with tcgen05.st moves 177 B/clk/SM at most.)
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
constexpr int PF_MMA_WARP = 1 + PF_EPI_WARPS;        // the MMA thread's own warp
constexpr int PF_THREADS = 32 * (2 + PF_EPI_WARPS);  // warp 0: lane 0 copies; the last warp: lane 0 issues MMAs
constexpr int PF_SL = 272;                           // Q8_0: bytes per row per K-slice
constexpr uint32_t PF_W_BYTES = kChunkRows * PF_SL;                // 34816
constexpr uint32_t PF_X_BYTES = (PF_NT / 8) * kActTileBytes;       // 49152
constexpr uint32_t PF_STAGE = PF_W_BYTES + PF_X_BYTES;             // 83968
constexpr uint32_t PF_HEAD = 1024;
constexpr uint32_t PF_XCHG = 64 * PF_NT * 4;                        // SwiGLU exchange, 32 KiB
constexpr uint32_t PF_SMEM = PF_HEAD + 2 * PF_STAGE + PF_XCHG;      // 201728
constexpr uint32_t PF_TMEM_COLS = 512;                              // two buffers of two blocks' dots
constexpr uint32_t PF_TBUF = 2;
constexpr uint32_t PF_TSTRIDE = PF_TMEM_COLS / PF_TBUF;
constexpr int PF_BUF_BLOCKS = PF_TSTRIDE / PF_NT;

enum { PF_GATEUP = 0, PF_DOWN = 1 };

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

struct PfItem {
    int shared, expert, chunk, pos0, tc, nst;
    int part, s0;          // part of K; its first stage
    int n_mma;             // tc rounded up to the MMA's N granularity of 16 (ragged last tiles)
    const uint8_t* wsrc;   // stage s0 of the chunk's weights; stage s is s * PF_W_BYTES further
};

template <int MODE>
__global__ void __launch_bounds__(PF_THREADS, 1)
experts_prefill_kernel(const PrefillArgs A) {
    pdl_launch_dependents();
    extern __shared__ __align__(1024) uint8_t smem[];
    uint64_t* full = (uint64_t*)smem;            // [2] copies landed
    uint64_t* empty = full + 2;                  // [2] stage free: MMAs done + the epilogue warps
    uint64_t* tfull = full + 16;                 // [4] a block dot is in tensor memory
    uint64_t* tempty = full + 20;                // [2] drained by the epilogue warps
    uint64_t* xbar = full + 8;                   // [1] meeting point of the epilogue warps
    uint64_t* mmas = full + 9;                   // [1] everything the MMA thread issued has completed
    uint32_t* s_tmem = (uint32_t*)(smem + 256);
    int* s_abort = (int*)(smem + 260);
    uint8_t* stages = smem + PF_HEAD;
    float* s_xchg = (float*)(smem + PF_HEAD + 2 * PF_STAGE);   // [128 tokens][64 rows]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int CH = MODE == PF_GATEUP ? 64 : 128;   // output rows per chunk

    if (tid == 0) {
        for (int i = 0; i < 2; i++) {
            pf_bar_init(&full[i], 1);
            pf_bar_init(&empty[i], 1 + PF_EPI_WARPS);
        }
        for (int i = 0; i < (int)PF_TBUF; i++) {
            pf_bar_init(&tfull[i], 1);
            pf_bar_init(&tempty[i], PF_EPI_WARPS);
        }
        pf_bar_init(xbar, PF_EPI_WARPS);
        pf_bar_init(mmas, 1);
        *s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {   // tensor memory: all 512 columns for the whole kernel
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

    // items are dealt round-robin: every role walks the same sequence on its own
    auto decode = [&](int idx) -> PfItem {
        PfItem it;
        it.part = MODE == PF_DOWN ? idx % A.parts : 0;
        if (MODE == PF_DOWN) idx /= A.parts;
        const int tile = tile_lo + idx / A.chunks;
        it.chunk = idx % A.chunks;
        const int gi = A.ptile_group[tile], t0 = A.ptile_t0[tile];
        it.expert = A.grp_expert[gi];
        it.shared = it.expert == A.n_expert;
        it.pos0 = A.grp_start[gi] + t0;
        it.tc = min(PF_NT, A.grp_count[gi] - t0);
        it.n_mma = (it.tc + 15) & ~15;
        const DevTiles& m = it.shared ? A.sh : A.w;
        const int nst = it.chunk < m.chunks ? m.nslices : 0;
        it.s0 = MODE == PF_DOWN ? nst * it.part / A.parts : 0;
        it.nst = (MODE == PF_DOWN ? nst * (it.part + 1) / A.parts : nst) - it.s0;
        it.wsrc = m.stage(it.shared ? 0 : it.expert, min(it.chunk, max(m.chunks - 1, 0)), it.s0);
        return it;
    };
    auto give_up = [&]() {
        atomicExch(A.status, BIVMOE_ERR_TIMEOUT);
        atomicExch(s_abort, 1);
    };

    if (warp == 0) {
        // ---------------- copy thread: two bulk copies per stage
        if (lane == 0) {
            uint32_t q = 0;
            bool dead = false;
            for (int idx = blockIdx.x; idx < total && !dead && !*(volatile int*)s_abort; idx += gridDim.x) {
                const PfItem it = decode(idx);
                for (int s = 0; s < it.nst && !dead; s++, q++) {
                    const uint32_t slot = q & 1;
                    if (!pf_bar_wait(&empty[slot], ((q >> 1) & 1) ^ 1)) { give_up(); dead = true; break; }
                    uint8_t* dst = stages + slot * PF_STAGE;
                    const uint32_t x_bytes = (uint32_t)(it.n_mma / 8) * kActTileBytes;
                    pf_bar_expect_tx(&full[slot], PF_W_BYTES + x_bytes);
                    pf_bulk_g2s(dst, it.wsrc + (size_t)s * PF_W_BYTES, PF_W_BYTES, &full[slot]);
                    pf_bulk_g2s(dst + PF_W_BYTES,
                                A.x_t + ((size_t)(it.s0 + s) * (A.act_rows / 8) + it.pos0 / 8) * kActTileBytes,
                                x_bytes, &full[slot]);
                }
            }
            // no copy is in flight when the block ends, whoever gave up on it
            for (uint32_t p = q > 2 ? q - 2 : 0; p < q; p++) pf_bar_wait(&full[p & 1], (p >> 1) & 1);
        }
    } else if (warp == PF_MMA_WARP) {
        // ---------------- MMA thread: one MMA per 32-column block, two per buffer.  In a warp of its own:
        // as a second lane of the copy thread's warp it ran only when that lane's waits
        // let the warp switch paths.
        if (lane == 0) {
            uint32_t q = 0, kb = 0;
            bool dead = false;
            for (int idx = blockIdx.x; idx < total && !dead && !*(volatile int*)s_abort; idx += gridDim.x) {
                const PfItem it = decode(idx);
                const uint32_t idesc = pf_idesc(kChunkRows, it.n_mma);
                for (int s = 0; s < it.nst && !dead; s++, q++) {
                    const uint32_t slot = q & 1;
                    if (!pf_bar_wait(&full[slot], (q >> 1) & 1)) { give_up(); dead = true; break; }
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
                            const uint64_t bd = pf_desc(xa + 2 * (b + i) * 128, 128, kActTileBytes);
                            pf_mma_i8(tmem + buf * PF_TSTRIDE + i * PF_NT, ad, bd, idesc);
                        }
                        pf_commit(&tfull[buf]);
                    }
                    if (!dead) pf_commit(&empty[slot]);   // the stage's operands are no longer read
                }
            }
            pf_commit(mmas);                              // nor is an MMA
            if (!pf_bar_wait(mmas, 0)) give_up();
        }
    } else {
        // ---------------- epilogue warps
        const int ew = warp - 1;                 // 0..15
        const int quad = warp & 3;               // the tensor-memory lanes this warp may read
        const int cg = ew >> 2;                  // which quarter of the token columns
        const int g = lane >> 2, c = lane & 3;   // places 32 quad + g + 8 i of the chunk, token columns 8 j + 2 c, + 1
        const uint32_t tlane = tmem + ((uint32_t)(32 * quad) << 16);
        uint32_t q = 0, kb = 0, xphase = 0;
        // the epilogue warps meet (bounded): false when the wait gave up
        auto meet = [&]() -> bool {
            __syncwarp();
            if (lane == 0) pf_bar_arrive(xbar);
            const bool ok = pf_together(pf_bar_wait(xbar, xphase));
            xphase ^= 1;
            return ok;
        };
        for (int idx = blockIdx.x; idx < total && pf_together(!*(volatile int*)s_abort); idx += gridDim.x) {
            const PfItem it = decode(idx);
            bool ok = true;
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
                    if (!pf_bar_wait(&full[slot], (q >> 1) & 1)) { ok = false; return; }
                    const uint8_t* wst = stages + slot * PF_STAGE;
                    const uint8_t* xst = wst + PF_W_BYTES + cg * J * kActTileBytes + kActOffDx + c * 8;
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
                            const f32x2 dx = *(const f32x2*)(xst + j * kActTileBytes + b * 32);
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
            if (it.nst == 0) continue;
            // ---- the item's outputs
            if (MODE == PF_GATEUP) {
                // A thread of quadrants 0-1 holds gate rows, its partner in quadrants 2-3 the up
                // rows of the same outputs, for the same tokens.  Each finishes half of them:
                // the gate thread those of the even columns (and hands over its gate values of
                // the odd ones), the up thread the odd ones.
                const int half = quad >> 1;              // 0: gate rows, finishes the even columns
                const int orow = 32 * (quad & 1) + 4 * g;    // output rows orow + i of the chunk (common.cuh: places g + 8 i)
                auto swiglu = [&](auto cols) {
                    constexpr int J = decltype(cols)::value / 8;
                    float* xc = s_xchg + ((quad & 1) * 4 + cg) * 32 + lane;   // [half][i][j][quad, cg, lane]
#pragma unroll
                    for (int i = 0; i < 4; i++)
#pragma unroll
                        for (int j = 0; j < J; j++)
                            xc[((1 - half) * 4 * J + i * J + j) * 256] = half ? lo_of(acc[i][j]) : hi_of(acc[i][j]);
                    if (!meet()) { ok = false; return; }
                    const int r0 = it.chunk * CH + orow;  // rows r0 + i of mid
                    const int tok0 = cg * 8 * J + 2 * c + half;
                    float* mid = A.out + ((size_t)(r0 / 64) * A.act_rows + it.pos0) * 64 + r0 % 64;
                    uint8_t* rec0 = A.out_t + ((size_t)(r0 / 256) * (A.act_rows / 8) + it.pos0 / 8) * kActTileBytes;
#pragma unroll
                    for (int j = 0; j < J; j++) {
                        const int tok = tok0 + 8 * j;
                        float v[4], amax = 0.0f;
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            const float other = xc[(half * 4 * J + i * J + j) * 256];
                            const float gt = half ? other : lo_of(acc[i][j]);
                            const float u = half ? hi_of(acc[i][j]) : other;
                            // ops.rs:160-167: silu(x) = x * (1 / (1 + exp(-x)))
                            v[i] = (gt * __fdiv_rn(1.0f, 1.0f + expf(-gt))) * u;
                            amax = i ? fmaxf(amax, fabsf(v[i])) : fabsf(v[i]);
                        }
                        // Q8Act of the mid rows (quant.rs:368-394; q8_quantize_lane's arithmetic): the
                        // 32 rows of the lanes with the same c are one block of their token
#pragma unroll
                        for (int o = 4; o < 32; o <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
                        const float dd = __fdiv_rn(amax, 127.0f);
                        const float id = dd != 0.0f ? __fdiv_rn(1.0f, dd) : 0.0f;
                        int sum = 0;
                        uint32_t qw = 0;
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            const int q = (int)roundf(__fmul_rn(v[i], id));
                            sum += q;
                            qw |= ((uint32_t)q & 0xffu) << (8 * i);
                        }
#pragma unroll
                        for (int o = 4; o < 32; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
                        if (tok >= it.tc) continue;
                        uint8_t* rec = rec0 + (tok >> 3) * kActTileBytes;
                        *(float4*)(mid + (size_t)tok * 64) = make_float4(v[0], v[1], v[2], v[3]);
                        *(uint32_t*)(rec + act_q_off(tok & 7, r0 % 256)) = qw;
                        if (g < 4) {   // the token's four scales, one lane each
                            const float ss = __fmul_rn(dd, (float)sum);
                            float shi, slo;
                            split_tf32(ss, &shi, &slo);
                            const float val = g == 0 ? dd : g == 1 ? shi : g == 2 ? slo : ss;
                            *(float*)(rec + act_scale_off(g, (r0 % 256) / 32, tok & 7)) = val;
                        }
                    }
                    if (!meet()) ok = false;   // the exchange tile is free again
                };
                if (T == 8) swiglu(std::integral_constant<int, 8>{});
                else if (T == 16) swiglu(std::integral_constant<int, 16>{});
                else swiglu(std::integral_constant<int, 32>{});
                if (!ok) { if (lane == 0) give_up(); break; }
            } else {
                const int rows = (it.shared ? A.sh : A.w).rows;
                const int tok0 = cg * T + 2 * c;
                // the thread's four rows are neighbours, and with those of eight lanes 128 bytes of a token's row
                float* dst = A.out + ((size_t)it.part * A.part_rows + it.pos0 + tok0) * rows + it.chunk * CH + 32 * quad + 4 * g;
#pragma unroll
                for (int j = 0; j < PF_COLS / 8; j++) {
                    if (8 * j >= T) break;
                    if (tok0 + 8 * j < it.tc)
                        *(float4*)(dst + (size_t)(8 * j) * rows) = make_float4(lo_of(acc[0][j]), lo_of(acc[1][j]), lo_of(acc[2][j]), lo_of(acc[3][j]));
                    if (tok0 + 8 * j + 1 < it.tc)
                        *(float4*)(dst + (size_t)(8 * j + 1) * rows) = make_float4(hi_of(acc[0][j]), hi_of(acc[1][j]), hi_of(acc[2][j]), hi_of(acc[3][j]));
                }
            }
        }
    }
    pf_fence_before();
    __syncthreads();
    pf_fence_after();
    if (warp == 0) {
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
    count_launch();
    return launch_after(c.stream, experts_prefill_kernel<MODE>, dim3(c.sm_count), dim3(PF_THREADS), PF_SMEM, A);
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
    return launch_prefill_one<PF_DOWN>(c, D);
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
