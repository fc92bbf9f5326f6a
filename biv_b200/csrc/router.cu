// Router product, softmax / top-k / renormalisation, and the stable
// token-to-expert sort.  Reference: engine/src/model.rs:259-268 (route),
// 864-873 (logits and per-expert lists), engine/src/ops.rs:192-201 (softmax),
// engine/src/quant.rs:1177-1206 (the AVX2 f32 dot whose summation order the
// logits kernel reproduces bit for bit).
#include <algorithm>

#include "common.cuh"
#include "formats.cuh"
#include "launch.cuh"
#include "tcgen05.cuh"
#include "topk.cuh"

namespace bivmoe {

// ---------------------------------------------------------------------------
// logits[t][r] = dot(W[r], h[t]) for the n_expert router rows plus, as row
// n_expert, the shared expert's gate vector.
//
// The reference's x86 dot keeps 4 accumulators of 8 lanes: element i goes to
// lane (i mod 32) of a 32-wide accumulator set, with one fused multiply-add per
// element in ascending i, and the 32 lanes are then summed as
// (k0+k1)+(k2+k3) per lane j (lane = 8k+j), then j with j+4, j+2, j+1.  A warp
// lane per accumulator lane and the butterfly 8,16,4,2,1 give the same bits.
constexpr int RT_TOKS = 4, RT_BTOKS = 16;        // tokens of one warp (with one row) and of one block
constexpr int RT_THREADS = 256;
constexpr uint32_t RT_WAIT_LIMIT = 1u << 20;

__device__ __forceinline__ uint32_t rt_smem_u32(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

// Few tokens: the block's two weight rows and the activation rows there are (16 at most)
// are brought into shared memory with one bulk copy each, all in flight together, so the
// kernel pays one memory round trip instead of one per step of the dot.  Two rows a block
// put 129 blocks of 257 rows on the 148 SMs, and what one SM has to bring in and
// work off is what bounds the kernel: with 8 rows and always 16 tokens one token took 5.9 us.
template <int RT_ROWS>
__global__ void __launch_bounds__(RT_THREADS, 1)
router_logits_kernel(const float* __restrict__ W, const float* __restrict__ h,
                     float* __restrict__ logits, int n, int e, int n_rows, int* status,
                     const float* __restrict__ norm_w, float norm_eps, float* __restrict__ row_scale) {
    constexpr int RT_BROWS = 2 * RT_ROWS;
    pdl_enter();
    extern __shared__ __align__(128) uint8_t rt_smem[];
    uint64_t* bar = (uint64_t*)rt_smem;
    float* s_w = (float*)(rt_smem + 128);              // [RT_BROWS][e]
    float* s_x = s_w + (size_t)RT_BROWS * e;           // [RT_BTOKS][e]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int br0 = blockIdx.x * RT_BROWS, bt0 = blockIdx.y * RT_BTOKS;
    const int toks = min(RT_BTOKS, n - bt0);
    const uint32_t row_bytes = (uint32_t)e * 4;
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(rt_smem_u32(bar)));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (warp == 0) {
        if (lane == 0)
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(rt_smem_u32(bar)),
                         "r"(row_bytes * (uint32_t)(RT_BROWS + toks))
                         : "memory");
        __syncwarp();
        if (lane < RT_BROWS + toks) {   // router rows past the end repeat the last one; never stored
            const float* src = lane < RT_BROWS ? W + (size_t)min(br0 + lane, n_rows - 1) * e
                                               : h + (size_t)(bt0 + lane - RT_BROWS) * e;
            float* dst = lane < RT_BROWS ? s_w + (size_t)lane * e : s_x + (size_t)(lane - RT_BROWS) * e;
            asm volatile(
                "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
                    "r"(rt_smem_u32(dst)),
                "l"(src), "r"(row_bytes), "r"(rt_smem_u32(bar))
                : "memory");
        }
    }
    bool ok = false;
    for (uint32_t i = 0; i < RT_WAIT_LIMIT && !ok; i++) {
        uint32_t p;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(p)
            : "r"(rt_smem_u32(bar))
            : "memory");
        ok = p != 0;
    }
    if (!ok) {   // bounded wait gave up: every thread waits on the same barrier
        if (threadIdx.x == 0) atomicExch(status, BIVMOE_ERR_TIMEOUT);
        return;
    }
    if (norm_w) {
        // The rows are the residual x: the layer's input is rms_norm(x) (ops.rs:136-149),
        // h = x * (scale * w) with scale = 1 / sqrt(dot(x, x) / e + eps), the dot in the
        // lane order of the reference's AVX2 kernel.  Normalised in place in shared
        // memory, so the normed rows never travel through HBM; the block of the first
        // router rows publishes the scales for the kernels that read x after this one.
        for (int tr = warp; tr < toks; tr += RT_THREADS / 32) {
            float* xr = s_x + (size_t)tr * e;
            float ss = 0.0f;
            for (int i = lane; i < e; i += 32) ss = fmaf(xr[i], xr[i], ss);
            ss = __fadd_rn(ss, __shfl_xor_sync(0xffffffffu, ss, 8));
            ss = __fadd_rn(ss, __shfl_xor_sync(0xffffffffu, ss, 16));
            ss = __fadd_rn(ss, __shfl_xor_sync(0xffffffffu, ss, 4));
            ss = __fadd_rn(ss, __shfl_xor_sync(0xffffffffu, ss, 2));
            ss = __fadd_rn(ss, __shfl_xor_sync(0xffffffffu, ss, 1));
            const float scale = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ss, (float)e), norm_eps)));
            for (int i = lane; i < e; i += 32) xr[i] = __fmul_rn(xr[i], __fmul_rn(scale, norm_w[i]));
            if (lane == 0 && blockIdx.x == 0) row_scale[bt0 + tr] = scale;
        }
        __syncthreads();
    }
    const int r0 = (warp & 1) * RT_ROWS, t0 = (warp >> 1) * RT_TOKS;   // inside the block
    if (t0 >= toks) return;   // (a token past the end beside others: its row is read as it lies, never stored)
    float acc[RT_ROWS][RT_TOKS] = {};
#pragma unroll 4
    for (int i = lane; i < e; i += 32) {
        float w[RT_ROWS], x[RT_TOKS];
#pragma unroll
        for (int r = 0; r < RT_ROWS; r++) w[r] = s_w[(size_t)(r0 + r) * e + i];
#pragma unroll
        for (int t = 0; t < RT_TOKS; t++) x[t] = s_x[(size_t)(t0 + t) * e + i];
#pragma unroll
        for (int r = 0; r < RT_ROWS; r++)
#pragma unroll
            for (int t = 0; t < RT_TOKS; t++) acc[r][t] = fmaf(w[r], x[t], acc[r][t]);
    }
#pragma unroll
    for (int r = 0; r < RT_ROWS; r++)
#pragma unroll
        for (int t = 0; t < RT_TOKS; t++) {
            float v = acc[r][t];
            v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 8));
            v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 16));
            v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 4));
            v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 2));
            v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 1));
            const int row = br0 + r0 + r, tok = bt0 + t0 + t;
            if (lane == 0 && row < n_rows && tok < n) logits[(size_t)tok * n_rows + row] = v;
        }
}

// The same product for more tokens: a block of 8 warps computes 16 rows x 4 TOKS
// tokens, a warp 8 rows x TOKS tokens (16: 128 accumulators per lane, so 24 shared-
// memory loads feed 128 multiply-adds), over K in chunks of 256 values that a
// two-stage ring of 16-byte asynchronous copies keeps in flight (a chunk of
// one row is 1024 bytes: too small for bulk copies to pay; chunks of 128 in three
// stages, twice the barriers, took 467 us instead of 450 for 16 384 tokens).  The multiply-adds are issued
// two tokens at a time (fma.rn.f32x2; measured 0.64 -> 0.56 ms at 16 384 tokens).  The per-lane order of the
// multiply-adds and the order of the final lane sums are those of the small
// kernel above, so the logits are the same bits.
constexpr int RL_ROWS = 8, RL_BROWS = 16;             // rows of one warp and of one block
constexpr int RL_KC = 256, RL_STAGES = 2;
__host__ __device__ constexpr int rl_stage_floats(int toks) { return (RL_BROWS + 4 * toks) * RL_KC; }
__host__ __device__ constexpr int rl_smem(int toks) { return 128 + RL_STAGES * rl_stage_floats(toks) * 4; }   // 163968 for 16

// one step of the lane sums: the lanes of a pair (lane ^ M) split the 2 * HALF values
template <int HALF, int M, int N>
__device__ __forceinline__ void rl_reduce_step(float (&acc)[N], int lane, int& base) {
    const bool up = (lane & M) != 0;
#pragma unroll
    for (int j = 0; j < HALF; j++) {
        const float a = acc[j], b = acc[j + HALF];
        const float send = up ? a : b, keep = up ? b : a;
        acc[j] = __fadd_rn(keep, __shfl_xor_sync(0xffffffffu, send, M));
    }
    if (up) base += HALF;
}

template <int RL_TOKS>
__global__ void __launch_bounds__(RT_THREADS, RL_TOKS == 16 ? 1 : 2)
router_logits_tiled_kernel(const float* __restrict__ W, const float* __restrict__ h,
                           float* __restrict__ logits, int n, int e, int n_rows) {
    constexpr int RL_BTOKS = 4 * RL_TOKS, RL_STAGE_FLOATS = rl_stage_floats(RL_TOKS);
    pdl_enter();
    extern __shared__ __align__(128) uint8_t rt_smem[];
    float* ring = (float*)(rt_smem + 128);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int br0 = blockIdx.x * RL_BROWS, bt0 = blockIdx.y * RL_BTOKS;
    const int nchunk = e / RL_KC;
    // every thread copies 16-byte pieces of chunk c into stage `c % RL_STAGES`: columns `lane`
    // and `lane + 32` of rows `warp + 8j` of the stage (rows 0-15 router rows, then token
    // rows); the rows' addresses are worked out once.  Token rows past the end repeat the last one;
    // router rows past the end are not loaded: their sums, of whatever the stage held, are not stored
    static_assert(RT_THREADS == 256 && RL_KC % 128 == 0, "8 warps, 128 values a warp-wide piece");
    constexpr int RL_PIECES = (RL_BROWS + RL_BTOKS) / 8;
    const float* rowp[RL_PIECES];
#pragma unroll
    for (int j = 0; j < RL_PIECES; j++) {
        const int r = warp + 8 * j;
        rowp[j] = (r < RL_BROWS ? W + (size_t)min(br0 + r, n_rows - 1) * e
                                : h + (size_t)min(bt0 + r - RL_BROWS, n - 1) * e) + lane * 4;
    }
    const uint32_t ring_u32 = rt_smem_u32(ring) + (uint32_t)(warp * RL_KC + lane * 4) * 4;
    const int wrows = min(RL_BROWS, n_rows - br0);   // router rows there are
    auto fill = [&](int c) {
        const uint32_t st = ring_u32 + (uint32_t)(c % RL_STAGES) * (RL_STAGE_FLOATS * 4);
#pragma unroll
        for (int j = 0; j < RL_PIECES; j++) {
            if (j < 2 && warp + 8 * j >= wrows) continue;
#pragma unroll
            for (int p = 0; p < RL_KC / 128; p++)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(st + j * 8 * RL_KC * 4 + p * 512),
                             "l"(rowp[j] + (size_t)c * RL_KC + p * 128)
                             : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int c = 0; c < RL_STAGES - 1; c++) {
        if (c < nchunk) fill(c);
        else asm volatile("cp.async.commit_group;" ::: "memory");
    }
    if (br0 + 1 == n_rows) {
        // One row is left for the last row block (256 experts and the shared gate): a warp takes it
        // with an eighth of the tokens, in the same order, instead of sixteen rows of which fifteen
        // are repeats of it (16384 tokens 454 -> 444 us, 4096 tokens 128 -> 122).
        constexpr int LT = RL_BTOKS / 8;
        float acc[LT] = {};
        for (int c = 0; c < nchunk; c++) {
            asm volatile("cp.async.wait_group %0;" ::"n"(RL_STAGES - 2) : "memory");
            __syncthreads();
            if (c + RL_STAGES - 1 < nchunk) fill(c + RL_STAGES - 1);
            else asm volatile("cp.async.commit_group;" ::: "memory");
            const float* sw = ring + (size_t)(c % RL_STAGES) * RL_STAGE_FLOATS + lane;
            const float* sx = sw + (size_t)(RL_BROWS + warp * LT) * RL_KC;
#pragma unroll
            for (int kk = 0; kk < RL_KC / 32; kk++) {
                const float w = sw[kk * 32];
#pragma unroll
                for (int t = 0; t < LT; t++) acc[t] = fmaf(w, sx[t * RL_KC + kk * 32], acc[t]);
            }
        }
#pragma unroll
        for (int t = 0; t < LT; t++) {
            float v = acc[t];
            v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 8));
            v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 16));
            v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 4));
            v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 2));
            v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 1));
            const int tok = bt0 + warp * LT + t;
            if (lane == 0 && tok < n) logits[(size_t)tok * n_rows + br0] = v;
        }
        return;
    }
    const int r0 = (warp & 1) * RL_ROWS, t0 = (warp >> 1) * RL_TOKS;   // inside the block
    // two tokens per multiply-add (fma.rn.f32x2: each half rounds as the scalar form does,
    // so the logits keep their bits): acc2[r][j] = tokens 2j, 2j+1 of row r
    f32x2 acc2[RL_ROWS * RL_TOKS / 2];
#pragma unroll
    for (int i = 0; i < RL_ROWS * RL_TOKS / 2; i++) acc2[i] = 0ull;
    for (int c = 0; c < nchunk; c++) {
        // chunk c has landed (one younger group may still be in flight); after the barrier
        // everyone is also done with chunk c - 1, whose stage chunk c + RL_STAGES - 1 reuses
        asm volatile("cp.async.wait_group %0;" ::"n"(RL_STAGES - 2) : "memory");
        __syncthreads();
        if (c + RL_STAGES - 1 < nchunk) fill(c + RL_STAGES - 1);
        else asm volatile("cp.async.commit_group;" ::: "memory");
        const float* sw = ring + (size_t)(c % RL_STAGES) * RL_STAGE_FLOATS + (size_t)r0 * RL_KC;
        const float* sx = ring + (size_t)(c % RL_STAGES) * RL_STAGE_FLOATS +
                          (size_t)(RL_BROWS + t0) * RL_KC;
#pragma unroll
        for (int kk = 0; kk < RL_KC / 32; kk++) {
            const int i = kk * 32 + lane;
            float w[RL_ROWS];
            f32x2 x2[RL_TOKS / 2];
#pragma unroll
            for (int r = 0; r < RL_ROWS; r++) w[r] = sw[r * RL_KC + i];
#pragma unroll
            for (int t = 0; t < RL_TOKS / 2; t++) x2[t] = pk(sx[(2 * t) * RL_KC + i], sx[(2 * t + 1) * RL_KC + i]);
#pragma unroll
            for (int r = 0; r < RL_ROWS; r++) {
                const f32x2 w2 = pk(w[r], w[r]);
#pragma unroll
                for (int t = 0; t < RL_TOKS / 2; t++)
                    acc2[r * (RL_TOKS / 2) + t] = fma2(w2, x2[t], acc2[r * (RL_TOKS / 2) + t]);
            }
        }
    }
    float acc[RL_ROWS * RL_TOKS];
#pragma unroll
    for (int i = 0; i < RL_ROWS * RL_TOKS / 2; i++) {
        acc[2 * i] = lo_of(acc2[i]);
        acc[2 * i + 1] = hi_of(acc2[i]);
    }
    // Lane sums in the order 8, 16, 4, 2, 1.  Each step halves the values a lane
    // carries: a lane keeps the half chosen by its bit of the step and gives the
    // other half to its partner, which adds the same two numbers as a full
    // butterfly would.  A lane ends with 4 of the warp's 128 outputs.
    int base = 0;
    constexpr int N = RL_ROWS * RL_TOKS;
    rl_reduce_step<N / 2, 8>(acc, lane, base);
    rl_reduce_step<N / 4, 16>(acc, lane, base);
    rl_reduce_step<N / 8, 4>(acc, lane, base);
    rl_reduce_step<N / 16, 2>(acc, lane, base);
    rl_reduce_step<N / 32, 1>(acc, lane, base);
#pragma unroll
    for (int j = 0; j < N / 32; j++) {
        const int o = base + j;
        const int row = br0 + r0 + o / RL_TOKS, tok = bt0 + t0 + o % RL_TOKS;
        if (row < n_rows && tok < n) logits[(size_t)tok * n_rows + row] = acc[j];
    }
}

// The same product for many tokens: a persistent block of 8 warps works off tiles of 32 rows x 4 TOKS tokens, a
// warp 16 rows x TOKS tokens, i.e. 28 shared-memory loads for 192 multiply-adds a lane at TOKS = 12.  The rows'
// chunks of 256 values come by bulk copy, a few lanes of every warp, one chunk ahead and on into the
// next tile, so that neither addresses nor the start of a tile cost anything.  What bounds it: the f32
// multiply-adds, two an instruction, of which one is issued every 2.3 clk per scheduler (a loop of nothing else),
// 285 us for 16384 rows of 2048 / 257; it takes 385 to 393 (the kernel above 441, tiles of 32 x 48 by it 405),
// 4096 rows 103 (117), 2048 rows 55 (64).
constexpr int RS_ROWS = 16, RS_BROWS = 2 * RS_ROWS;
__host__ __device__ constexpr int rs_row_tiles(int n_rows) { return (n_rows + RS_BROWS - 2) / RS_BROWS; }   // without a last row by itself
__host__ __device__ constexpr int rs_stage_floats(int toks) { return (RS_BROWS + 4 * toks) * RL_KC; }
__host__ __device__ constexpr int rs_smem(int toks) { return 128 + 2 * rs_stage_floats(toks) * 4; }

template <int TOKS>
__global__ void __launch_bounds__(RT_THREADS, 1)
router_logits_stream_kernel(const float* __restrict__ W, const float* __restrict__ h, float* __restrict__ logits, int n,
                            int e, int n_rows, int* status) {
    constexpr int BTOKS = 4 * TOKS, STAGE_FLOATS = rs_stage_floats(TOKS), COPIES = (RS_BROWS + BTOKS) / 8;
    static_assert(COPIES <= 32 && RS_BROWS % 8 == 0, "a lane a row");
    extern __shared__ __align__(128) uint8_t rt_smem[];
    uint64_t *full = (uint64_t*)rt_smem, *empty = full + 2;   // [2] of a stage: every warp's copies; every warp is done with it
    float* ring = (float*)(rt_smem + 128);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        for (int i = 0; i < 4; i++) pf_bar_init(&full[i], RT_THREADS / 32);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    pdl_enter();
    const int nchunk = e / RL_KC, tiles_t = (n + BTOKS - 1) / BTOKS;
    // The block's tiles: of the whole row tiles' every gridDim.x-th, the row tiles of the same tokens next to each
    // other; then of the tiles of one last row, which take a third of the time: the first ones go to the
    // blocks that had one of the others fewer, three each.
    const int G = gridDim.x, b = blockIdx.x, tiles_r = rs_row_tiles(n_rows), whole = tiles_r * tiles_t;
    const int ends = n_rows % RS_BROWS == 1 ? tiles_t : 0, more = whole % G, fewer = G - more, ahead = min(ends, 3 * fewer);
    auto share = [](int count, int first, int step) { return count > first ? (count - first + step - 1) / step : 0; };
    const int mine_whole = share(whole, b, G), mine_ahead = b >= more ? share(ahead, b - more, fewer) : 0;
    const int tiles = mine_whole + mine_ahead + share(ends - ahead, b, G);
    auto rows_of = [&](int i) { return i < mine_whole ? (b + i * G) % tiles_r * RS_BROWS : tiles_r * RS_BROWS; };
    auto toks_of = [&](int i) {
        if (i < mine_whole) return (b + i * G) / tiles_r * BTOKS;
        i -= mine_whole;
        return (i < mine_ahead ? b - more + i * fewer : ahead + b + (i - mine_ahead) * G) * BTOKS;
    };
    bool ok = true;
    // chunk c of the block's i-th tile, its q-th chunk: lane l copies row warp + 8 l of the stage (router rows,
    // then token rows; token rows past the end repeat the last one, router rows past the end stay away: their
    // sums, of whatever the stage held, are not stored).  `landed`: what the lane got of its wait for the chunk
    // that it has begun with.  The lanes of a warp go on, or leave, together: this vote is for both waits.
    auto fill = [&](uint32_t q, int i, int c, bool landed) {
        const uint32_t slot = q & 1;
        if (!pf_together(landed && pf_bar_wait(&empty[slot], ((q >> 1) & 1) ^ 1))) { ok = false; return; }
        const int r = warp + 8 * lane, row0 = rows_of(i) + warp, tok = min(toks_of(i) + r - RS_BROWS, n - 1);
        const int rows = min(RS_BROWS / 8, (n_rows - row0 + 7) / 8);   // router rows there are (a tile has one: n_rows - row0 > -7)
        const bool mine = lane < COPIES && (r >= RS_BROWS || lane < rows);
        if (lane == 0) pf_bar_expect_tx(&full[slot], (rows + BTOKS / 8) * RL_KC * 4);
        __syncwarp();
        if (mine)
            pf_bulk_g2s(ring + (size_t)slot * STAGE_FLOATS + r * RL_KC,
                        (r < RS_BROWS ? W + (size_t)(row0 + 8 * lane) * e : h + (size_t)tok * e) + c * RL_KC, RL_KC * 4, &full[slot]);
    };
    uint32_t q = 0;   // chunks worked off
    if (tiles > 0) fill(0, 0, 0, true);
    for (int i = 0; i < tiles && ok; i++) {
        const int br0 = rows_of(i), bt0 = toks_of(i);
        auto next = [&](int c, bool landed) {   // the chunk after this one
            if (c + 1 < nchunk) fill(q + 1, i, c + 1, landed);
            else if (i + 1 < tiles) fill(q + 1, i + 1, 0, landed);
            else ok = pf_together(landed);
        };
        if (i >= mine_whole) {   // as in the kernel above
            constexpr int LT = (BTOKS + 7) / 8;
            float acc[LT] = {};
            for (int c = 0; c < nchunk; c++, q++) {
                next(c, pf_bar_wait(&full[q & 1], (q >> 1) & 1));
                if (!ok) break;
                const float* sw = ring + (size_t)(q & 1) * STAGE_FLOATS + lane;
#pragma unroll
                for (int kk = 0; kk < RL_KC / 32; kk++) {
                    const float w = sw[kk * 32];
#pragma unroll
                    for (int t = 0; t < LT; t++) acc[t] = fmaf(w, sw[(RS_BROWS + warp * LT + t) * RL_KC + kk * 32], acc[t]);
                }
                __syncwarp();
                if (lane == 0) pf_bar_arrive(&empty[q & 1]);
            }
#pragma unroll
            for (int t = 0; t < LT; t++) {
                float v = acc[t];
                v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 8));
                v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 16));
                v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 4));
                v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 2));
                v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 1));
                const int tok = bt0 + warp * LT + t;
                if (lane == 0 && tok < n && warp * LT + t < BTOKS) logits[(size_t)tok * n_rows + br0] = v;
            }
            continue;
        }
        const int r0 = (warp & 1) * RS_ROWS, t0 = (warp >> 1) * TOKS;   // inside the tile
        f32x2 acc2[TOKS * RS_ROWS / 2];   // [token][two rows]
#pragma unroll
        for (int i = 0; i < TOKS * RS_ROWS / 2; i++) acc2[i] = 0ull;
        for (int c = 0; c < nchunk; c++, q++) {
            const bool landed = pf_bar_wait(&full[q & 1], (q >> 1) & 1);
            const float* sw = ring + (size_t)(q & 1) * STAGE_FLOATS + r0 * RL_KC + lane;
            const float* sx = ring + (size_t)(q & 1) * STAGE_FLOATS + (RS_BROWS + t0) * RL_KC + lane;
#pragma unroll
            for (int kk = 0; kk < RL_KC / 32; kk++) {
                float x[TOKS];
                f32x2 w2[RS_ROWS / 2];
#pragma unroll
                for (int t = 0; t < TOKS; t++) x[t] = sx[t * RL_KC + kk * 32];
#pragma unroll
                for (int r = 0; r < RS_ROWS / 2; r++) w2[r] = pk(sw[2 * r * RL_KC + kk * 32], sw[(2 * r + 1) * RL_KC + kk * 32]);
#pragma unroll
                for (int t = 0; t < TOKS; t++) {
                    const f32x2 x2 = pk(x[t], x[t]);
#pragma unroll
                    for (int r = 0; r < RS_ROWS / 2; r++) acc2[t * (RS_ROWS / 2) + r] = fma2(x2, w2[r], acc2[t * (RS_ROWS / 2) + r]);
                }
                if (kk == 0) next(c, landed);   // by now the others are done with the chunk before, whose stage it takes
            }
            __syncwarp();
            if (!ok) break;
            if (lane == 0) pf_bar_arrive(&empty[q & 1]);
        }
        float acc[TOKS * RS_ROWS];
#pragma unroll
        for (int i = 0; i < TOKS * RS_ROWS / 2; i++) {
            acc[2 * i] = lo_of(acc2[i]);
            acc[2 * i + 1] = hi_of(acc2[i]);
        }
        int base = 0;   // lane sums in the order 8, 16, 4, 2, 1, as above
        constexpr int N = TOKS * RS_ROWS;
        rl_reduce_step<N / 2, 8>(acc, lane, base);
        rl_reduce_step<N / 4, 16>(acc, lane, base);
        rl_reduce_step<N / 8, 4>(acc, lane, base);
        rl_reduce_step<N / 16, 2>(acc, lane, base);
        rl_reduce_step<N / 32, 1>(acc, lane, base);
#pragma unroll
        for (int j = 0; j < N / 32; j++) {
            const int o = base + j, row = br0 + r0 + o % RS_ROWS, tok = bt0 + t0 + o / RS_ROWS;
            if (row < n_rows && tok < n) logits[(size_t)tok * n_rows + row] = acc[j];
        }
    }
    if (!ok) {   // every copy this warp began has landed, or was waited for, when the block ends
        if (lane == 0) atomicExch(status, BIVMOE_ERR_TIMEOUT);
        pf_bar_wait(&full[q & 1], (q >> 1) & 1);
        pf_bar_wait(&full[(q + 1) & 1], ((q + 1) >> 1) & 1);
    }
}

// The kernel that stages whole rows serves up to 16 tokens with one row a warp, and more with
// four while its blocks (8 rows, 16 tokens, one per SM) fit on the chip at once, if the rows
// fit in shared memory.
static size_t router_stage_bytes(int rows, int e) { return 128 + (2 * (size_t)rows + RT_BTOKS) * e * 4; }
static bool router_stages_few(int n, int e) { return n <= RT_BTOKS && router_stage_bytes(1, e) <= 227 * 1024; }
static bool router_stages_more(const LaunchCfg& c) {
    return (c.n_expert + 8) / 8 * ((c.n + RT_BTOKS - 1) / RT_BTOKS) <= c.sm_count && router_stage_bytes(4, c.e) <= 227 * 1024;
}
// It also applies a norm, for one block of tokens: for more rows the norm would be done again
// by every block of router rows (27 us for 160 tokens; by themselves the norm and the product
// take 4 + 11).
bool router_fuses_norm(int n, int e) { return router_stages_few(n, e); }

template <int ROWS>
static cudaError_t launch_router_staged(const LaunchCfg& c, const float* router_dev, const float* h, const Workspace& ws,
                                        const RowNorm* norm) {
    const int n_rows = c.n_expert + 1;
    static std::atomic<uint64_t> attr_set{0};
    if (cudaError_t err = ensure_dynamic_smem(router_logits_kernel<ROWS>, 227 * 1024, attr_set)) return err;
    count_launch();
    return launch_after(c.stream, router_logits_kernel<ROWS>,
                        dim3((n_rows + 2 * ROWS - 1) / (2 * ROWS), (c.n + RT_BTOKS - 1) / RT_BTOKS), dim3(RT_THREADS),
                        router_stage_bytes(ROWS, c.e), router_dev, h, ws.logits, c.n, c.e, n_rows, ws.status,
                        norm ? norm->w : (const float*)nullptr, norm ? norm->eps : 0.0f, ws.row_scale);
}

template <int TOKS>
static cudaError_t launch_router_tiled(const LaunchCfg& c, const float* router_dev, const float* h, const Workspace& ws) {
    const int n_rows = c.n_expert + 1;
    static std::atomic<uint64_t> attr_set{0};
    if (cudaError_t err = ensure_dynamic_smem(router_logits_tiled_kernel<TOKS>, rl_smem(TOKS), attr_set)) return err;
    dim3 grid((n_rows + RL_BROWS - 1) / RL_BROWS, (c.n + 4 * TOKS - 1) / (4 * TOKS));
    count_launch();
    return launch_after(c.stream, router_logits_tiled_kernel<TOKS>, grid, dim3(RT_THREADS), rl_smem(TOKS), router_dev, h,
                        ws.logits, c.n, c.e, n_rows);
}

template <int TOKS>
static cudaError_t launch_router_stream(const LaunchCfg& c, const float* router_dev, const float* h, const Workspace& ws) {
    const int n_rows = c.n_expert + 1, tiles = (n_rows + RS_BROWS - 1) / RS_BROWS * ((c.n + 4 * TOKS - 1) / (4 * TOKS));
    static std::atomic<uint64_t> attr_set{0};
    if (cudaError_t err = ensure_dynamic_smem(router_logits_stream_kernel<TOKS>, rs_smem(TOKS), attr_set)) return err;
    count_launch();
    return launch_after(c.stream, router_logits_stream_kernel<TOKS>, dim3(std::min(tiles, c.sm_count)), dim3(RT_THREADS), rs_smem(TOKS),
                        router_dev, h, ws.logits, c.n, c.e, n_rows, ws.status);
}

cudaError_t launch_router(const LaunchCfg& c, const float* router_dev, const float* h,
                          const Workspace& ws, const RowNorm* norm) {
    if (router_stages_few(c.n, c.e)) return launch_router_staged<1>(c, router_dev, h, ws, norm);
    if (norm) return cudaErrorInvalidValue;
    if (router_stages_more(c)) return launch_router_staged<4>(c, router_dev, h, ws, nullptr);
    // K travels in chunks of 256 values.  The more a block takes at a time the fewer loads its
    // multiply-adds need and the longer it runs.  Where all blocks of 16 or 32 tokens are on the chip at once, those
    // (8.4 and 11.5 us); else whichever takes the fewest turns: by its tiles, a turn of 16 x 64
    // is 16.5 us (2048 columns), of 32 x 40 18, of 32 x 48 20.  (16384 rows 441, 419 and 385 us.)  Turns
    // grow with the columns alike: from 512 to 4096 of them, 60 to 512 experts and 700 to 6000 rows, what the rule takes was
    // never slower than blocks of 16 x 64 and 1.05 to 1.5 times as fast where it differs.
    if (c.e % RL_KC) return cudaErrorInvalidValue;
    const int row_blocks = (c.n_expert + RL_BROWS) / RL_BROWS;
    auto at_once = [&](int toks) { return row_blocks * ((c.n + toks - 1) / toks) <= c.sm_count; };
    if (at_once(16)) return launch_router_tiled<4>(c, router_dev, h, ws);
    if (at_once(32)) return launch_router_tiled<8>(c, router_dev, h, ws);
    auto cost = [&](int row_tiles, int toks, int turn) {
        return ((long long)row_tiles * ((c.n + toks - 1) / toks) + c.sm_count - 1) / c.sm_count * turn;
    };
    const long long c16 = cost((c.n_expert + RL_BROWS - 1) / RL_BROWS, 64, 165), c10 = cost(rs_row_tiles(c.n_expert + 1), 40, 180),
                    c12 = cost(rs_row_tiles(c.n_expert + 1), 48, 200);
    return c16 <= std::min(c10, c12) ? launch_router_tiled<16>(c, router_dev, h, ws)
         : c10 < c12 ? launch_router_stream<10>(c, router_dev, h, ws) : launch_router_stream<12>(c, router_dev, h, ws);
}

// ---------------------------------------------------------------------------
// A warp per token (topk.cuh).
constexpr int TK_WARPS = 4, TK_MAX_EXPERTS = 1024, TK_MAX_K = 32;

// The blocks behind those of the top-k, one a row, make the rows ready, which the routing has no part in: the
// top-k is a chain of latencies that leaves the chip to them, and a launch of their own took 2 us (509
// rows quantised) to 36 (16384 split) more.
template <int M>
__global__ void __launch_bounds__(TK_WARPS * 32)
route_topk_kernel(const float* __restrict__ logits, int32_t* __restrict__ ids,
                  float* __restrict__ weights, int n, int n_expert, int k, const float* __restrict__ h, Workspace ws, int e,
                  int rows) {
    pdl_enter();
    extern __shared__ __align__(16) float tk_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, topk_blocks = (n + TK_WARPS - 1) / TK_WARPS;
    if ((int)blockIdx.x >= topk_blocks) {
        const size_t row = blockIdx.x - topk_blocks, at = row * e;
        if (rows == ROWS_QUANT) quantize_row(h + at, ws.tok_q + at, ws.tok_s + at / 32, e);
        else split_row(h + at, ws.tok_b + row * (e / 64) * kTokBRec, e);
        return;
    }
    const int t = blockIdx.x * TK_WARPS + warp;
    if (t >= n) return;
    int id;
    float w;
    topk_token<M>(logits + (size_t)t * (n_expert + 1), tk_smem + (size_t)warp * ((n_expert + 3) & ~3), n_expert, k, lane,
                  id, w);
    if (lane < k) {
        ids[(size_t)t * k + lane] = id;
        weights[(size_t)t * k + lane] = w;
    }
}

cudaError_t launch_route_topk(const LaunchCfg& c, const Workspace& ws, const float* h, RowsReady rows) {
    if (c.n_expert > TK_MAX_EXPERTS || c.k > TK_MAX_K) return cudaErrorInvalidValue;
    const size_t smem = (size_t)TK_WARPS * ((c.n_expert + 3) & ~3) * sizeof(float);
    count_launch();
    return launch_early(c.n, c.stream, c.n_expert <= 256 ? route_topk_kernel<8> : route_topk_kernel<TK_MAX_EXPERTS / 32>,
                        dim3((c.n + TK_WARPS - 1) / TK_WARPS + (rows != ROWS_NONE ? c.n : 0)), dim3(TK_WARPS * 32), smem,
                        (const float*)ws.logits, ws.ids, ws.weights, c.n, c.n_expert, c.k, rows != ROWS_NONE ? h : (const float*)nullptr, ws,
                        c.e, (int)rows);
}

// ---------------------------------------------------------------------------
// Stable grouping of the n*k (token, expert) pairs by expert: inside an expert
// pairs keep ascending pair index t*k+j, which is the order the reference
// pushes them in (model.rs:867-873; Metal moe_sort, kernels.metal:1723-1729).
// A block owns SORT_TOKENS consecutive tokens.  Phase 1 counts per (block,
// expert); phase 2 turns the counts into bases (exclusive over blocks, then
// over experts) and builds the list of non-empty groups; phase 3 places every
// pair by its base and its rank in the expert's bitmask.  With one block the three
// phases run in a single launch (509 tokens 10.8 us; by one block 18, by a cluster of two, one launch, 10.3).
constexpr int SORT_TOKENS = 256, SORT_THREADS = 256, SORT_MANY = 1024;   // threads, and with more than SORT_THREADS pairs
constexpr uint16_t kNoExpert = 0xFFFF;
constexpr int SORT_TILE = 8;   // every group starts at a multiple of this

// A token selects an expert at most once: an expert's bitmask over the block's tokens gives its count, and
// the rank of pair (t, j) inside it, the number of earlier tokens that selected the expert.
constexpr int SORT_WORDS = SORT_TOKENS / 32;
__device__ __forceinline__ int sort_count(const uint32_t* s_mask, int e) {
    const uint4 a = *(const uint4*)(s_mask + e * SORT_WORDS), b = *(const uint4*)(s_mask + e * SORT_WORDS + 4);
    return __popc(a.x) + __popc(a.y) + __popc(a.z) + __popc(a.w) + __popc(b.x) + __popc(b.y) + __popc(b.z) + __popc(b.w);
}
// id(i) of pair i, to s_ids and into the masks.  A thread has the same pairs here and in sort_scatter.
template <class Id>
__device__ void sort_build_masks(Id id, int npairs, int k, int n_expert, uint16_t* s_ids, uint32_t* s_mask) {
    // a negative id marks an empty slot (a row with fewer than k experts: expert parallelism)
    const int first = threadIdx.x < npairs ? id(threadIdx.x) : -1;   // on its way while the masks are cleared
    for (int i = threadIdx.x; i < n_expert * SORT_WORDS; i += blockDim.x) s_mask[i] = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < npairs; i += blockDim.x) {
        const int e = i == threadIdx.x ? first : id(i), t = i / k;
        s_ids[i] = e < 0 ? kNoExpert : (uint16_t)e;
        if (e >= 0) atomicOr(&s_mask[e * SORT_WORDS + (t >> 5)], 1u << (t & 31));
    }
    __syncthreads();
}
// Exclusive scans over the block of N sequences at once (one set of barriers), ITEMS
// consecutive slots per thread: v[k][i] becomes the sum of sequence k before slot i.  The
// totals go to total[k].
template <int N, int ITEMS>
__device__ void block_exclusive_scan(int (&v)[N][ITEMS], int (*s_warp)[32], int* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    int local[N], inc[N];
#pragma unroll
    for (int k = 0; k < N; k++) {
        local[k] = 0;
#pragma unroll
        for (int i = 0; i < ITEMS; i++) { int t = v[k][i]; v[k][i] = local[k]; local[k] += t; }
        inc[k] = local[k];
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
#pragma unroll
        for (int k = 0; k < N; k++) {
            int t = __shfl_up_sync(0xffffffffu, inc[k], o);
            if (lane >= o) inc[k] += t;
        }
    if (lane == 31)
#pragma unroll
        for (int k = 0; k < N; k++) s_warp[k][warp] = inc[k];
    __syncthreads();
    if (warp < N) {   // warp k: sequence k (at least N warps)
        int w = lane < nwarp ? s_warp[warp][lane] : 0, winc = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int t = __shfl_up_sync(0xffffffffu, winc, o);
            if (lane >= o) winc += t;
        }
        if (lane < nwarp) s_warp[warp][lane] = winc - w;
        if (lane == 31) total[warp] = winc;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < N; k++) {
        const int base = s_warp[k][warp] + inc[k] - local[k];
#pragma unroll
        for (int i = 0; i < ITEMS; i++) v[k][i] += base;
    }
}

// One block: bases over blocks and experts, the list of non-empty groups, the
// list of token tiles, counters reset.  Positions: the shared expert's group
// (the tokens, in order) comes first at position 0; every routed group starts
// at a multiple of 8 so that a tile of 8 positions never straddles two groups.
// `s_mask` (shared memory) gives the per-expert counts when one block sorts
// everything; otherwise they are summed from the per-block counts.
// SORT_EPT: experts per thread, 1 where the block has a thread for each (64 threads with four
// experts each wrote the lists one store after the other: 1.5 us more), else 4 (n_expert <= 1024).
template <int SORT_EPT>
__device__ void sort_scan(const Workspace& ws, int n_expert, int nblk, int n, int k,
                          int has_shared, const BigGroups& big_rule, int ptile, int dtile, const uint32_t* s_mask, int* s_off) {
    int prefill_min = big_rule.min;
    __shared__ int s_warp[4][32];
    __shared__ int s_total[4], s_again;
    int cnt[SORT_EPT], seq[4][SORT_EPT];   // positions, groups, tiles, tcgen05 tiles
    int (&off)[SORT_EPT] = seq[0], (&act)[SORT_EPT] = seq[1], (&til)[SORT_EPT] = seq[2], (&ptl)[SORT_EPT] = seq[3];
    int again = 0;
    if (threadIdx.x == 0) s_again = 0;
    __syncthreads();
    const int e0 = threadIdx.x * SORT_EPT;
#pragma unroll
    for (int i = 0; i < SORT_EPT; i++) {
        const int e = e0 + i;
        int run = 0;
        if (e < n_expert) {
            if (s_mask) {
                run = sort_count(s_mask, e);
            } else {
                // eight blocks' counts in flight at a time
                for (int b0 = 0; b0 < nblk; b0 += 8) {
                    int c[8];
#pragma unroll
                    for (int b = 0; b < 8; b++) c[b] = b0 + b < nblk ? ws.blk_counts[(size_t)(b0 + b) * n_expert + e] : 0;
#pragma unroll
                    for (int b = 0; b < 8; b++) {
                        if (b0 + b < nblk) ws.blk_counts[(size_t)(b0 + b) * n_expert + e] = run;
                        run += c[b];
                    }
                }
            }
        }
        cnt[i] = run;
        if (prefill_min > 0 && run >= prefill_min) again += (run - 1) / dtile;
    }
    if (again) atomicAdd(&s_again, again);
    __syncthreads();
    // the tcgen05 kernels are given work only when the groups large enough for them would have
    // the small groups' kernels read enough of their weights again (every tile but a group's first)
    if (prefill_min > 0 && s_again * big_rule.tile_bytes +
                                   (has_shared && n >= prefill_min ? (n - 1) / dtile * big_rule.sh_tile_bytes : 0) <
                               big_rule.worth)
        prefill_min = 0;
#pragma unroll
    for (int i = 0; i < SORT_EPT; i++) {
        // a group of at least prefill_min tokens is cut into tiles of `ptile` for the
        // tcgen05 kernels, a smaller one into tiles of `dtile` for the small groups' kernels
        const int run = cnt[i];
        const bool big = prefill_min > 0 && run >= prefill_min;
        off[i] = (run + SORT_TILE - 1) / SORT_TILE * SORT_TILE;
        til[i] = big ? 0 : (run + dtile - 1) / dtile;
        ptl[i] = big ? (run + ptile - 1) / ptile : 0;
        act[i] = run > 0;
    }
    block_exclusive_scan(seq, s_warp, s_total);
    const int g_sh = has_shared ? 1 : 0;
    const bool big_sh = has_shared && prefill_min > 0 && n >= prefill_min;
    const int p_sh = has_shared ? (n + SORT_TILE - 1) / SORT_TILE * SORT_TILE : 0;
    const int t_sh = has_shared && !big_sh ? (n + dtile - 1) / dtile : 0;
    const int pt_sh = big_sh ? (n + ptile - 1) / ptile : 0;
#pragma unroll
    for (int i = 0; i < SORT_EPT; i++) {
        const int e = e0 + i;
        if (e >= n_expert) continue;
        const int start = p_sh + off[i];
        ws.counts[e] = cnt[i];
        ws.offsets[e] = start;
        if (s_off) s_off[e] = start;
        if (cnt[i]) {
            const int g = g_sh + act[i];
            ws.grp_expert[g] = e;
            ws.grp_start[g] = start;
            ws.grp_count[g] = cnt[i];
            const bool big = prefill_min > 0 && cnt[i] >= prefill_min;
            const int nt = big ? 0 : (cnt[i] + dtile - 1) / dtile;
            for (int j = 0; j < nt; j++) {
                ws.tile_desc[t_sh + til[i] + j] =
                    make_int4(e, start + j * dtile, min(dtile, cnt[i] - j * dtile), 0);
            }
            const int npt = big ? (cnt[i] + ptile - 1) / ptile : 0;
            for (int j = 0; j < npt; j++) {
                ws.ptile_group[pt_sh + ptl[i] + j] = g;
                ws.ptile_t0[pt_sh + ptl[i] + j] = j * ptile;
            }
        }
    }
    for (int j = threadIdx.x; j < t_sh; j += blockDim.x) {
        ws.tile_desc[j] = make_int4(n_expert, j * dtile, min(dtile, n - j * dtile), 0);
    }
    for (int j = threadIdx.x; j < pt_sh; j += blockDim.x) {
        ws.ptile_group[j] = 0;
        ws.ptile_t0[j] = j * ptile;
    }
    if (threadIdx.x == 0) {
        if (has_shared) {
            ws.grp_expert[0] = n_expert;
            ws.grp_start[0] = 0;
            ws.grp_count[0] = n;
        }
        ws.offsets[n_expert] = p_sh + s_total[0];
        *ws.big_min = prefill_min;
        *ws.n_groups = g_sh + s_total[1];
        ws.n_tiles[0] = t_sh + s_total[2];
        ws.n_tiles[1] = t_sh;
        ws.n_ptiles[0] = pt_sh + s_total[3];
        ws.n_ptiles[1] = pt_sh;
    }
    __syncthreads();
}
__device__ void sort_scatter(const Workspace& ws, const uint16_t* s_ids, const uint32_t* s_mask,
                             int pair0, int npairs, int k, int n_expert, int blk, const int* s_off) {
    for (int i = threadIdx.x; i < npairs; i += blockDim.x) {
        const int e = s_ids[i], t = i / k;
        if (e == kNoExpert) {
            ws.pos_of[pair0 + i] = -1;
            continue;
        }
        const uint32_t* m = s_mask + e * SORT_WORDS;
        int rank = __popc(m[t >> 5] & ((1u << (t & 31)) - 1u));
        for (int w = 0; w < (t >> 5); w++) rank += __popc(m[w]);
        const int pos = (s_off ? s_off[e] : ws.offsets[e] + ws.blk_counts[(size_t)blk * n_expert + e]) + rank;
        ws.order[pos] = pair0 + i;
        ws.pos_of[pair0 + i] = pos;
    }
}

enum { SORT_ALL, SORT_HIST, SORT_SCAN, SORT_SCATTER };   // phases of a launch

__global__ void __launch_bounds__(SORT_MANY)
sort_kernel(Workspace ws, int n, int k, int n_expert, int has_shared, BigGroups big, int ptile,
            int dtile, int phase) {
    pdl_enter();
    extern __shared__ __align__(16) uint8_t sort_smem[];
    uint32_t* s_mask = (uint32_t*)sort_smem;                       // [n_expert][SORT_WORDS]
    int* s_off = (int*)(s_mask + (size_t)n_expert * SORT_WORDS);   // [n_expert]
    uint16_t* s_ids = (uint16_t*)(s_off + n_expert);
    const int nblk = (n + SORT_TOKENS - 1) / SORT_TOKENS;
    const int blk = blockIdx.x;
    const int tok0 = blk * SORT_TOKENS, ntok = min(SORT_TOKENS, n - tok0);
    const int pair0 = tok0 * k, npairs = ntok * k;
    if (phase != SORT_SCAN) sort_build_masks([&](int i) { return ws.ids[pair0 + i]; }, npairs, k, n_expert, s_ids, s_mask);
    auto scan = [&](const uint32_t* mask, int* off) {
        if (n_expert <= (int)blockDim.x) sort_scan<1>(ws, n_expert, nblk, n, k, has_shared, big, ptile, dtile, mask, off);
        else sort_scan<4>(ws, n_expert, nblk, n, k, has_shared, big, ptile, dtile, mask, off);
    };
    if (phase == SORT_ALL) {   // one block does everything, bases stay in shared memory
        scan(s_mask, s_off);
        sort_scatter(ws, s_ids, s_mask, pair0, npairs, k, n_expert, 0, s_off);
        return;
    }
    if (phase == SORT_HIST)
        for (int e = threadIdx.x; e < n_expert; e += blockDim.x) ws.blk_counts[(size_t)blk * n_expert + e] = sort_count(s_mask, e);
    if (phase == SORT_SCAN) scan(nullptr, nullptr);
    if (phase == SORT_SCATTER) sort_scatter(ws, s_ids, s_mask, pair0, npairs, k, n_expert, blk, nullptr);
}

// Top-k and sort of a few tokens in one block, a warp per token and then as sort_kernel's
// phase 0: at these sizes both are chains of latencies, and the second launch and the way of
// the ids through memory a third of them (one token 11.9 -> 7.6 us; from 16 tokens on one SM's warps get in each
// other's way: 16 us for 33, against 3.4 + 7.1).
constexpr int TS_MAX_TOKENS = 8, TS_MAX_EXPERTS = 256;
__global__ void __launch_bounds__(TS_MAX_EXPERTS, 1)
topk_sort_kernel(Workspace ws, int n, int k, int n_expert, int has_shared, BigGroups big, int ptile,
                 int dtile) {
    pdl_enter();
    extern __shared__ __align__(16) uint8_t sort_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, ne4 = (n_expert + 3) & ~3;
    float* s_p = (float*)sort_smem;                                   // [warps][ne4]
    uint32_t* s_mask = (uint32_t*)(s_p + (size_t)(blockDim.x >> 5) * ne4);   // [ne4][SORT_WORDS]
    int* s_off = (int*)(s_mask + ne4 * SORT_WORDS);                   // [ne4]
    uint16_t *s_ids = (uint16_t*)(s_off + ne4), *s_sel = s_ids + TS_MAX_TOKENS * TK_MAX_K;
    for (int t = warp; t < n; t += blockDim.x >> 5) {
        int id;
        float w;
        topk_token<TS_MAX_EXPERTS / 32>(ws.logits + (size_t)t * (n_expert + 1), s_p + (size_t)warp * ne4, n_expert, k,
                                        lane, id, w);
        if (lane < k) {
            ws.ids[(size_t)t * k + lane] = id;
            ws.weights[(size_t)t * k + lane] = w;
            s_sel[t * k + lane] = (uint16_t)id;
        }
        __syncwarp();
    }
    __syncthreads();
    sort_build_masks([&](int i) { return (int)s_sel[i]; }, n * k, k, n_expert, s_ids, s_mask);
    sort_scan<1>(ws, n_expert, 1, n, k, has_shared, big, ptile, dtile, s_mask, s_off);
    sort_scatter(ws, s_ids, s_mask, 0, n * k, k, n_expert, 0, s_off);
}

bool topk_and_sort_fuse(int n, int n_expert) { return n <= TS_MAX_TOKENS && n_expert <= TS_MAX_EXPERTS; }

cudaError_t launch_topk_sort(const LaunchCfg& c, const Workspace& ws) {
    if (c.k > TK_MAX_K || !topk_and_sort_fuse(c.n, c.n_expert)) return cudaErrorInvalidValue;
    constexpr int warps = TS_MAX_EXPERTS / 32;   // a thread per expert in the scan
    const size_t ne4 = (c.n_expert + 3) & ~3;
    const size_t smem = warps * ne4 * 4 + ne4 * (SORT_WORDS + 1) * 4 + 2 * TS_MAX_TOKENS * TK_MAX_K * 2;
    static_assert(warps * TS_MAX_EXPERTS * 4 + TS_MAX_EXPERTS * 36 + TS_MAX_TOKENS * TK_MAX_K * 4 <= 48 * 1024, "without raising the limit");
    count_launch();
    return launch_early(c.n, c.stream, topk_sort_kernel, dim3(1), dim3(32 * warps), smem, ws, c.n, c.k, c.n_expert,
                        c.has_shared, c.big, c.prefill_tile, c.tile_rows);
}

// The lists of a pass whose rows are all in one group, at position = token: what sort_kernel
// writes for that group.
__device__ void one_group_lists(const Workspace& ws, int n, int expert, bool shared, int prefill_min, int ptile,
                                int dtile) {
    const bool big = prefill_min > 0 && n >= prefill_min;
    const int nt = big ? 0 : (n + dtile - 1) / dtile, npt = big ? (n + ptile - 1) / ptile : 0;
    for (int j = threadIdx.x; j < nt; j += blockDim.x)
        ws.tile_desc[j] = make_int4(expert, j * dtile, min(dtile, n - j * dtile), 0);
    for (int j = threadIdx.x; j < npt; j += blockDim.x) {
        ws.ptile_group[j] = 0;
        ws.ptile_t0[j] = j * ptile;
    }
    if (threadIdx.x == 0) {
        ws.grp_expert[0] = expert;
        ws.grp_start[0] = 0;
        ws.grp_count[0] = n;
        ws.offsets[expert] = shared ? (n + SORT_TILE - 1) / SORT_TILE * SORT_TILE : 0;
        *ws.n_groups = 1;
        *ws.big_min = prefill_min;
        ws.n_tiles[0] = nt;
        ws.n_tiles[1] = shared ? nt : 0;
        ws.n_ptiles[0] = npt;
        ws.n_ptiles[1] = shared ? npt : 0;
    }
}

// The shared expert's group alone, for a rank of an expert-parallel layer, whose routed
// pairs are sorted where their experts live.
__global__ void __launch_bounds__(SORT_THREADS)
shared_lists_kernel(Workspace ws, int n, int n_expert, int prefill_min, int ptile, int dtile) {
    pdl_enter();
    one_group_lists(ws, n, n_expert, true, prefill_min, ptile, dtile);
}

// Routing of a dense layer: one expert behind a router of zeros.  The logit of a row is the
// sum of 0 * h[i], 0 unless the row holds a NaN or an infinity, then NaN; a softmax over one
// logit is 1 (NaN); the sort's result is the identity.  Bound by reading the rows once (one
// token of 4096: 3 us, where the router product, the top-k and the sort took 37).  The rows of a
// quantised layer are laid out on the way (dispatch_q8_kernel does it for the others): their positions
// are the tokens, and a launch of its own took 2 us more (one token, 4096 / 12288 Q4_K, 36.8 -> 34.8 us a pass).
constexpr int DR_THREADS = 256;
template <bool QUANT>
__global__ void __launch_bounds__(DR_THREADS)
route_dense_kernel(const float* __restrict__ h, Workspace ws, int n, int e, int prefill_min, int ptile, int dtile, int half) {
    pdl_enter();
    const int t = blockIdx.x;
    float s = 0.0f;
    for (int i = threadIdx.x * 8; i < e; i += DR_THREADS * 8) {   // e % 256 == 0: whole warps
        const float4 a = *(const float4*)(h + (size_t)t * e + i), b = *(const float4*)(h + (size_t)t * e + i + 4);
        const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
        for (int j = 0; j < 8; j++) s += 0.0f * v[j];
        if (QUANT) put_q8_unit(ws.act_t, ws.act_rows, t, i, threadIdx.x & 31, half != 0, q8_unit(v, threadIdx.x & 31, half != 0));
    }
    const int bad = __syncthreads_or(isnan(s));
    if (threadIdx.x == 0) {
        const float nan = __int_as_float(0x7fffffff);
        ws.logits[2 * (size_t)t] = ws.logits[2 * (size_t)t + 1] = bad ? nan : 0.0f;
        ws.ids[t] = 0;
        ws.weights[t] = bad ? nan : 1.0f;
        ws.order[t] = ws.pos_of[t] = t;
    }
    if (t == 0) {
        one_group_lists(ws, n, 0, false, prefill_min, ptile, dtile);
        if (threadIdx.x == 0) {
            ws.counts[0] = n;
            ws.offsets[1] = (n + SORT_TILE - 1) / SORT_TILE * SORT_TILE;
        }
    }
}

cudaError_t launch_route_dense(const LaunchCfg& c, const float* h, const Workspace& ws) {
    if (c.n_expert != 1 || c.k != 1 || c.has_shared || c.e % 256) return cudaErrorInvalidValue;
    count_launch();
    return launch_after(c.stream, ws.act_t ? route_dense_kernel<true> : route_dense_kernel<false>, dim3(c.n), dim3(DR_THREADS), 0,
                        h, ws, c.n, c.e, c.big.min, c.prefill_tile, c.tile_rows, c.wide ? 1 : 0);
}

cudaError_t launch_shared_lists(const LaunchCfg& c, const Workspace& ws) {
    count_launch();
    return launch_after(c.stream, shared_lists_kernel, dim3(1), dim3(SORT_THREADS), 0, ws, c.n, c.n_expert,
                        c.big.min, c.prefill_tile, c.tile_rows);
}

cudaError_t launch_sort(const LaunchCfg& c, const Workspace& ws) {
    const int nblk = (c.n + SORT_TOKENS - 1) / SORT_TOKENS;
    const size_t smem = (size_t)c.n_expert * (SORT_WORDS + 1) * 4 + (size_t)SORT_TOKENS * c.k * 2;   // <= 36 + 16 KiB
    static std::atomic<uint64_t> attr_set{0};
    if (cudaError_t err = ensure_dynamic_smem(sort_kernel, 64 * 1024, attr_set)) return err;
    auto phase = [&](int blocks, int ph) {
        const int threads = ph != SORT_SCAN && min(c.n, SORT_TOKENS) * c.k > SORT_THREADS ? SORT_MANY : SORT_THREADS;
        return launch_early(c.n, c.stream, sort_kernel, dim3(blocks), dim3(threads), smem, ws, c.n, c.k, c.n_expert,
                            c.has_shared, c.big, c.prefill_tile, c.tile_rows, ph);
    };
    if (nblk == 1) {
        count_launch();
        return phase(1, SORT_ALL);
    }
    count_launch(3);
    if (cudaError_t err = phase(nblk, SORT_HIST)) return err;
    if (cudaError_t err = phase(1, SORT_SCAN)) return err;
    return phase(nblk, SORT_SCATTER);
}

}  // namespace bivmoe
