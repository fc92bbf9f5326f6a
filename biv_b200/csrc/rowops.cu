// Row-wise helpers around the expert products: the Q8 activation quantiser,
// rms_norm, the weighted gather-combine, and the upload-time repack of GGUF
// rows into the device row layout.
#include <cuda_bf16.h>

#include "common.cuh"
#include "formats.cuh"
#include "launch.cuh"

namespace bivmoe {

// ---------------------------------------------------------------------------
// Dispatch: the rows the expert kernels consume, laid out by position
// (slice-major, see common.cuh).  Token t's row goes to position t (the
// shared expert's group) and to the position of each of its k pairs.  For
// quantised weight types the row is quantised once, Q8Act::quantize_into
// (quant.rs:368-394) - the reference quantises it again for every expert it is
// routed to (model.rs:876-884), with the same result, the quantiser being a
// function of the row alone.  One block per token.
constexpr int DP_THREADS = 256, DP_MAX_K = 32;

// s_pos[j]: the position of pair j (j < k) and, as entry k, the token's position in the
// shared expert's group; s_big[j]: whether that position's group is large enough for
// the tcgen05 kernels.  Without a shared expert entry k repeats the first pair.
__device__ __forceinline__ void dispatch_positions(const Workspace& ws, int t, int n, int k, int has_shared,
                                                   bool skip_big, int* s_pos,
                                                   int* s_big) {
    const int prefill_min = skip_big ? *ws.big_min : 0;
    if (threadIdx.x < k) {   // a negative position: an empty slot, nothing is written for it
        const int id = ws.ids[(size_t)t * k + threadIdx.x];
        s_pos[threadIdx.x] = id < 0 ? -1 : ws.pos_of[(size_t)t * k + threadIdx.x];
        s_big[threadIdx.x] = id >= 0 && prefill_min > 0 && ws.counts[id] >= prefill_min;
    }
    if (threadIdx.x == k) {
        s_pos[k] = has_shared ? t : -1;
        s_big[k] = has_shared && prefill_min > 0 && n >= prefill_min;
    }
}

__global__ void __launch_bounds__(DP_THREADS)
dispatch_q8_kernel(const float* __restrict__ h, Workspace ws, int n, int k, int e, int has_shared,
                   const float* __restrict__ norm_w, int half) {
    __shared__ int s_pos[DP_MAX_K + 1], s_big[DP_MAX_K + 1];
    pdl_enter();
    const int t = blockIdx.x, lane = threadIdx.x & 31;
    const int R = ws.act_rows;
    const float* x = h + (size_t)t * e;
    // with norm_w the rows are the residual and h = x * (scale * w), rms_norm on the fly
    const float nscale = norm_w ? ws.row_scale[t] : 1.0f;
    Q8Unit u;
    auto quantize = [&](int i0) {                     // e % 256 == 0: whole warps
        float4 a = *(const float4*)(x + i0), b = *(const float4*)(x + i0 + 4);
        if (norm_w) {
            const float4 wa = *(const float4*)(norm_w + i0), wb = *(const float4*)(norm_w + i0 + 4);
            a.x = __fmul_rn(a.x, __fmul_rn(nscale, wa.x)); a.y = __fmul_rn(a.y, __fmul_rn(nscale, wa.y));
            a.z = __fmul_rn(a.z, __fmul_rn(nscale, wa.z)); a.w = __fmul_rn(a.w, __fmul_rn(nscale, wa.w));
            b.x = __fmul_rn(b.x, __fmul_rn(nscale, wb.x)); b.y = __fmul_rn(b.y, __fmul_rn(nscale, wb.y));
            b.z = __fmul_rn(b.z, __fmul_rn(nscale, wb.z)); b.w = __fmul_rn(b.w, __fmul_rn(nscale, wb.w));
        }
        const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        u = q8_unit(v, lane, half != 0);
    };
    auto store = [&](int i0) {
        for (int j = 0; j <= k; j++)
            if (s_pos[j] >= 0) put_q8_unit(ws.act_t, R, s_pos[j], i0, lane, half != 0, u);
    };
    // the first values are read and quantised while the positions are on their way
    dispatch_positions(ws, t, n, k, has_shared, false, s_pos, s_big);
    const int first = threadIdx.x * 8;
    if (first < e) quantize(first);
    __syncthreads();
    if (first < e) store(first);
    for (int i0 = first + DP_THREADS * 8; i0 < e; i0 += DP_THREADS * 8) {
        quantize(i0);
        store(i0);
    }
}

// Quantised rows for many tokens, in two steps: each row is quantised once into a row of its
// own, [token][e] int8 and [token][e / 32] (d, s), and the records are then written a tile of
// 8 positions at a time, whole and in order.  (The kernel above writes 16 bytes here and there
// in the records of k + 1 positions; what L2 then merges half-written sectors from took 85 us
// for 4096 tokens of 8 experts, 126 MB; the two steps 7 + 29.)
constexpr int DQ_MIN_TOKENS = 256;   // from here on, if a row has more than one position (300 dense rows: 4.2 us in one step, 6.9 in two)
__global__ void __launch_bounds__(DP_THREADS)
quant_rows_kernel(const float* __restrict__ h, int8_t* __restrict__ tok_q, float2* __restrict__ tok_s, int e) {
    pdl_enter();
    const int t = blockIdx.x;
    quantize_row(h + (size_t)t * e, tok_q + (size_t)t * e, tok_s + (size_t)t * e / 32, e);
}

// 128 (HALF, the f16 records: 256) 16-byte units of q and 64 block scales of a record
template <bool HALF> constexpr int GQ_THREADS = HALF ? 320 : 192;
template <bool HALF>
__global__ void __launch_bounds__(GQ_THREADS<HALF>)
gather_q8_kernel(const int8_t* __restrict__ tok_q, const float2* __restrict__ tok_s, Workspace ws, int n, int k, int e,
                 int n_expert, int has_shared) {
    pdl_enter();
    const int R = ws.act_rows, t = threadIdx.x, tk = t & 7;
    const int p_sh = has_shared ? (n + 7) / 8 * 8 : 0;
    const int tiles = ws.offsets[n_expert] / 8;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int pos = tile * 8 + tk;
        // positions past the end of a group hold any row: nothing reads their results
        const int tok = min(max(pos < p_sh ? pos : ws.order[pos] / k, 0), n - 1);
        constexpr int REC = HALF ? kHalfRec : kActTileBytes, QT = GQ_THREADS<HALF> - 64;
        uint8_t* rec = ws.act_t + (size_t)tile * REC;
        const size_t step = (size_t)(R / 8) * REC;
        if (HALF && t < QT) {
            const uint2* src = (const uint2*)(tok_q + (size_t)tok * e + (t >> 3) * 8);
            uint8_t* dst = rec + t * 16;
#pragma unroll 4
            for (int sl = 0; sl < e / 256; sl++) {
                const uint2 w = src[sl * 32];
                *(uint4*)(dst + sl * step) = half_unit(w.x, w.y);
            }
        } else if (t < QT) {
            const uint4* src = (const uint4*)(tok_q + (size_t)tok * e + (t >> 3) * 16);
            uint4* dst = (uint4*)(rec + t * 16);
#pragma unroll 4
            for (int sl = 0; sl < e / 256; sl++) *(uint4*)((uint8_t*)dst + sl * step) = src[sl * 16];
        } else {
            const int b = (t - QT) >> 3;
            const float2* src = tok_s + (size_t)tok * (e / 32) + b;
#pragma unroll 4
            for (int sl = 0; sl < e / 256; sl++) {
                const float2 ds = src[sl * 8];
                float shi, slo;
                split_tf32(ds.y, &shi, &slo);
                uint8_t* at = rec + sl * step;
                const float val[4] = {ds.x, shi, slo, ds.y};
#pragma unroll
                for (int i = 0; i < 4; i++) *(float*)(at + (HALF ? half_scale_off(i, b, tk) : act_scale_off(i, b, tk))) = val[i];
            }
        }
    }
}

// The three bf16 terms of 8 consecutive values into a three-term record (`at`: of the values'
// unit and token).
__device__ __forceinline__ void store_terms(uint8_t* at, const float4& a, const float4& b) {
    const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    uint16_t t[8][3];
#pragma unroll
    for (int i = 0; i < 8; i++) split_bf16_3(v[i], t[i]);
#pragma unroll
    for (int i = 0; i < 3; i++)
        *(uint4*)(at + i * kAct3Term) = make_uint4(t[0][i] | (uint32_t)t[1][i] << 16, t[2][i] | (uint32_t)t[3][i] << 16,
                                                   t[4][i] | (uint32_t)t[5][i] << 16, t[6][i] | (uint32_t)t[7][i] << 16);
}

// Float rows.  A thread owns 8 consecutive values: two float4 stores per position of a
// decode-sized group (slice-major f32 rows), or three 16-byte ones (three-term records).  Positions of groups the
// tcgen05 kernel takes get nothing: that kernel gathers its rows by token from the
// bf16 terms split_rows_kernel writes.
__global__ void __launch_bounds__(DP_THREADS)
dispatch_f32_kernel(const float* __restrict__ h, Workspace ws, int n, int k, int e, int has_shared,
                    const float* __restrict__ norm_w) {
    __shared__ int s_pos[DP_MAX_K + 1], s_big[DP_MAX_K + 1];
    pdl_enter();
    const int t = blockIdx.x;
    const int R = ws.act_rows;
    dispatch_positions(ws, t, n, k, has_shared, ws.tok_b != nullptr, s_pos, s_big);
    __syncthreads();
    const float* x = h + (size_t)t * e;
    const float nscale = norm_w ? ws.row_scale[t] : 1.0f;
    for (int i0 = threadIdx.x * 8; i0 < e; i0 += DP_THREADS * 8) {
        float4 a = *(const float4*)(x + i0), b = *(const float4*)(x + i0 + 4);
        if (norm_w) {   // rms_norm on the fly: h = x * (scale * w)
            const float4 wa = *(const float4*)(norm_w + i0), wb = *(const float4*)(norm_w + i0 + 4);
            a.x = __fmul_rn(a.x, __fmul_rn(nscale, wa.x)); a.y = __fmul_rn(a.y, __fmul_rn(nscale, wa.y));
            a.z = __fmul_rn(a.z, __fmul_rn(nscale, wa.z)); a.w = __fmul_rn(a.w, __fmul_rn(nscale, wa.w));
            b.x = __fmul_rn(b.x, __fmul_rn(nscale, wb.x)); b.y = __fmul_rn(b.y, __fmul_rn(nscale, wb.y));
            b.z = __fmul_rn(b.z, __fmul_rn(nscale, wb.z)); b.w = __fmul_rn(b.w, __fmul_rn(nscale, wb.w));
        }
        const int sl = i0 / 64, off = i0 % 64;
        for (int j = 0; j <= k; j++) {
            const int pos = s_pos[j];
            if (pos < 0 || s_big[j]) continue;
            if (ws.act_3) {
                store_terms(ws.act_3 + ((size_t)sl * (R / 8) + pos / 8) * kAct3Rec + act_b_off(pos % 8, off), a, b);
                continue;
            }
            float* dst = ws.act_f + ((size_t)sl * R + pos) * 64 + off;
            *(float4*)dst = a;
            *(float4*)(dst + 4) = b;
        }
    }
}

// The rows as two bf16 terms, x = hi + lo, by token: [token][K / 64][hi 64 | lo 64], 256
// bytes per token and K-slice.  The tcgen05 kernel gathers a tile's rows from here in
// 16-byte units (experts_prefill_bf16.cu), so a row is split once, not once per position
// it occupies.  A row no group wants (an expert-parallel receive slot that is empty) is
// skipped.
__global__ void __launch_bounds__(DP_THREADS)
split_rows_kernel(const float* __restrict__ h, Workspace ws, int n, int k, int e, int has_shared,
                  const float* __restrict__ norm_w) {
    pdl_enter();
    const int t = blockIdx.x;
    if (!has_shared) {
        bool any = false;
        for (int j = 0; j < k; j++) any |= ws.ids[(size_t)t * k + j] >= 0;
        if (!any) return;
    }
    split_row(h + (size_t)t * e, ws.tok_b + (size_t)t * (e / 64) * kTokBRec, e, norm_w, norm_w ? ws.row_scale[t] : 1.0f);
}

// Float rows by position, for many tokens: a block per tile of 8 positions of a
// decode-sized group, taken from the sort's tile list (groups the tcgen05 kernel takes
// have no tiles there).  It reads the tile's 8 source rows and writes them slice-major.
// (For quantised rows the same arrangement measured slower than the by-token kernel:
// it quantises a row once per position.)
constexpr int DP_MIN_TOKENS = 256;   // from here on the by-position kernel is the faster one

__global__ void __launch_bounds__(DP_THREADS)
dispatch_pos_f32_kernel(const float* __restrict__ h, Workspace ws, int k, int e, int n_expert,
                        int only_shared) {
    pdl_enter();
    const int n_tiles = ws.n_tiles[only_shared ? 1 : 0];   // the shared group's tiles come first
    // thread (tk, u): 8 consecutive values of token tk
    const int tk = threadIdx.x & 7, u0 = threadIdx.x >> 3;
    const int R = ws.act_rows;
    for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
        const int4 td = ws.tile_desc[tile];   // {expert (n_expert: shared), first position, tokens, 0}
        if (tk >= td.z) continue;
        const int pos = td.y + tk;
        const int tok = td.x == n_expert ? pos : ws.order[pos] / k;
        const float* x = h + (size_t)tok * e;
        for (int i0 = u0 * 8; i0 < e; i0 += (DP_THREADS / 8) * 8) {
            const float4 a = *(const float4*)(x + i0), b = *(const float4*)(x + i0 + 4);
            const int sl = i0 / 64, off = i0 % 64;
            if (ws.act_3) {
                store_terms(ws.act_3 + ((size_t)sl * (R / 8) + pos / 8) * kAct3Rec + act_b_off(pos % 8, off), a, b);
                continue;
            }
            float* dst = ws.act_f + ((size_t)sl * R + pos) * 64 + off;
            *(float4*)dst = a;
            *(float4*)(dst + 4) = b;
        }
    }
}

// whether the products' rows come from rows by token, quantised or split, which the top-k's launch can make
static bool quantised_by_token(const LaunchCfg& c, const Workspace& ws, bool quant) {
    return quant && ws.tok_q && c.n >= DQ_MIN_TOKENS && c.k + c.has_shared > 1;
}
static bool split_by_token(const LaunchCfg& c, const Workspace& ws, bool f32) { return f32 && ws.tok_b && c.big.min > 0; }

RowsReady rows_with_topk(const LaunchCfg& c, const Workspace& ws, bool quant, bool f32) {
    if (c.n < DQ_MIN_TOKENS || c.e % 256) return ROWS_NONE;
    return quantised_by_token(c, ws, quant) ? ROWS_QUANT : split_by_token(c, ws, f32) ? ROWS_SPLIT : ROWS_NONE;
}

cudaError_t launch_dispatch(const LaunchCfg& c, const float* h, const Workspace& ws, bool quant,
                            bool f32, const RowNorm* norm) {
    if (c.k > DP_MAX_K || c.e % 256) return cudaErrorInvalidValue;
    if (norm && c.n >= DP_MIN_TOKENS) return cudaErrorInvalidValue;   // the by-position kernel reads normed rows
    const float* nw = norm ? norm->w : nullptr;
    if (quantised_by_token(c, ws, quant)) {
        if (c.rows_ready != ROWS_QUANT) {
            if (cudaError_t err = launch_early(c.n, c.stream, quant_rows_kernel, dim3(c.n), dim3(DP_THREADS), 0, h, ws.tok_q,
                                               ws.tok_s, c.e))
                return err;
            count_launch();
        }
        const int tiles = (c.n + 7) / 8 * c.has_shared + c.n * c.k / 8 + c.n_expert;
        if (cudaError_t err = launch_early(c.n, c.stream, c.wide ? gather_q8_kernel<true> : gather_q8_kernel<false>,
                                           dim3(min(tiles, 32 * c.sm_count)), dim3(c.wide ? GQ_THREADS<true> : GQ_THREADS<false>), 0,
                                           (const int8_t*)ws.tok_q, (const float2*)ws.tok_s, ws, c.n, max(c.k, 1), c.e,
                                           c.n_expert, c.has_shared))
            return err;
        count_launch();
    } else if (quant) {
        if (cudaError_t err = launch_early(c.n, c.stream, dispatch_q8_kernel, dim3(c.n), dim3(DP_THREADS), 0, h, ws,
                                           c.n, c.k, c.e, c.has_shared, nw, c.wide ? 1 : 0))
            return err;
        count_launch();
    }
    if (split_by_token(c, ws, f32) && c.rows_ready != ROWS_SPLIT) {
        if (cudaError_t err = launch_early(c.n, c.stream, split_rows_kernel, dim3(c.n), dim3(DP_THREADS), 0, h, ws, c.n,
                                           c.k, c.e, c.has_shared, nw))
            return err;
        count_launch();
    }
    if (f32 && c.n >= DP_MIN_TOKENS) {
        // the tiles in use are known on the device only: blocks stride over the list
        const int shared_tiles = c.has_shared ? (c.n + 7) / 8 : 0;
        const int tiles = c.k == 0 ? shared_tiles : shared_tiles + (c.n * c.k) / 8 + c.n_expert;
        if (cudaError_t err = launch_early(c.n, c.stream, dispatch_pos_f32_kernel, dim3(min(tiles, 16 * c.sm_count)),
                                           dim3(DP_THREADS), 0, h, ws, max(c.k, 1), c.e, c.n_expert,
                                           c.only_shared || c.k == 0 ? 1 : 0))
            return err;
        count_launch();
    } else if (f32) {
        if (cudaError_t err = launch_early(c.n, c.stream, dispatch_f32_kernel, dim3(c.n), dim3(DP_THREADS), 0, h, ws, c.n,
                                           c.k, c.e, c.has_shared, nw))
            return err;
        count_launch();
    }
    return cudaGetLastError();
}

__global__ void __launch_bounds__(256)
copy_words_kernel(const uint4* __restrict__ src, uint4* __restrict__ dst, int words) {
    pdl_enter();
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i < words) dst[i] = src[i];
}
cudaError_t launch_copy_words(const LaunchCfg& c, const void* src, void* dst, size_t bytes) {
    const int words = (int)(bytes / 16);
    count_launch();
    return launch_after(c.stream, copy_words_kernel, dim3((words + 255) / 256), dim3(256), 0, (const uint4*)src,
                        (uint4*)dst, words);
}

// ---------------------------------------------------------------------------
// ops.rs:136-149: out = x * (1/sqrt(dot(x,x)/e + eps)) * w, one warp per row.
// The sum of squares uses the reference's AVX2 dot order (see router.cu).
template <class At>
__device__ __forceinline__ float rms_scale(At x, int e, float eps, int lane) {   // of the row x(0) .. x(e - 1), by a warp
    float acc = 0.0f;
    for (int i0 = lane; i0 < e; i0 += 32 * 32) {   // 32 loads in flight (e % 256 == 0)
        float v[32];
#pragma unroll
        for (int j = 0; j < 32; j++) v[j] = i0 + 32 * j < e ? x(i0 + 32 * j) : 0.0f;
#pragma unroll
        for (int j = 0; j < 32; j++)
            if (i0 + 32 * j < e) acc = fmaf(v[j], v[j], acc);
    }
    acc = __fadd_rn(acc, __shfl_xor_sync(0xffffffffu, acc, 8));
    acc = __fadd_rn(acc, __shfl_xor_sync(0xffffffffu, acc, 16));
    acc = __fadd_rn(acc, __shfl_xor_sync(0xffffffffu, acc, 4));
    acc = __fadd_rn(acc, __shfl_xor_sync(0xffffffffu, acc, 2));
    acc = __fadd_rn(acc, __shfl_xor_sync(0xffffffffu, acc, 1));
    const float ss = __fdiv_rn(acc, (float)e);
    return __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(ss, eps)));
}
__device__ __forceinline__ float4 rms_apply(const float4& x, float scale, const float4& w) {
    return make_float4(__fmul_rn(x.x, __fmul_rn(scale, w.x)), __fmul_rn(x.y, __fmul_rn(scale, w.y)),
                       __fmul_rn(x.z, __fmul_rn(scale, w.z)), __fmul_rn(x.w, __fmul_rn(scale, w.w)));
}
__global__ void __launch_bounds__(128)
rms_norm_kernel(const float* __restrict__ x, const float* __restrict__ w, float eps,
                float* __restrict__ out, int n, int e) {
    pdl_enter();
    const int lane = threadIdx.x & 31;
    const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= n) return;
    const float* xr = x + (size_t)row * e;
    const float scale = rms_scale([&](int i) { return xr[i]; }, e, eps, lane);
    for (int i = lane * 4; i < e; i += 128)
        *(float4*)(out + (size_t)row * e + i) = rms_apply(*(const float4*)(xr + i), scale, *(const float4*)(w + i));
}

cudaError_t launch_rms_norm(const LaunchCfg& c, const float* x, const float* w, float eps,
                            float* out) {
    count_launch();
    return launch_after(c.stream, rms_norm_kernel, dim3((c.n + 1) / 2), dim3(64), 0, x, w, eps, out, c.n, c.e);
}

// ---------------------------------------------------------------------------
// Weighted gather-combine (model.rs:886-896; Metal moe_combine,
// kernels.metal:1885-1908): out[t] (+)= sum over the token's experts in
// ascending expert id of w * y, then sigmoid(gate) * shared, each step one
// fused multiply-add as the reference's axpy.  No atomics: run-to-run identical.
constexpr int CB_THREADS = 256, CBN_THREADS = 512, CB_MAX_K = 32;

// PEER: the rows are an owner rank's receive regions (expert parallelism by peer stores,
// ep.cu); row t = region t / cap, slot t % cap; a slot past the region's count has no row,
// and the sum of a row goes straight into region `me`, same slot, of the return buffer of
// the rank the row came from - the weighted sum and its way home are one kernel.
struct PeerDest {
    PeerTable peers;
    PeerLayout lay;
    const int32_t* counts;
    int me;
};

// WAY: blocks of 256 float4 columns that fit on the chip at once take the time of trips to memory, more are bound by
// bytes and want many on an SM.  us with three blocks an SM and everything asked for at once / four of 56 registers a thread / eight of
// 32: 128 rows of 2048, 8 experts a token 4.4 / 4.7 / 5.1; 256 rows 6.8 / 5.2 / 5.7; 384 rows 7.0 / 6.9 / 6.2; 512 rows
// 9.0 / 7.6 / 7.0; of 4096 columns 64, 128, 192 rows 4.4 / 4.7 / 4.9, 6.3 / 5.3 / 5.4, 6.9 / 6.9 / 6.0; so at 1024
// and 8192 columns and with 2 to 16 experts (rule: launch_combine).
enum { CB_FEW, CB_SOME, CB_MANY };
constexpr int cb_per_sm(int way) { return way == CB_FEW ? 3 : way == CB_SOME ? 4 : 8; }
// NORM: a block has a whole row and leaves it normed for the next layer of a stack, too (rms_norm_kernel's
// arithmetic); by itself that took 4.4 us for 160 rows.
struct NormDest {
    const float* w;
    float eps;
    float* rows;
};

template <bool PEER, int WAY, bool NORM>
__global__ void __launch_bounds__(NORM ? CBN_THREADS : CB_THREADS, NORM ? 2 : cb_per_sm(WAY))
combine_kernel(const int32_t* __restrict__ ids, const float* __restrict__ weights,
               const float* __restrict__ routed_rows, const int32_t* __restrict__ routed_pos,
               const float* __restrict__ shared_rows, const float* __restrict__ logits,
               float* __restrict__ out, int n, int k, int e, int n_expert, int has_shared, int accumulate,
               PeerDest pd, NormDest nd) {
    static_assert(!PEER || (WAY != CB_FEW && !NORM), "those write to out");
    __shared__ int s_pos[CB_MAX_K];
    __shared__ float s_w[CB_MAX_K];
    __shared__ float s_gate;
    __shared__ int s_valid;
    // the norm's weights are long out of the caches
    float4 nw = make_float4(0.f, 0.f, 0.f, 0.f);
    if (NORM && threadIdx.x * 4 < e) nw = *(const float4*)(nd.w + threadIdx.x * 4);
    pdl_enter();
    const int t = blockIdx.x;
    if (PEER && t % pd.lay.cap >= pd.counts[t / pd.lay.cap]) return;   // the whole block
    if (threadIdx.x == 0) s_valid = 0;
    __syncthreads();
    if (threadIdx.x < k) {
        // rank of this pair among the token's pairs by expert id (ids are distinct; a
        // negative id is an empty slot and takes no rank)
        const int my = ids[(size_t)t * k + threadIdx.x];
        if (my >= 0) {
            int rank = 0;
            for (int j = 0; j < k; j++) {
                const int o = ids[(size_t)t * k + j];
                rank += o >= 0 && o < my;
            }
            s_pos[rank] = routed_pos[(size_t)t * k + threadIdx.x];
            s_w[rank] = weights[(size_t)t * k + threadIdx.x];
            atomicAdd(&s_valid, 1);
        }
    }
    if (threadIdx.x == 32 && has_shared) {
        const float g = logits[(size_t)t * (n_expert + 1) + n_expert];
        s_gate = __fdiv_rn(1.0f, __fadd_rn(1.0f, expf(-g)));   // ops.rs:160-162
    }
    __syncthreads();
    const int kv = s_valid;
    extern __shared__ __align__(16) float cb_row[];           // NORM: the row's sums
    auto column = [&](int c4) {                               // of a float4
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        auto add = [&](float w, const float4& y) {
            acc.x = fmaf(w, y.x, acc.x); acc.y = fmaf(w, y.y, acc.y);
            acc.z = fmaf(w, y.z, acc.z); acc.w = fmaf(w, y.w, acc.w);
        };
        float4* o = (float4*)(out + (size_t)t * e + c4 * 4);
        if constexpr (WAY == CB_FEW) {
            // everything that a column needs is asked for at once, eight experts' rows at a time
            float4 old = acc, sh = acc;
            if (accumulate) old = *o;
            if (has_shared) sh = *(const float4*)(shared_rows + (size_t)t * e + c4 * 4);
            for (int j0 = 0; j0 < kv; j0 += 8) {
                float4 y[8];
#pragma unroll
                for (int j = 0; j < 8; j++)
                    if (j0 + j < kv) y[j] = *(const float4*)(routed_rows + (size_t)s_pos[j0 + j] * e + c4 * 4);
#pragma unroll
                for (int j = 0; j < 8; j++)
                    if (j0 + j < kv) add(s_w[j0 + j], y[j]);
            }
            if (has_shared) add(s_gate, sh);
            if (accumulate) {
                acc.x += old.x; acc.y += old.y; acc.z += old.z; acc.w += old.w;
            }
        } else {
            for (int j = 0; j < kv; j++) add(s_w[j], *(const float4*)(routed_rows + (size_t)s_pos[j] * e + c4 * 4));
            if (has_shared) add(s_gate, *(const float4*)(shared_rows + (size_t)t * e + c4 * 4));
            if (PEER)
                o = (float4*)(pd.peers.base[t / pd.lay.cap] + pd.lay.returned) +
                    ((size_t)pd.me * pd.lay.cap + t % pd.lay.cap) * (e / 4) + c4;
            if (accumulate) {
                const float4 old = *o;
                acc.x += old.x; acc.y += old.y; acc.z += old.z; acc.w += old.w;
            }
        }
        *o = acc;
        if (NORM) *(float4*)(cb_row + c4 * 4) = acc;
    };
    if constexpr (!NORM) {
        const int c4 = blockIdx.y * CB_THREADS + threadIdx.x;
        if (c4 * 4 < e) column(c4);
    } else {
        for (int c4 = threadIdx.x; c4 * 4 < e; c4 += CBN_THREADS) column(c4);
        __syncthreads();
        if (threadIdx.x < 32) {
            const float scale = rms_scale([&](int i) { return cb_row[i]; }, e, nd.eps, threadIdx.x);
            if (threadIdx.x == 0) s_gate = scale;
        }
        __syncthreads();
        const float scale = s_gate;
        for (int i = threadIdx.x * 4; i < e; i += blockDim.x * 4)
            *(float4*)(nd.rows + (size_t)t * e + i) =
                rms_apply(*(const float4*)(cb_row + i), scale, i < blockDim.x * 4 ? nw : *(const float4*)(nd.w + i));
    }
}

// a row in shared memory, and the blocks, one a row and two on an SM, on the chip at once
bool combine_norms(int n, int e) { return n < 256 && (size_t)e * 4 <= 40 * 1024; }

cudaError_t launch_combine(const LaunchCfg& c, const CombineSrc& src, float* out, int accumulate, const RowNorm* next,
                           float* next_rows) {
    if (c.k > CB_MAX_K || c.e % 4) return cudaErrorInvalidValue;
    count_launch();
    const bool early = pdl_mode() == 1 || (pdl_mode() != 0 && c.n <= kEarlyCombine);
    if (next)
        return launch_with(early, c.stream, combine_kernel<false, CB_FEW, true>, dim3(c.n), dim3(CBN_THREADS), (size_t)c.e * 4, src.ids,
                           src.weights, src.routed_rows, src.routed_pos, src.shared_rows, src.logits, out, c.n, c.k, c.e,
                           c.n_expert, c.has_shared, accumulate, PeerDest{}, NormDest{next->w, next->eps, next_rows});
    const dim3 grid(c.n, (c.e / 4 + CB_THREADS - 1) / CB_THREADS);
    auto at_once = [&](int way) { return (long long)grid.x * grid.y <= (long long)cb_per_sm(way) * c.sm_count; };
    auto kernel = at_once(CB_FEW) ? combine_kernel<false, CB_FEW, false>
                : at_once(CB_SOME) ? combine_kernel<false, CB_SOME, false> : combine_kernel<false, CB_MANY, false>;
    return launch_with(early, c.stream, kernel, grid, dim3(CB_THREADS), 0, src.ids, src.weights, src.routed_rows, src.routed_pos, src.shared_rows, src.logits,
                       out, c.n, c.k, c.e, c.n_expert, c.has_shared, accumulate, PeerDest{}, NormDest{});
}

// A dense layer's output: out[t] (+)= weight[t] * y[t], the weight 1 or (a row with a NaN or
// an infinity) NaN; with K in parts y[t] is their sum, in order, and is kept as the pair's row.
__global__ void __launch_bounds__(CB_THREADS)
combine_dense_kernel(const float* __restrict__ weights, float* __restrict__ pair_out, const float* __restrict__ sums,
                     float* __restrict__ out, int n, int e, int parts, int accumulate) {
    pdl_enter();
    const int t = blockIdx.x, c4 = blockIdx.y * CB_THREADS + threadIdx.x;
    if (c4 * 4 >= e) return;
    const size_t at = (size_t)t * e + c4 * 4, stride = (size_t)n * e;
    float4 y;
    if (parts > 1) {
        y = *(const float4*)(sums + at);
#pragma unroll 8
        for (int p = 1; p < parts; p++) {
            const float4 v = *(const float4*)(sums + p * stride + at);
            y.x += v.x; y.y += v.y; y.z += v.z; y.w += v.w;
        }
        *(float4*)(pair_out + at) = y;
    } else {
        y = *(const float4*)(pair_out + at);
    }
    const float w = weights[t];
    float4 acc = make_float4(fmaf(w, y.x, 0.0f), fmaf(w, y.y, 0.0f), fmaf(w, y.z, 0.0f), fmaf(w, y.w, 0.0f));
    float4* o = (float4*)(out + at);
    if (accumulate) {
        const float4 r = *o;
        acc.x += r.x; acc.y += r.y; acc.z += r.z; acc.w += r.w;
    }
    *o = acc;
}

cudaError_t launch_combine_dense(const LaunchCfg& c, const Workspace& ws, float* out, int accumulate) {
    if (c.e % 4) return cudaErrorInvalidValue;
    count_launch();
    return launch_with(pdl_mode() == 1 || (pdl_mode() != 0 && c.n <= kEarlyCombine), c.stream, combine_dense_kernel, dim3(c.n, (c.e / 4 + CB_THREADS - 1) / CB_THREADS),
                        dim3(CB_THREADS), 0, (const float*)ws.weights, ws.pair_out, (const float*)ws.parts, out, c.n,
                        c.e, c.down_parts, accumulate);
}

// The SwiGLU rows of a dense layer whose gate+up product came in parts ([part][n][gate ff | up
// ff]): what the product kernels' own tail does, a warp per token and 32-row block.
__global__ void __launch_bounds__(DP_THREADS)
swiglu_parts_kernel(const float* __restrict__ sums, float* __restrict__ mid, uint8_t* __restrict__ mid_t,
                    uint8_t* __restrict__ mid_3, int n, int ff, int parts, int R) {
    pdl_enter();
    const int t = blockIdx.y, lane = threadIdx.x & 31;
    const int r = (blockIdx.x * (DP_THREADS / 32) + (threadIdx.x >> 5)) * 32 + lane;
    if (r >= ff) return;   // ff is a multiple of 64: whole warps
    const size_t stride = (size_t)n * 2 * ff;
    const float* s = sums + (size_t)t * 2 * ff + r;
    float gt = s[0], u = s[ff];
#pragma unroll 4
    for (int p = 1; p < parts; p++) {
        gt += s[p * stride];
        u += s[p * stride + ff];
    }
    // ops.rs:160-167: silu(x) = x * (1 / (1 + exp(-x)))
    const float v = (gt * __fdiv_rn(1.0f, 1.0f + expf(-gt))) * u;
    mid[((size_t)(r / 64) * R + t) * 64 + r % 64] = v;
    if (mid_3) {
        uint16_t term[3];
        split_bf16_3(v, term);
        uint8_t* rec = mid_3 + ((size_t)(r / 64) * (R / 8) + t / 8) * kAct3Rec + act_b_off(t % 8, r % 64);
#pragma unroll
        for (int i = 0; i < 3; i++) *(uint16_t*)(rec + i * kAct3Term) = term[i];
    }
    if (!mid_t) return;
    float dd, ss;
    const int q = q8_quantize_lane(v, dd, ss);
    uint8_t* rec = mid_t + ((size_t)(r / 256) * (R / 8) + t / 8) * kActTileBytes;
    rec[act_q_off(t % 8, r % 256)] = (uint8_t)(int8_t)q;
    if (lane < 4) {
        float shi, slo;
        split_tf32(ss, &shi, &slo);
        const float val = lane == 0 ? dd : lane == 1 ? shi : lane == 2 ? slo : ss;
        *(float*)(rec + act_scale_off(lane, (r % 256) / 32, t % 8)) = val;
    }
}

cudaError_t launch_swiglu_parts(const LaunchCfg& c, const Workspace& ws) {
    count_launch();
    return launch_after(c.stream, swiglu_parts_kernel, dim3((c.ff + DP_THREADS - 1) / DP_THREADS, c.n), dim3(DP_THREADS),
                        0, (const float*)ws.parts, ws.mid, ws.mid_t, ws.mid_3, c.n, c.ff, c.gateup_parts, ws.act_rows);
}

cudaError_t launch_combine_to_peers(const LaunchCfg& c, const CombineSrc& src, const uint8_t* block, int me,
                                    const PeerTable& peers, const PeerLayout& lay) {
    if (c.k > CB_MAX_K || c.e % 4) return cudaErrorInvalidValue;
    dim3 grid(c.n, (c.e / 4 + CB_THREADS - 1) / CB_THREADS);
    const PeerDest pd{peers, lay, (const int32_t*)(block + lay.counts), me};
    count_launch();
    return launch_after(c.stream, combine_kernel<true, CB_MANY, false>, grid, dim3(CB_THREADS), 0, src.ids, src.weights,
                        src.routed_rows, src.routed_pos, src.shared_rows, src.logits, (float*)nullptr, c.n, c.k,
                        c.e, c.n_expert, c.has_shared, 0, pd, NormDest{});
}

// ---------------------------------------------------------------------------
// Upload-time repack: GGUF rows -> tiled device layout (common.cuh).  One
// thread per 16-byte unit of the destination, the lanes of a warp one unit of 32 neighbouring
// places: it is written as 512 contiguous bytes, and the block's warps read on in the same rows
// (a row's units a warp, a byte at a time, wrote 16 bytes in 32 places: 256 experts of 2048 / 512 in Q4_K and
// Q6_K were made in 21.6 ms, so in 17.8; in BF16 54 and 42).  `tile_base` places the source
// matrix inside the chunk: 0 for gate and for down, 2 for up (chunk rows 64..127).
__device__ __forceinline__ uint32_t two_halves(const uint8_t* p) {   // every block format is made of 16-bit words
    return *(const uint16_t*)p | (uint32_t)*(const uint16_t*)(p + 2) << 16;
}
__global__ void repack_kernel(DevTiles dt, const uint8_t* __restrict__ src, int tile_base) {
    const int units = dt.slice_bytes / 16;
    const int64_t groups = (int64_t)dt.n * (dt.rows / 32);   // of 32 rows, which one matrix has a multiple of
    const int64_t total = groups * dt.nslices * units * 32;
    const int64_t grb = gguf_row_bytes(dt.ty, dt.cols);
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int u = (int)(i / 32 % units);
        const int s = (int)(i / (32 * units) % dt.nslices);
        const int64_t rg = i / ((int64_t)32 * units * dt.nslices) * 32 + row_of_place(dt.ty, (int)(i % 32));   // row over all experts
        const int64_t e = rg / dt.rows;
        const int r = (int)(rg % dt.rows);
        const int chunk = r / dt.chunk_rows, place = place_of_row(dt.ty, tile_base * 32 + r % dt.chunk_rows);
        const uint8_t* row = src + rg * grb;
        uint8_t* slice = dt.data + e * dt.expert_bytes + ((int64_t)chunk * dt.nslices + s) * dt.stage_bytes;
        const uint8_t* from = nullptr;
        switch (dt.ty) {
            case BIVMOE_Q4_K: from = row + 144 * (int64_t)s + 16 * u; break;
            case BIVMOE_Q5_K: from = row + 176 * (int64_t)s + 16 * u; break;
            case BIVMOE_BF16:
            case BIVMOE_F16: from = row + 128 * (int64_t)s + 16 * u; break;
            case BIVMOE_F32: from = row + 256 * (int64_t)s + 16 * u; break;
            case BIVMOE_Q4_0:
                if (u < 8) from = row + 18 * (int64_t)(8 * s + u) + 2;
                break;
            case BIVMOE_Q4_1:
                if (u < 8) from = row + 20 * (int64_t)(8 * s + u) + 4;
                break;
            case BIVMOE_Q6_K: from = row + 210 * (int64_t)s + 16 * u; break;   // ql, qh, scales in order
            case BIVMOE_Q8_0:
                if (u < 16) from = row + 34 * (int64_t)(8 * s + u / 2) + 2 + 16 * (u % 2);
                break;
        }
        uint4 v;
        if (from && ((uintptr_t)from & 15) == 0) {
            v = *(const uint4*)from;
        } else if (from) {
            v = make_uint4(two_halves(from), two_halves(from + 4), two_halves(from + 8), two_halves(from + 12));
        } else {   // the eight f16 scales of the slice (Q4_1 unit 9: its eight f16 minimums)
            const int bb = dt.ty == BIVMOE_Q8_0 ? 34 : dt.ty == BIVMOE_Q4_0 ? 18 : 20;
            const uint8_t* p = row + bb * (int64_t)(8 * s) + (dt.ty == BIVMOE_Q4_1 && u == 9 ? 2 : 0);
            uint32_t w[4];
            for (int b = 0; b < 4; b++)
                w[b] = *(const uint16_t*)(p + 2 * b * bb) | (uint32_t)*(const uint16_t*)(p + (2 * b + 1) * bb) << 16;
            v = make_uint4(w[0], w[1], w[2], w[3]);
        }
        *(uint4*)(slice + ((int64_t)u * kChunkRows + (place ^ unit_shift(dt.ty, u))) * 16) = v;
        if (dt.ty == BIVMOE_Q6_K && u == 0)
            *(uint16_t*)(slice + kChunkRows * (int64_t)dt.slice_bytes + 2 * place) = *(const uint16_t*)(row + 210 * (int64_t)s + 208);
    }
}

cudaError_t launch_repack(const DevTiles& dst, const uint8_t* gguf_rows, int tile_base,
                          cudaStream_t stream) {
    repack_kernel<<<2048, 256, 0, stream>>>(dst, gguf_rows, tile_base);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Parity tap: the int32 dot of each 32-element block of one weight row with one
// Q8 activation row, decoded byte by byte as the reference's scalar kernels
// define the values (quant.rs:599-686).  One thread per block; not on the
// timed path.
__device__ inline uint8_t tile_byte(const DevTiles& t, const uint8_t* chunk0, int place, int s, int off) {
    // chunk0: K-slice 0 of the row's chunk, where the row lies at `place`; byte `off` of the row's slice s
    return chunk0[(int64_t)s * t.stage_bytes + ((off >> 4) * kChunkRows + (place ^ unit_shift(t.ty, off >> 4))) * 16 +
                  (off & 15)];
}

__global__ void block_dots_kernel(DevTiles t, int tile_base, int expert, int row,
                                  const uint8_t* __restrict__ act_t, int act_rows, int pos, int half,
                                  int32_t* __restrict__ out) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;   // 32-element block of the row
    if (b >= t.cols / 32) return;
    const int chunk = row / t.chunk_rows, rr = place_of_row(t.ty, tile_base * 32 + row % t.chunk_rows);
    const uint8_t* t0 = t.stage(expert, chunk, 0);
    const int s = b / 8, sb = b % 8;
    const uint8_t* rec = act_t + ((size_t)s * (act_rows / 8) + pos / 8) * (half ? kHalfRec : kActTileBytes);
    int8_t x[32];
    for (int l = 0; l < 32; l++)
        x[l] = half ? (int8_t)__half2int_rn(*(const __half*)(rec + half_q_off(pos % 8, 32 * sb + l)))
                    : *(const int8_t*)(rec + act_q_off(pos % 8, 32 * sb + l));
    int32_t sum = 0;
    if (t.ty == BIVMOE_Q8_0) {
        for (int l = 0; l < 32; l++) sum += (int)(int8_t)tile_byte(t, t0, rr, s, 32 * sb + l) * x[l];
    } else if (t.ty == BIVMOE_Q4_0 || t.ty == BIVMOE_Q4_1) {
        // quant.rs:574-577, 589-592: byte j = element j (low half) and j + 16 (high half)
        for (int l = 0; l < 32; l++) {
            const int q = (tile_byte(t, t0, rr, s, 16 * sb + (l & 15)) >> (4 * (l >> 4))) & 0xF;
            sum += (t.ty == BIVMOE_Q4_0 ? q - 8 : q) * x[l];
        }
    } else if (t.ty == BIVMOE_Q4_K || t.ty == BIVMOE_Q5_K) {
        const int qoff = (t.ty == BIVMOE_Q4_K ? 16 : 48) + 32 * (sb / 2);
        for (int l = 0; l < 32; l++) {
            int q = (tile_byte(t, t0, rr, s, qoff + l) >> (4 * (sb % 2))) & 0xF;
            if (t.ty == BIVMOE_Q5_K) q |= ((tile_byte(t, t0, rr, s, 16 + l) >> sb) & 1) << 4;
            sum += q * x[l];
        }
    } else if (t.ty == BIVMOE_Q6_K) {
        const int n = sb / 4, kq = sb % 4;
        for (int half = 0; half < 2; half++) {
            int32_t part = 0;
            for (int l = 16 * half; l < 16 * half + 16; l++) {
                const int ql = tile_byte(t, t0, rr, s, 64 * n + 32 * (kq & 1) + l);
                const int qh = tile_byte(t, t0, rr, s, 128 + 32 * n + l);
                const int nib = kq >= 2 ? ql >> 4 : ql & 0xF;
                part += ((nib | (((qh >> (2 * kq)) & 3) << 4)) - 32) * x[l];
            }
            sum += (int)(int8_t)tile_byte(t, t0, rr, s, 192 + 8 * n + 2 * kq + half) * part;
        }
    }
    out[b] = sum;
}

cudaError_t launch_block_dots(const DevTiles& t, int tile_base, int expert, int row,
                              const uint8_t* act_t, int act_rows, int pos, bool half, int32_t* out,
                              cudaStream_t stream) {
    const int nb = t.cols / 32;
    block_dots_kernel<<<(nb + 63) / 64, 64, 0, stream>>>(t, tile_base, expert, row, act_t, act_rows,
                                                         pos, half ? 1 : 0, out);
    return cudaGetLastError();
}

}  // namespace bivmoe
