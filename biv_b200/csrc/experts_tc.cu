// Grouped expert products with k-quant weights (Q4_K, Q5_K, Q6_K) on the 5th generation tensor
// cores, for passes whose groups have some tens of rows: gate+up with the SwiGLU and the Q8
// re-quantisation of its output fused, then down.  (Groups of a few rows: experts_quant.cu.)
// Reference: dense_ffn (engine/src/model.rs:1119-1126) over matmul
// (engine/src/ops.rs:84-127) and the per-type dots (engine/src/quant.rs:609-686), for each
// expert's token list (model.rs:875-889) and for the shared expert (model.rs:890-896).
//
// A 32-element block dot is a sum of products of small integers, scaled by the weight block's
// scale and the activation block's.  Both operands are fed as f16 - integers up to 2048 are exact
// there - and the f32 sums of a block's products are exact (below 2^24).  What makes the
// tensor core worth it is that the integer part of the scale goes into the weight on the way:
// sc * q of Q4_K and Q5_K is at most 63 * 31 = 1953, one exact f16; sc * (q - 32) of Q6_K is an
// f16 and a remainder of -1, 0 or 1, two terms that meet the same activations.  What is left to
// do for each of the 128 x tokens sums of a block is one multiply-add with d_x; the row's d comes in
// once per 256 columns.
//
// Design.  One block per SM and twenty-six warps.  A work item is a tile of up to 64 tokens of one
// group times one chunk of 128 weight rows (64 gate rows with their 64 up rows, or 128 down rows).
//   warp 0      one lane walks the block's items (item i of a launch belongs to block i mod
//               gridDim.x) and keeps a ring of stages full: one K-slice of 256 columns of the
//               chunk and the tile's activation records, two bulk copies, with a descriptor
//   warp 1      one lane issues the MMAs: per block two tcgen05.mma kind::f16 (128 x N x 16; four
//               for Q6_K), the weights from tensor memory, the activations from the stage
//   warps 2-9   unpack the weights: a thread has a row (= a tensor-memory lane), four warps the
//               first four blocks of a stage, four the others, each half into its own place in
//               tensor memory, so that the halves' MMAs and unpacking overlap
//   warps 10-25 drain the sums: a warp has 32 lanes and a quarter of the tokens, a thread four rows and
//               two of every eight tokens (tcgen05.ld 16x256b), so that the two d_x of a block it needs
//               for eight sums are one load - shared memory is the busiest unit (a row and sixteen
//               tokens a thread: twice as fast out of tensor memory, 448 bytes a clock and SM, but four
//               times the loads of d_x); the sums of two blocks come at a time, in two buffers
// The lanes of a gate+up chunk are dealt so that a thread's rows are gate rows and the up rows of
// the same outputs.  The min term sum m * s_x of Q4_K and Q5_K is one tf32 MMA per half of s_x (m is a
// 6-bit integer, s_x is kept as two tf32-exact halves), whose sums follow those of the stage's last block.
// What bounds it: neither MMAs, unpacking nor arithmetic - with any of them left out it takes as long -
// but the way of the sums, four fills a stage, each a chain of commit, wait, tensor-memory loads
// (256 bytes a clock; all left out, 211 us of 287) and arrivals: with them alone it takes half of the
// time.  About 3550 clocks for 128 rows x 256 columns x 64 tokens, where the warp-MMA kernel takes some
// 5000.  (Fills of one block in four buffers 8 % slower; the loads of a fill issued together, unpacking
// by four warps, or a warp pair of its own for the Q8 records of gate+up within 3 % either way.)
// gate+up + down of 2048 / 512, us, warp MMA -> this: Q4_K / Q6_K, 4096 rows over 256 experts 797 +
// 565 -> 571 + 318; 500 rows over 64 (6 each) 99 + 46 -> 72 + 43; dense 4096 / 8192, 512 rows 310 + 248 ->
// 208 + 125.
// Every wait of a role for another is bounded.  The copying lane's by 2 s: it is there as long as the
// others, and when a slot, or the end, is not reached in that time it records BIVMOE_ERR_TIMEOUT (and
// which wait it was) in the status words and raises a block-wide flag on which every role leaves its
// loop, a warp as a whole (the copying lane waits, bounded again, for its copies still in flight, the
// MMA lane for its MMAs).
// No atomics on data: results are run-to-run identical.
#include <cuda_fp16.h>

#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "formats.cuh"
#include "tcgen05.cuh"
#include "launch.cuh"

namespace bivmoe {

enum { TC_GATEUP = 0, TC_DOWN = 1 };
constexpr int TC_DEQ_WARPS = 8, TC_EPI_WARPS = 16;
constexpr int TC_WARPS = 2 + TC_DEQ_WARPS + TC_EPI_WARPS, TC_THREADS = 32 * TC_WARPS;
constexpr int TC_HEAD = 1024;             // barriers, abort flag, stage descriptors
constexpr int TC_MID_STRIDE = 68;         // floats a token of the SwiGLU tile: 8 tokens apart fall into different banks
constexpr uint32_t TC_TMEM_COLS = 512;
constexpr int TC_N = kWideTile;           // tokens of a tile at most

struct TcArgs {
    DevTiles w, sh;        // the routed experts' and the shared expert's tiles for this product
    const uint8_t* x_t;    // Q8 records of the inputs by position, [K/256][R/8]
    int act_rows;          // R
    float* out;            // GATEUP: mid f32 slice-major; DOWN: pair_out [R][rows]
    uint8_t* out_t;        // GATEUP with a quantised down type: Q8 records of mid
    const int4* tile_desc; // {expert (n_expert: shared), first position, tokens, 0}
    const int32_t* n_tiles;
    int32_t* status;
    int n_expert;
    int tiles_mode;        // 0: every tile, 1: skip the shared group's, 2: only the shared group's
    int chunks;            // row chunks per group in this launch
    int parts;             // DOWN: K is cut into this many parts, a work item each (1: not cut) ...
    int part_rows;         // ... whose sums go to out as [part][part_rows][rows]
};

struct TcStage {        // what the copying lane tells the others about a stage
    int pos0, tc;       // the tile: first position, tokens
    int chunk, rows;    // chunk of the expert's matrix; its rows (down: the stride of the output rows)
    int flags;          // TCS_*
    int part;
    int pad[2];
};
enum { TCS_FIRST = 1, TCS_LAST = 2, TCS_END = 4 };
// which bounded wait gave up (status word 2, for the error text)
enum { TC_SITE_COPY = 21, TC_SITE_MMA, TC_SITE_UNPACK, TC_SITE_EPILOGUE };

__device__ __forceinline__ uint32_t h2_bits(__half2 v) { return *(uint32_t*)&v; }
__device__ __forceinline__ __half2 as_h2(uint32_t v) { return *(__half2*)&v; }
__device__ __forceinline__ __half2 h2_both(__half v) { return __halves2half2(v, v); }
// bytes 0 and 2, or 1 and 3, of w as the low mantissa bytes of two f16 numbers of 1024
__device__ __forceinline__ uint32_t bytes02(uint32_t w) { return __byte_perm(w, 0x64646464u, 0x4240); }
__device__ __forceinline__ uint32_t bytes13(uint32_t w) { return __byte_perm(w, 0x64646464u, 0x4341); }

// 16 columns of tensor memory, this warp's 32 lanes
__device__ __forceinline__ void tc_tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
        "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}
// Bounded waits (bounded_wait.h) of a lane by itself and of a whole warp.  (There are some hundred waits
// a stage, most of which find their phase complete: with a look at the clock in each of them, if only
// once in 256 tries, the kernel takes 3 to 6 % longer.)  SLEEP: a role that waits long - its tries would
// take issue slots from the others.
template <bool SLEEP = false>
__device__ __forceinline__ bool tc_wait(uint64_t* bar, uint32_t parity, const int* s_abort) {
    return bounded_wait<256>(PfWait<false, SLEEP>{bar, parity, s_abort});
}
template <bool SLEEP = false>
__device__ __forceinline__ bool tc_wait_warp(uint64_t* bar, uint32_t parity, const int* s_abort) {
    return bounded_wait_together<256>(PfWait<false, SLEEP>{bar, parity, s_abort});
}
__device__ __forceinline__ void tc_tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// D (+)= A * B, 16 f16 values of K per instruction, A (rows = lanes) in tensor memory
__device__ __forceinline__ void tc_mma_f16(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc,
                                           uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
        "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// D (+)= A * B, 8 tf32 values of K per instruction, both in shared memory
__device__ __forceinline__ void tc_mma_tf32(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                            uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// instruction descriptors: f32 accumulator, both operands K-major; f16 x f16, tf32 x tf32
__device__ __forceinline__ uint32_t tc_idesc_f16(int n) {
    return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kChunkRows >> 4) << 24);
}
__device__ __forceinline__ uint32_t tc_idesc_tf32(int n) { return tc_idesc_f16(n) | (2u << 7) | (2u << 10); }

// ---------------------------------------------------------------------------
// The formats.  unpack(at, h, put, put_min): the thread's row of a stage, `at` its 16-byte piece
// of unit 0, `alt` that of odd units (unit u is 2048 u further); put(b, t, v) stores term t of block
// 4 h + b, the sixteen f16 pairs of its K values in the order 0 2 1 3 of every four; put_min(m) the
// minimums of the four blocks.
//   MIN      a minimum per block         TERMS   f16 terms of a weight
template <int TY> struct TcFmt;

template <int TY> struct TcK45 {   // Q4_K, Q5_K (quant.rs:609-649)
    static constexpr bool MIN = true;
    static constexpr int TERMS = 1;
    template <class Put, class PutMin>
    static __device__ __forceinline__ void unpack(uint32_t at, uint32_t alt, int h, Put put, PutMin put_min) {
        const uint4 hd = lds128(at);
        uint4 qh[2];
        if (TY == BIVMOE_Q5_K) {
            qh[0] = lds128(alt + 2048);
            qh[1] = lds128(at + 2 * 2048);
        }
        // 32-byte groups 2 h and 2 h + 1: blocks 2 j (low nibbles) and 2 j + 1 (high nibbles) each
        constexpr int QU = TY == BIVMOE_Q4_K ? 1 : 3;   // odd
        const K4Scales k = unpack_k4_scales(hd.y, hd.z, hd.w);
        const uint32_t sc = h ? k.sc_hi : k.sc_lo, mn = h ? k.m_hi : k.m_lo;
        float m[4];
#pragma unroll
        for (int b = 0; b < 4; b++) m[b] = (float)((mn >> (8 * b)) & 0xFFu);
        put_min(m);
        const uint32_t s02 = bytes02(sc), s13 = bytes13(sc);
        const __half2 k1024 = as_h2(0x64006400u);
        const __half2 sp[2] = {__hsub2(as_h2(s02), k1024), __hsub2(as_h2(s13), k1024)};   // scales 0, 2 and 1, 3
        const uint32_t hb[8] = {qh[0].x, qh[0].y, qh[0].z, qh[0].w, qh[1].x, qh[1].y, qh[1].z, qh[1].w};
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const uint4 w0 = lds128(alt + (QU + 4 * h + 2 * j) * 2048), w1 = lds128(at + (QU + 4 * h + 2 * j + 1) * 2048);
            const uint32_t ww[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
            const __half2 slo = j ? __high2half2(sp[0]) : __low2half2(sp[0]);
            const __half2 shi = j ? __high2half2(sp[1]) : __low2half2(sp[1]);
            uint32_t v[2][16];
            if (TY == BIVMOE_Q4_K) {
                // (1024 + q) sc - 1024 sc, and with the high nibble in place (1024 + 16 q) sc / 16 - 64 sc: exact
                const __half2 s16 = __hmul2(shi, as_h2(0x2C002C00u));
                const __half2 olo = __hmul2(slo, as_h2(0xE400E400u)), ohi = __hmul2(s16, as_h2(0xE400E400u));
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const uint32_t a = ww[i], b = ww[i] >> 8;
                    v[0][2 * i] = h2_bits(__hfma2(as_h2((a & 0x000F000Fu) | 0x64006400u), slo, olo));
                    v[0][2 * i + 1] = h2_bits(__hfma2(as_h2((b & 0x000F000Fu) | 0x64006400u), slo, olo));
                    v[1][2 * i] = h2_bits(__hfma2(as_h2((a & 0x00F000F0u) | 0x64006400u), s16, ohi));
                    v[1][2 * i + 1] = h2_bits(__hfma2(as_h2((b & 0x00F000F0u) | 0x64006400u), s16, ohi));
                }
            } else {
                const __half2 olo = __hmul2(slo, as_h2(0xE400E400u)), ohi = __hmul2(shi, as_h2(0xE400E400u));
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const uint32_t hs = h ? hb[i] >> (2 * j) : hb[i] << (4 - 2 * j);   // bit 4: block 4 h + 2 j
                    const uint32_t lo = (ww[i] & 0x0F0F0F0Fu) | (hs & 0x10101010u);
                    const uint32_t hi = ((ww[i] >> 4) & 0x0F0F0F0Fu) | ((hs >> 1) & 0x10101010u);
                    v[0][2 * i] = h2_bits(__hfma2(as_h2(bytes02(lo)), slo, olo));
                    v[0][2 * i + 1] = h2_bits(__hfma2(as_h2(bytes13(lo)), slo, olo));
                    v[1][2 * i] = h2_bits(__hfma2(as_h2(bytes02(hi)), shi, ohi));
                    v[1][2 * i + 1] = h2_bits(__hfma2(as_h2(bytes13(hi)), shi, ohi));
                }
            }
            put(2 * j, 0, v[0]);
            put(2 * j + 1, 0, v[1]);
        }
    }
    // d and dmin of a row (`at`: the row's piece of unit 0)
    static __device__ __forceinline__ float2 factors(uint32_t at) {
        const uint32_t v = lds32(at);
        return __half22float2(as_h2(v));
    }
};
template <> struct TcFmt<BIVMOE_Q4_K> : TcK45<BIVMOE_Q4_K> {};
template <> struct TcFmt<BIVMOE_Q5_K> : TcK45<BIVMOE_Q5_K> {};

template <> struct TcFmt<BIVMOE_Q6_K> {   // quant.rs:651-686: sc (q - 32) per 16 values
    static constexpr bool MIN = false;
    static constexpr int TERMS = 2;
    template <class Put, class PutMin>
    static __device__ __forceinline__ void unpack(uint32_t at, uint32_t alt, int h, Put put, PutMin) {
        // half h is the super-block's 128-value half: ql units 4 h .. + 3, qh units 8 + 2 h, + 1
        uint4 ql[4], qh[2];
#pragma unroll
        for (int u = 0; u < 4; u++) ql[u] = lds128((u & 1 ? alt : at) + (4 * h + u) * 2048);
        qh[0] = lds128(at + (8 + 2 * h) * 2048);
        qh[1] = lds128(alt + (9 + 2 * h) * 2048);
        const uint4 sc4 = lds128(at + 12 * 2048);
        const uint32_t sc[2] = {h ? sc4.z : sc4.x, h ? sc4.w : sc4.y};   // sub-blocks 8 h .. + 3, + 4 .. + 7
        const __half2 bias = as_h2(0xE420E420u);   // -1056
#pragma unroll
        for (int kq = 0; kq < 4; kq++) {           // block 4 h + kq
            uint32_t hi[16], lo[16];
#pragma unroll
            for (int s = 0; s < 2; s++) {
                const int8_t si = (int8_t)(sc[kq >> 1] >> (8 * (2 * (kq & 1) + s)));
                const __half2 ss = h2_both(__int2half_rn((int)si));
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const uint4 &l4 = ql[2 * (kq & 1) + s], &h4 = qh[s];
                    const uint32_t lw = i == 0 ? l4.x : i == 1 ? l4.y : i == 2 ? l4.z : l4.w;
                    const uint32_t hw = i == 0 ? h4.x : i == 1 ? h4.y : i == 2 ? h4.z : h4.w;
                    const uint32_t nib = (kq < 2 ? lw : lw >> 4) & 0x0F0F0F0Fu;
                    const uint32_t top = kq == 0 ? hw << 4 : kq == 1 ? hw << 2 : kq == 2 ? hw : hw >> 2;
                    const uint32_t q = nib | (top & 0x30303030u);
#pragma unroll
                    for (int p = 0; p < 2; p++) {
                        const __half2 x = __hadd2(as_h2(p ? bytes13(q) : bytes02(q)), bias);
                        const __half2 y = __hmul2_rn(x, ss);
                        hi[8 * s + 2 * i + p] = h2_bits(y);
                        lo[8 * s + 2 * i + p] = h2_bits(__hfma2(x, ss, __hneg2(y)));
                    }
                }
            }
            put(kq, 0, hi);
            put(kq, 1, lo);
        }
    }
    static __device__ __forceinline__ float factor(uint32_t d_at) {   // d of a row
        unsigned short v;
        asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(d_at));
        return __half2float(__ushort_as_half(v));
    }
};

// ---------------------------------------------------------------------------
// sizes
template <int TY> struct TcSize {
    using F = TcFmt<TY>;
    static constexpr uint32_t W = slice_stage_bytes(TY), M = F::MIN ? 4096 : 0;
    static constexpr uint32_t X_LAST = F::MIN ? kHalfOffS : kHalfOffSHi;      // of a tile's last record
    // tensor memory: two buffers of sums, then the unpacked halves of a stage
    static constexpr uint32_t D = F::MIN ? 192 : 128;
    static constexpr uint32_t A_HALF = 64 * F::TERMS, A0 = 2 * D;
    static_assert(A0 + 2 * A_HALF <= TC_TMEM_COLS, "tensor memory");
};
template <int TY> __host__ __device__ constexpr uint32_t tc_stage_bytes() {
    return TcSize<TY>::W + TcSize<TY>::M + TC_N / 8 * kHalfRec;
}
template <int MODE> __host__ __device__ constexpr uint32_t tc_mid_bytes() {
    return MODE == TC_GATEUP ? TC_N * TC_MID_STRIDE * 4 : 0;
}
template <int TY, int MODE> __host__ __device__ constexpr int tc_slots() {
    const int s = (227 * 1024 - TC_HEAD - (int)tc_mid_bytes<MODE>()) / (int)tc_stage_bytes<TY>();
    return s < 8 ? s : 8;
}
template <int TY, int MODE> __host__ __device__ constexpr int tc_smem() {
    return TC_HEAD + (int)tc_mid_bytes<MODE>() + tc_slots<TY, MODE>() * (int)tc_stage_bytes<TY>();
}

// The epilogue warps meet; one that gave up arrives for the others (arrive_until_all_left).
__device__ __forceinline__ void tc_epi_sync() { asm volatile("bar.sync 1, %0;" ::"n"(32 * TC_EPI_WARPS) : "memory"); }

// The place in the chunk of the row that a tensor-memory lane holds.  Gate+up: lanes 16 m .. + 7 the gate rows
// at places 8 m .., the next eight lanes the up rows of the same outputs; down: as they lie.
template <int MODE> __device__ __forceinline__ int tc_row(int l) {
    return MODE == TC_GATEUP ? ((l >> 3) & 1) * 64 + (l >> 4) * 8 + (l & 7) : l;
}

// The sums of a stage come in four fills of two buffers, two blocks each (for every N, so that a fill's
// buffer and the parities of its barriers are constants).
// One stage of a tile of up to N tokens, for the MMA lane.  False when a wait gave up.
template <int TY, int N>
__device__ __forceinline__ bool tc_mma_stage(int tc, uint32_t st, uint64_t* afull, uint64_t* aempty, uint64_t* dfull,
                                             uint64_t* dempty, uint32_t parity, const int* s_abort) {
    using F = TcFmt<TY>;
    using S = TcSize<TY>;
    const int n_mma = (tc + 15) & ~15;
    const uint32_t idesc = tc_idesc_f16(n_mma);
    // B: the tokens' units 4 b .. 4 b + 3 of 8 K values: 8-token groups one record apart, the two units of
    // an MMA 128 B apart
    const uint64_t bd = pf_desc(st + S::W + S::M, 128, kHalfRec);
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int h = i >> 1, buf = i & 1;
        if (buf == 0) {
            if (!tc_wait(&afull[h], parity, s_abort)) return false;
        }
        if (!tc_wait<true>(&dempty[buf], 1 - h, s_abort)) return false;
        pf_fence_after();
#pragma unroll
        for (int p = 0; p < 2; p++) {
            const int b = 2 * i + p;
            const uint32_t dt = buf * S::D + p * N, a0 = S::A0 + h * S::A_HALF + (b & 3) * F::TERMS * 16;
#pragma unroll
            for (int t = 0; t < F::TERMS; t++)
#pragma unroll
                for (int ks = 0; ks < 2; ks++)
                    tc_mma_f16(dt, a0 + t * 16 + ks * 8, bd + (b * 512 + ks * 256) / 16, idesc, (t | ks) != 0);
        }
        if (F::MIN && i == 3) {
            // A: the rows' minimums [2 units][128 lanes][4]; B: s_x, [2 units][8 tokens][4]
            const uint32_t id2 = tc_idesc_tf32(n_mma);
            const uint64_t ad = pf_desc(st + S::W, 2048, 128);
            tc_mma_tf32(buf * S::D + 128, ad, bd + kHalfOffSHi / 16, id2, 0);
            tc_mma_tf32(buf * S::D + 128, ad, bd + kHalfOffSLo / 16, id2, 1);
        }
        pf_commit(&dfull[buf]);
        if (buf == 1) pf_commit(&aempty[h]);
    }
    return true;
}

// One stage of a tile of up to N tokens, for an epilogue thread: the rows at places `rows` (lanes g + 8 i of its warp's
// 32), the token pairs 2 c of the N / 32 octets from `oct` on (N = 16: one, or none).  False when a wait
// gave up.
template <int TY, int N, int JMAX>
__device__ __forceinline__ bool tc_epi_stage(f32x2 (&acc)[4][JMAX], uint32_t tlane, uint32_t w, uint32_t x, const int (&rows)[4],
                                             int oct, int lane, uint64_t* dfull, uint64_t* dempty, const int* s_abort) {
    using F = TcFmt<TY>;
    using S = TcSize<TY>;
    constexpr int J = N == 64 ? 2 : 1;
    const bool any = N > 16 || oct < 2;          // uniform
    const uint32_t xd = x + kHalfOffDx + oct * kHalfRec + (lane & 3) * 8;
    f32x2 ts[4][J];
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
        for (int j = 0; j < J; j++) ts[r][j] = 0ull;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int buf = i & 1;
        if (!tc_wait_warp(&dfull[buf], i >> 1, s_abort)) return false;
        pf_fence_after();
        const uint32_t at = tlane + buf * S::D + 8 * oct;
#pragma unroll
        for (int p = 0; p < 2; p++) {
            const int b = 2 * i + p;
            int v[2][4 * J];
            f32x2 dx[J];
            if (any) {
                pf_tmem_ld_16x8<J>(at + p * N, v[0]);
                pf_tmem_ld_16x8<J>(at + p * N + (16u << 16), v[1]);
            }
#pragma unroll
            for (int j = 0; j < J; j++) dx[j] = lds_f2(xd + j * kHalfRec + b * 32);
            pf_tmem_wait_ld();
            if (p == 1 && !(F::MIN && i == 3)) {
                pf_fence_before();
                __syncwarp();
                if (lane == 0) pf_bar_arrive(&dempty[buf]);
            }
#pragma unroll
            for (int r = 0; r < 4; r++)
#pragma unroll
                for (int j = 0; j < J; j++) {
                    const int* d2 = &v[r >> 1][4 * j + 2 * (r & 1)];
                    ts[r][j] = fma2(dx[j], pk(__int_as_float(d2[0]), __int_as_float(d2[1])), ts[r][j]);
                }
        }
        if constexpr (F::MIN) if (i == 3) {
            // the minimums' sums, and the stage is complete
            int m[2][4 * J];
            if (any) {
                pf_tmem_ld_16x8<J>(at + 128, m[0]);
                pf_tmem_ld_16x8<J>(at + 128 + (16u << 16), m[1]);
            }
            float2 f[4];
#pragma unroll
            for (int r = 0; r < 4; r++) f[r] = F::factors(w + rows[r] * 16);
            pf_tmem_wait_ld();
            pf_fence_before();
            __syncwarp();
            if (lane == 0) pf_bar_arrive(&dempty[buf]);
#pragma unroll
            for (int r = 0; r < 4; r++)
#pragma unroll
                for (int j = 0; j < J; j++) {
                    const int* m2 = &m[r >> 1][4 * j + 2 * (r & 1)];
                    const f32x2 tm = pk(__int_as_float(m2[0]), __int_as_float(m2[1]));
                    acc[r][j] = add2(acc[r][j], fma2(pk(f[r].x, f[r].x), ts[r][j], mul2(pk(-f[r].y, -f[r].y), tm)));
                }
        }
    }
    if constexpr (!F::MIN) {
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const float d = F::factor(w + kChunkRows * 208 + rows[r] * 2);
#pragma unroll
            for (int j = 0; j < J; j++) acc[r][j] = fma2(pk(d, d), ts[r][j], acc[r][j]);
        }
    }
    return true;
}

template <int TY, int MODE>
__global__ void __launch_bounds__(TC_THREADS, 1)
experts_tc_kernel(const TcArgs A) {
    using F = TcFmt<TY>;
    using S = TcSize<TY>;
    constexpr int SLOTS = tc_slots<TY, MODE>(), JMAX = TC_N / 32;
    constexpr uint32_t SB = tc_stage_bytes<TY>();
    constexpr int CH = MODE == TC_GATEUP ? 64 : 128;   // output rows per chunk
    static_assert(SLOTS >= 2, "stages");
    pdl_launch_dependents();
    extern __shared__ __align__(1024) uint8_t smem[];
    uint64_t* full = (uint64_t*)smem;            // [SLOTS] a stage has landed
    uint64_t* empty = full + 8;                  // [SLOTS] the unpacking and the epilogue warps, and with them the MMAs, are done with it
    uint64_t* afull = full + 16;                 // [2] a half of the stage is unpacked
    uint64_t* aempty = full + 18;                // [2] its MMAs are done
    uint64_t* dfull = full + 20;                 // [2] a buffer of sums is complete
    uint64_t* dempty = full + 22;                // [2] it is drained
    uint64_t* done = full + 24;                  // everything the MMA lane issued has completed
    uint64_t* left = full + 25;                  // the unpacking and the epilogue warps have left their loops
    uint32_t* s_tmem = (uint32_t*)(smem + 256);
    int* s_abort = (int*)(smem + 260);
    TcStage* s_desc = (TcStage*)(smem + 512);    // [SLOTS]
    float* s_mid = (float*)(smem + TC_HEAD);     // [TC_N][TC_MID_STRIDE]
    uint8_t* ring = smem + TC_HEAD + tc_mid_bytes<MODE>();
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);   // uniform

    if (tid == 0) {
        for (int i = 0; i < SLOTS; i++) {
            pf_bar_init(&full[i], 1);
            pf_bar_init(&empty[i], TC_DEQ_WARPS + TC_EPI_WARPS);
        }
        for (int i = 0; i < 2; i++) {
            pf_bar_init(&afull[i], TC_DEQ_WARPS / 2);
            pf_bar_init(&aempty[i], 1);
            pf_bar_init(&dfull[i], 1);
            pf_bar_init(&dempty[i], TC_EPI_WARPS);
        }
        pf_bar_init(done, 1);
        pf_bar_init(left, TC_DEQ_WARPS + TC_EPI_WARPS);
        *s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {   // tensor memory: all 512 columns for the whole kernel
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         pf_smem(s_tmem)),
                     "r"(TC_TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    pf_fence_before();
    __syncthreads();
    pf_fence_after();
    constexpr uint32_t tmem = 0;   // all 512 columns are the block's: they start at 0
    pdl_wait();   // the tile lists and the activation records are the previous kernels'

    auto give_up = [&](int site) {
        if (atomicExch(A.status, BIVMOE_ERR_TIMEOUT) == 0) atomicExch(A.status + 2, site);
        atomicExch(s_abort, 1);
    };

    if (*s_tmem != tmem) {
        if (tid == 0) give_up(TC_SITE_COPY);
    } else if (warp == 0) {
        // ---------------- the copying lane
        if (pf_elect()) {
            const int tiles_all = A.n_tiles[0], tiles_sh = A.n_tiles[1];
            const int tile_lo = A.tiles_mode == 1 ? tiles_sh : 0;
            const int tile_hi = A.tiles_mode == 2 ? tiles_sh : tiles_all;
            const int parts = MODE == TC_DOWN ? A.parts : 1;
            const int units = (tile_hi - tile_lo) * A.chunks * parts;
            uint32_t q = 0;
            bool dead = false;
            auto wait_slot = [&]() {
                if (bounded_wait<256>(PfWait<true, true>{&empty[q % SLOTS], ((q / SLOTS) & 1) ^ 1, s_abort})) return true;
                give_up(TC_SITE_COPY);
                return false;
            };
            for (int idx = blockIdx.x; idx < units && !dead; idx += gridDim.x) {
                TcStage d{};
                d.part = idx % parts;
                const int rest = idx / parts;
                d.chunk = rest % A.chunks;
                const int4 td = A.tile_desc[tile_lo + rest / A.chunks];
                const bool shared = td.x == A.n_expert;
                const DevTiles& m = shared ? A.sh : A.w;
                const int all = d.chunk < m.chunks ? m.nslices : 0;
                const int from = all * d.part / parts, to = all * (d.part + 1) / parts;
                if (from >= to) continue;
                d.pos0 = td.y;
                d.tc = td.z;
                d.rows = m.rows;
                const uint8_t* src = m.stage(shared ? 0 : td.x, d.chunk, 0);
                const uint32_t x_bytes = (uint32_t)((d.tc + 7) / 8 - 1) * kHalfRec + S::X_LAST;
                for (int s = from; s < to; s++, q++) {
                    if (!wait_slot()) { dead = true; break; }
                    const uint32_t slot = q % SLOTS;
                    d.flags = (s == from ? TCS_FIRST : 0) | (s == to - 1 ? TCS_LAST : 0);
                    s_desc[slot] = d;
                    uint8_t* dst = ring + (size_t)slot * SB;
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the slot was last read through the generic proxy
                    pf_bar_expect_tx(&full[slot], S::W + x_bytes);
                    pf_bulk_g2s(dst, src + (size_t)s * S::W, S::W, &full[slot]);
                    pf_bulk_g2s(dst + S::W + S::M, A.x_t + ((size_t)s * (A.act_rows / 8) + d.pos0 / 8) * kHalfRec,
                                x_bytes, &full[slot]);
                }
            }
            const bool ended = !dead && wait_slot();
            if (ended) {   // the end marker: a stage without data
                TcStage d{};
                d.flags = TCS_END;
                s_desc[q % SLOTS] = d;
                pf_bar_arrive(&full[q % SLOTS]);
            }
            // no copy is left in flight when the block ends, whoever gave up on it: the last one of
            // every slot has landed, or was waited for
            for (uint32_t last = q + ended, p = last > SLOTS ? last - SLOTS : 0; p < q; p++)
                pf_bar_wait(&full[p % SLOTS], (p / SLOTS) & 1);
            // and the clock that bounds the others' waits runs until they are done
            if (!bounded_wait<256>(PfWait<true, true>{left, 0, s_abort})) give_up(TC_SITE_COPY);
        }
    } else if (warp == 1) {
        // ---------------- the MMA lane
        if (pf_elect()) {
            uint32_t slot = 0, phase = 0, parity = 0;
            const uint32_t ring_a = pf_smem(ring);
            while (true) {
                if (!tc_wait(&full[slot], phase, s_abort)) { give_up(TC_SITE_MMA); break; }
                const int tc = s_desc[slot].tc;
                if (s_desc[slot].flags & TCS_END) break;
                const uint32_t st = ring_a + slot * SB;
                bool ok;
                if (tc > 32) ok = tc_mma_stage<TY, 64>(tc, st, afull, aempty, dfull, dempty, parity, s_abort);
                else if (tc > 16) ok = tc_mma_stage<TY, 32>(tc, st, afull, aempty, dfull, dempty, parity, s_abort);
                else ok = tc_mma_stage<TY, 16>(tc, st, afull, aempty, dfull, dempty, parity, s_abort);
                if (!ok) { give_up(TC_SITE_MMA); break; }
                parity ^= 1;
                if (++slot == SLOTS) { slot = 0; phase ^= 1; }
            }
            // no MMA and no arrival of a commit is left behind when the block ends
            pf_commit(done);
            if (!pf_bar_wait(done, 0)) give_up(TC_SITE_MMA);
        }
    } else if (warp < 2 + TC_DEQ_WARPS) {
        // ---------------- unpacking warps
        const int h = (warp - 2) >> 2, l = 32 * (warp & 3) + lane;   // half of the stage; tensor-memory lane
        const int row = tc_row<MODE>(l);
        const uint32_t ta = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + S::A0 + h * S::A_HALF;
        const uint32_t ring_a = pf_smem(ring);
        for (uint32_t slot = 0, phase = 0, parity = 1;; parity ^= 1, phase ^= ++slot == SLOTS, slot = slot == SLOTS ? 0 : slot) {
            if (!tc_wait_warp(&full[slot], phase, s_abort)) { give_up(TC_SITE_UNPACK); break; }
            if (s_desc[slot].flags & TCS_END) break;
            const uint32_t st = ring_a + slot * SB;
            bool waited = false, ok = true;
            auto put = [&](int b, int t, const uint32_t (&v)[16]) {
                if (!waited) {   // the place of the stage before: only when there is something to store
                    ok = tc_wait_warp<true>(&aempty[h], parity, s_abort);
                    pf_fence_after();
                    waited = true;
                }
                if (ok) tc_tmem_st16(ta + (b * F::TERMS + t) * 16, v);
            };
            auto put_min = [&](const float (&m)[4]) {
                asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(st + S::W + (h * 128 + l) * 16), "f"(m[0]),
                             "f"(m[1]), "f"(m[2]), "f"(m[3])
                             : "memory");
            };
            if (h == 0) F::unpack(st + row * 16, st + (row ^ unit_shift(TY, 1)) * 16, 0, put, put_min);
            else F::unpack(st + row * 16, st + (row ^ unit_shift(TY, 1)) * 16, 1, put, put_min);
            if (!ok) { give_up(TC_SITE_UNPACK); break; }
            tc_tmem_wait_st();
            if (F::MIN) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the minimums
            pf_fence_before();
            __syncwarp();
            if (lane == 0) {
                pf_bar_arrive(&afull[h]);
                pf_bar_arrive(&empty[slot]);
            }
        }
        if (lane == 0) pf_bar_arrive(left);
    } else {
        // ---------------- epilogue warps
        const int quad = warp & 3, tq = (warp - 2 - TC_DEQ_WARPS) >> 2;   // 32 lanes of tensor memory; part of the tokens
        const int g = lane >> 2, c = lane & 3;
        int rows[4];
#pragma unroll
        for (int r = 0; r < 4; r++) rows[r] = tc_row<MODE>(32 * quad + 8 * r + g);
        const uint32_t tlane = tmem + ((uint32_t)(32 * quad) << 16);
        const uint32_t ring_a = pf_smem(ring);
        const int et = tid - 32 * (2 + TC_DEQ_WARPS);         // thread of the epilogue
        f32x2 acc[4][JMAX];
        bool gave_up = true;
        for (uint32_t slot = 0, phase = 0;; phase ^= ++slot == SLOTS, slot = slot == SLOTS ? 0 : slot) {
            if (!tc_wait_warp(&full[slot], phase, s_abort)) { give_up(TC_SITE_EPILOGUE); break; }
            const TcStage d = s_desc[slot];
            if (d.flags & TCS_END) { gave_up = false; break; }
            if (d.flags & TCS_FIRST) {
#pragma unroll
                for (int r = 0; r < 4; r++)
#pragma unroll
                    for (int j = 0; j < JMAX; j++) acc[r][j] = 0ull;
            }
            const uint32_t st = ring_a + slot * SB, x = st + S::W + S::M;
            // the warp's octets: two of up to eight, or one
            const bool two = d.tc > 32;
            const int oct = two ? 2 * tq : tq;
            bool ok;
            if (two) ok = tc_epi_stage<TY, 64, JMAX>(acc, tlane, st, x, rows, oct, lane, dfull, dempty, s_abort);
            else if (d.tc > 16) ok = tc_epi_stage<TY, 32, JMAX>(acc, tlane, st, x, rows, oct, lane, dfull, dempty, s_abort);
            else ok = tc_epi_stage<TY, 16, JMAX>(acc, tlane, st, x, rows, oct, lane, dfull, dempty, s_abort);
            if (!ok) { give_up(TC_SITE_EPILOGUE); break; }
            __syncwarp();
            if (lane == 0) pf_bar_arrive(&empty[slot]);
            if (!(d.flags & TCS_LAST)) continue;

            // ---- the chunk is complete
            if (MODE == TC_GATEUP) {
                // SwiGLU into the staging tile [token][64 rows of the chunk]: rows 0 and 2 of the thread are gate
                // rows, 1 and 3 the up rows of the same outputs
#pragma unroll
                for (int j = 0; j < JMAX; j++) {
                    if ((j > 0 && !two) || 8 * (oct + j) >= d.tc) break;
#pragma unroll
                    for (int o = 0; o < 2; o++)
#pragma unroll
                        for (int tt = 0; tt < 2; tt++) {
                            // ops.rs:160-167: silu(x) = x * (1 / (1 + exp(-x)))
                            const float gt = tt ? hi_of(acc[2 * o][j]) : lo_of(acc[2 * o][j]);
                            const float u = tt ? hi_of(acc[2 * o + 1][j]) : lo_of(acc[2 * o + 1][j]);
                            s_mid[(8 * (oct + j) + 2 * c + tt) * TC_MID_STRIDE + row_of_place(TY, rows[2 * o])] = (gt * __fdiv_rn(1.0f, 1.0f + expf(-gt))) * u;
                        }
                }
                tc_epi_sync();
                // rows of mid: f32 (slice-major by 64) and, for quantised down types, the Q8Act of
                // each 32-row block (quant.rs:368-394): eight rows a thread, four threads a block
                const int u = et & 7;
                for (int tb = 0; tb < d.tc; tb += TC_EPI_WARPS * 4) {
                    const int t = tb + (et >> 3);
                    if (tb + ((et >> 5) << 2) >= d.tc) continue;   // a warp has four tokens: whole warps
                    const float* sv = s_mid + min(t, d.tc - 1) * TC_MID_STRIDE + 8 * u;
                    const float4 a = *(const float4*)sv, b = *(const float4*)(sv + 4);
                    const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
                    const size_t pos = (size_t)d.pos0 + t;
                    const int r = d.chunk * CH + 8 * u;
                    uint32_t q0, q1;
                    float dd, ss;
                    quantize_eight(v, q0, q1, dd, ss);
                    if (t >= d.tc) continue;
                    float* mid = A.out + ((size_t)(r / 64) * A.act_rows + pos) * 64 + r % 64;
                    *(float4*)mid = a;
                    *(float4*)(mid + 4) = b;
                    put_half_record(A.out_t + ((size_t)(r / 256) * (A.act_rows / 8) + pos / 8) * kHalfRec, (int)(pos % 8), r % 256, et & 3,
                                    half_unit(q0, q1), dd, ss);
                }
                tc_epi_sync();   // the staging tile is free for the next chunk
            } else {
                // the thread's four rows are neighbours, and with those of eight lanes 128 bytes of a token's row
                const size_t stride = d.rows;
                float* o = A.out + ((size_t)d.part * A.part_rows + d.pos0) * stride + d.chunk * CH + row_of_place(TY, rows[0]);
#pragma unroll
                for (int j = 0; j < JMAX; j++) {
                    const int t = 8 * (oct + j) + 2 * c;
                    if (j > 0 && !two) break;
                    if (t < d.tc) *(float4*)(o + (size_t)t * stride) = make_float4(lo_of(acc[0][j]), lo_of(acc[1][j]), lo_of(acc[2][j]), lo_of(acc[3][j]));
                    if (t + 1 < d.tc)
                        *(float4*)(o + (size_t)(t + 1) * stride) = make_float4(hi_of(acc[0][j]), hi_of(acc[1][j]), hi_of(acc[2][j]), hi_of(acc[3][j]));
                }
            }
        }
        __syncwarp();
        if (lane == 0) pf_bar_arrive(left);
        if (gave_up) arrive_until_all_left(PfMeeting{1, 32 * TC_EPI_WARPS, left}, kLeaveTurns);
    }
    pf_fence_before();
    __syncthreads();
    pf_fence_after();
    if (warp == 0) {
        __syncwarp();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(*s_tmem), "r"(TC_TMEM_COLS) : "memory");
    }
}

// ---------------------------------------------------------------------------
// host side

template <int TY, int MODE>
static cudaError_t launch_tc_one(const LaunchCfg& c, const TcArgs& A) {
    constexpr int smem = tc_smem<TY, MODE>();
    static_assert(smem <= 227 * 1024, "the block must fit in shared memory");
    static std::atomic<uint64_t> attr_set{0};
    if (cudaError_t e = ensure_dynamic_smem(experts_tc_kernel<TY, MODE>, smem, attr_set)) return e;
    count_launch();
    return launch_after(c.stream, experts_tc_kernel<TY, MODE>, dim3(c.sm_count), dim3(TC_THREADS), smem, A);
}
template <int MODE>
static cudaError_t launch_tc_mode(int ty, const LaunchCfg& c, const TcArgs& A) {
    switch (ty) {
        case BIVMOE_Q4_K: return launch_tc_one<BIVMOE_Q4_K, MODE>(c, A);
        case BIVMOE_Q5_K: return launch_tc_one<BIVMOE_Q5_K, MODE>(c, A);
        case BIVMOE_Q6_K: return launch_tc_one<BIVMOE_Q6_K, MODE>(c, A);
        default: return cudaErrorInvalidValue;
    }
}

// one product (gate+up, or down) over the tile list's groups; `tiles_mode` as in TcArgs
cudaError_t launch_experts_tc(const LaunchCfg& c, bool down, int ty, const DevTiles& w, const DevTiles& sh, const Workspace& ws,
                              int tiles_mode) {
    if (!down && c.gateup_parts > 1) return cudaErrorInvalidValue;   // the parts' SwiGLU writes int8 records
    TcArgs A{};
    A.w = w;
    A.sh = sh;
    A.x_t = down ? ws.mid_t : ws.act_t;
    A.act_rows = ws.act_rows;
    A.out = down ? ws.pair_out : ws.mid;
    A.out_t = down ? nullptr : ws.mid_t;
    A.tile_desc = ws.tile_desc;
    A.n_tiles = ws.n_tiles;
    A.status = ws.status;
    A.n_expert = c.n_expert;
    A.tiles_mode = tiles_mode;
    A.chunks = std::max(w.chunks, sh.chunks);
    A.parts = down ? c.down_parts : 1;
    A.part_rows = c.n;
    if (A.parts > 1) A.out = ws.parts;
    return down ? launch_tc_mode<TC_DOWN>(ty, c, A) : launch_tc_mode<TC_GATEUP>(ty, c, A);
}

}  // namespace bivmoe
