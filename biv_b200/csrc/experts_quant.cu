// Grouped expert products with quantised weights (every block format) or BF16 weights for
// decode-sized groups: gate+up with the SwiGLU and the Q8 re-quantisation (BF16: the three-term
// split) of its output fused, then down.
// Reference: dense_ffn (engine/src/model.rs:1119-1126) over matmul
// (engine/src/ops.rs:84-127) and the per-type dots (engine/src/quant.rs:570-686), for each
// expert's token list (model.rs:875-889) and for the shared expert (model.rs:890-896).
//
// What bounds it: the instructions per weight.  The weights have to come from HBM once, 23
// bytes per clock and SM, i.e. 800 clocks for 128 rows x 256 columns of Q4_K; the four warps
// that work on them should issue less than that.
//
// Design.  One block per SM: G consumer groups of four warps and one producer warp.  A
// group works on its own items - a tile of up to 8 (or 16) tokens of one group times one chunk of
// 128 weight rows (64 gate rows with their 64 up rows, or 128 down rows) - and owns a
// two-slot ring of stages (one K-slice of the chunk plus the tile's activation record)
// that lane g of the producer warp keeps full with bulk copies: the lane takes the group's
// next item from the block's own list - item i of a launch belongs to block i mod
// gridDim.x, so every SM gets the same number of (equal) items give or take one, and the
// groups of a block share its list through a counter in shared memory - and issues its
// stages as slots come free.  A consumer warp waits for a slot, computes its 32 rows of
// the stage, and hands the slot back with one mbarrier arrive: the consumer warps never
// meet per stage and carry no pipeline state - everything a stage needs to know (tile,
// chunk, whether it opens or closes an accumulation) comes in a small descriptor the
// producer writes beside it.  The groups of a block share nothing but the producer warp,
// so one group's epilogue overlaps the others' products.  The producer lanes never block:
// they stay together and poll their groups' slots in turn.
// Each 32-element block dot is an int8 tensor-core product (mma.sync m16n8k32, 16 weight
// rows x 8 tokens): its int32 results are the reference's block dots, scaled in f32 by the
// weight block scale and the activation block scale.
// What keeps the instruction count down (589 warp instructions per 32 rows and stage of
// Q4_K before, 460 now; 64 tokens Q4_K, gate+up, 36 -> 31 us, 160 tokens Q5_K / Q6_K 90 -> 75
// and 58 -> 48 us):
//   * a lane's fragments are 8-byte pieces: the K order inside a block is permuted alike for
//     both operands (lane c of a row holds bytes 8c .. 8c+7 of the block's 32), and the rows of
//     odd units lie four places on (common.cuh), which keeps those loads free of bank conflicts;
//   * the block scales of a row are unpacked and converted by ONE lane - lane l does row l of the
//     warp's 32 - and go to the four lanes that need them through shared memory, four rows'
//     scales of a block in one load (what that load brings is what counts: shared memory is
//     the busiest unit; as (s, s) pairs for two tokens at a time they kept it 72 % busy);
//   * where groups are large enough a tile has 16 tokens (k-quants): a stage's weights and
//     scales are unpacked once for both records, 670 instructions instead of 2 x 460 - with
//     three groups a block instead of four, for shared memory (Q6_K two instead of three).
//     509 tokens Q4_K / Q6_K 141 + 106 -> 136 + 91 us, 4096 skewed tokens Q4_K, the pass,
//     1.65 -> 1.38 ms;
//   * the accumulator input of the MMA is the bit pattern of 1.5*2^23, so the int32 result read
//     as f32 is 12582912 + dot and one f32 subtraction replaces an int->float conversion;
//   * Q4_K's high nibbles stay in place as unsigned bytes worth 16 times their value, Q6_K's
//     bytes are 4 (q - 32): the exact powers of two go into the scales;
//   * the min term sum m*s_x of Q4_K, Q5_K and Q4_1 is a 16x8x8 tf32 MMA, exact because m has
//     at most 11 significant bits and s_x is stored as two tf32-exact halves.
// BF16 weights keep the structure: a stage is 64 columns and a record of the tokens' three
// bf16 terms, x = hi + mid + lo exactly, so the products are those of the f32 activations; 24
// m16n8k16 MMAs and 14 ldmatrix per 32 rows and stage leave the kernel to HBM.  (Multiplied
// out in f32 on the CUDA cores, 8 tokens a weight, 33 tokens over 256 experts took 193 + 89 us;
// so 117 + 57, 5.8 TB/s.)
// (Two other forms were measured at 64 tokens Q4_K, gate+up: tcgen05.mma kind::i8 with the
// weights as M = 128, 63 us - the spread int8 operand passes through shared memory twice,
// and a stage crosses five barriers; and fragments loaded from global memory straight into
// registers, 50 us - what has to be in flight does not fit beside the rest in 128 registers.)
// Every mbarrier wait is bounded; a wait that gives up records BIVMOE_ERR_TIMEOUT (and which
// wait it was) in the status words and raises a block-wide flag on which every role leaves
// its loop (the producer first waits, bounded again, for its copies still in flight).
// No atomics on data: results are run-to-run identical.
#include <cuda_fp16.h>

#include <algorithm>

#include "common.cuh"
#include "formats.cuh"
#include "tcgen05.cuh"
#include "topk.cuh"
#include "launch.cuh"

namespace bivmoe {

enum { EQ_GATEUP = 0, EQ_DOWN = 1 };
constexpr int EQ_TT = kQuantTile;         // tokens per record; a tile has one or two
constexpr int EQ_SLOTS = 2;               // ring slots per group
constexpr int EQ_HEAD = 1024;             // barriers, abort flag, stage descriptors
// what the products read of a record: all of three terms, all but s of Q8
template <int TY, int NT = 1> __host__ __device__ constexpr int eq_x_bytes() { return TY == BIVMOE_BF16 ? kAct3Rec : (NT - 1) * kActTileBytes + kActOffS; }
static_assert(kAct3Rec == kActTileBytes, "both kinds of records lie equally far apart");

struct QuantArgs {
    DevTiles w, sh;        // the routed experts' and the shared expert's tiles for this product
    const uint8_t* x_t;    // Q8 records of the inputs by position, [K/256][R/8]
    int act_rows;          // R
    float* out;            // GATEUP: mid f32 slice-major; DOWN: pair_out [R][rows]
    uint8_t* out_t;        // GATEUP with a quantised down type: Q8 records of mid; BF16: its three-term records
    const int4* tile_desc; // {expert (n_expert: shared), first position, tokens, 0 or the rows wanted (a bit each)}
    const int32_t* n_tiles;
    int32_t* status;
    int n_expert;
    int tiles_mode;        // 0: every tile, 1: skip the shared group's, 2: only the shared group's
    int chunks;            // row chunks per group in this launch
    int parts;             // K is cut into this many parts, a work item each (1: not cut) ...
    int part_rows;         // ... whose sums go to out as [part][part_rows][rows], a gate row before its up row
};

__device__ __forceinline__ float ldsf(uint32_t a) { return __uint_as_float(lds32(a)); }
__device__ __forceinline__ uint2 lds64(uint32_t a) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
    return v;
}
__device__ __forceinline__ void sts_f4(uint32_t a, float x, float y, float z, float w) {
    asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(a), "f"(x), "f"(y), "f"(z), "f"(w) : "memory");
}

// D[16x8] = A[16x32] * B[32x8] + 1.5 * 2^23 in the integer's bits, with u8 or s8 A and s8 B;
// lane (g = lane / 4, c = lane % 4) holds A: a0 (row g), a1 (row g + 8) of four K values, a2, a3
// of four more, B: b0, b1 the same K values of column g, D: row g columns 2c, 2c + 1, then row
// g + 8.  The int32 result read as an f32 is 12582912 + sum exactly (|sum| < 2^22), so one
// subtraction on the multiply-add pipe gives float(sum), two columns at a time.
template <bool SIGNED>
__device__ __forceinline__ void mma_dots(f32x2 (&dot)[2], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                         uint32_t b0, uint32_t b1) {
    int d[4];
    if (SIGNED)
        asm volatile(
            "mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
            "{%10,%10,%10,%10};"
            : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0x4B400000));
    else
        asm volatile(
            "mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
            "{%10,%10,%10,%10};"
            : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0x4B400000));
    const f32x2 neg = pk(-12582912.0f, -12582912.0f);
    dot[0] = add2(pk(__int_as_float(d[0]), __int_as_float(d[1])), neg);
    dot[1] = add2(pk(__int_as_float(d[2]), __int_as_float(d[3])), neg);
}
// D[16x8] += A[16x8] * B[8x8] in tf32 with f32 accumulation.  a0 (row g, k c), a1 (row g+8, k c),
// a2 (row g, k c+4), a3 (row g+8, k c+4); b0 (k c, column g), b1 (k c+4, column g); D as above.
__device__ __forceinline__ void mma_tf32_k8(float (&d)[4], const float (&a)[4], float b0, float b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(__float_as_uint(a[0])), "r"(__float_as_uint(a[1])), "r"(__float_as_uint(a[2])),
          "r"(__float_as_uint(a[3])), "r"(__float_as_uint(b0)), "r"(__float_as_uint(b1)));
}

__device__ __forceinline__ float half_at(const uint4& v, int i) {   // f16 i of a unit's eight
    const uint32_t w = (i & 4) ? ((i & 2) ? v.w : v.z) : ((i & 2) ? v.y : v.x);
    return __half2float(__ushort_as_half((unsigned short)(w >> (16 * (i & 1)))));
}

// What a warp needs to know about a type.  Its 32 rows of a stage are two 16-row MMA tiles;
//   G          consumer groups per block (what fits in shared memory and registers)
//   bytes(w, b, a)   the two words of block b: w[0], w[1] are the lane's pieces of one row, in shared
//              memory: `at` + constants, unit u 2048 u further
//   scales(hdr...)   the scales of row `lane`
template <int TY> struct Fmt;

// ---- Q4_K / Q5_K (quant.rs:609-649): per sub-block d*sc*d_x*sum(q*q_x) - dmin*m*s_x; Q5_K
//      adds bit b of qh[l] as value bit 4
template <int TY> struct FmtK45 {
    static constexpr int G = 4, HDR = 0;
    static constexpr bool MIN = true, SIGNED = false, HALVES = false, NIBBLE16 = false;
    static constexpr int FACTORS = 2;                       // d and dmin, applied once per stage
    static constexpr int QU = TY == BIVMOE_Q4_K ? 1 : 3;    // unit of the first quants
    static constexpr int ODD = 1;                           // a 32-byte group starts at an odd unit
    struct Row { uint2 qh; };                               // what stays in registers over the stage
    static __device__ __forceinline__ void row(Row& R, uint32_t at) {
        if (TY == BIVMOE_Q5_K) R.qh = lds64(at + 2048);
    }
    struct Group { uint2 w; };                              // blocks 2j (low nibbles) and 2j + 1 (high nibbles)
    static __device__ __forceinline__ void group(Group& W, uint32_t at, int j) { W.w = lds64(at + (QU + 2 * j) * 2048); }
    static __device__ __forceinline__ void bytes(const Row& R, const Group& W, int b, uint32_t (&a)[2]) {
        const uint32_t ww[2] = {W.w.x, W.w.y};
#pragma unroll
        for (int i = 0; i < 2; i++) {
            if (TY == BIVMOE_Q4_K) {
                a[i] = ww[i] & (b & 1 ? 0xF0F0F0F0u : 0x0F0F0F0Fu);
            } else {
                const uint32_t hb = i ? R.qh.y : R.qh.x;
                const uint32_t bit = b <= 4 ? hb << (4 - b) : hb >> (b - 4);
                a[i] = ((b & 1 ? ww[i] >> 4 : ww[i]) & 0x0F0F0F0Fu) | (bit & 0x10101010u);
            }
        }
    }
    struct Own { float d, f; K4Scales k; };
    static __device__ __forceinline__ void own(Own& O, uint32_t at, uint32_t) {
        const uint4 v = lds128(at);
        const __half2 dd = *(const __half2*)&v.x;
        O.d = __low2float(dd);
        O.f = __high2float(dd);
        O.k = unpack_k4_scales(v.y, v.z, v.w);
    }
    // float(byte i) * f for a power of two f: the byte as the low mantissa bits of 2^23, then one
    // multiply-add takes 2^23 f off again (a conversion instruction has an eighth of the rate)
    static __device__ __forceinline__ float scaled(uint32_t w, int i, float f) {
        return fmaf(__uint_as_float(__byte_perm(w, 0x4B000000u, 0x7540 + i)), f, f * -8388608.0f);
    }
    static __device__ __forceinline__ float scale(const Own& O, int b) {
        return scaled(b < 4 ? O.k.sc_lo : O.k.sc_hi, b & 3, TY == BIVMOE_Q4_K && (b & 1) ? 0.0625f : 1.0f);
    }
    static __device__ __forceinline__ float minimum(const Own& O, int b) {
        return scaled(b < 4 ? O.k.m_lo : O.k.m_hi, b & 3, 1.0f);
    }
};
template <> struct Fmt<BIVMOE_Q4_K> : FmtK45<BIVMOE_Q4_K> {};
template <> struct Fmt<BIVMOE_Q5_K> : FmtK45<BIVMOE_Q5_K> {};

// ---- Q8_0 (quant.rs:599-607): term = d_w * d_x * sum(q_w * q_x)
template <> struct Fmt<BIVMOE_Q8_0> {
    static constexpr int G = 2, HDR = 16, ODD = 0;
    static constexpr bool MIN = false, SIGNED = true, HALVES = false, NIBBLE16 = false;
    static constexpr int FACTORS = 0;
    struct Row {};
    static __device__ __forceinline__ void row(Row&, uint32_t) {}
    struct Group { uint2 w[2]; };
    static __device__ __forceinline__ void group(Group& W, uint32_t at, int j) {
        W.w[0] = lds64(at + (4 * j) * 2048);
        W.w[1] = lds64(at + (4 * j + 2) * 2048);
    }
    static __device__ __forceinline__ void bytes(const Row&, const Group& W, int b, uint32_t (&a)[2]) {
        a[0] = W.w[b & 1].x;
        a[1] = W.w[b & 1].y;
    }
    struct Own { uint4 h; float d, f; };
    static __device__ __forceinline__ void own(Own& O, uint32_t at, uint32_t) { O.h = lds128(at); }
    static __device__ __forceinline__ float scale(const Own& O, int b) { return half_at(O.h, b); }
    static __device__ __forceinline__ float minimum(const Own&, int) { return 0.0f; }
};

// ---- Q6_K (quant.rs:651-686), slice = ql[128] qh[64] scales[16], then the rows' d: per
//      32-block d * d_x * (sc[2b]*sum16 + sc[2b+1]*sum16), 6-bit values minus 32.  The bytes
//      are 4 (q - 32) = (4 q) ^ 0x80 as int8, the exact 1/4 goes into d.
template <> struct Fmt<BIVMOE_Q6_K> {
    static constexpr int G = 3, HDR = 12, ODD = 0;
    static constexpr bool MIN = false, SIGNED = true, HALVES = true, NIBBLE16 = false;
    static constexpr int FACTORS = 1;                       // d
    struct Row { uint2 qh[2]; };   // of the 128-value halves
    static __device__ __forceinline__ void row(Row& R, uint32_t at) {
        R.qh[0] = lds64(at + 8 * 2048);
        R.qh[1] = lds64(at + 10 * 2048);
    }
    // groups are (half n, parity): blocks 4n + par (low nibbles) and 4n + par + 2 (high)
    struct Group { uint2 w; };
    static __device__ __forceinline__ void group(Group& W, uint32_t at, int j) { W.w = lds64(at + 2 * j * 2048); }
    static __device__ __forceinline__ void bytes(const Row& R, const Group& W, int b, uint32_t (&a)[2]) {
        const int kq = b & 3;
        const uint2 h2 = R.qh[b >> 2];
        const uint32_t lw[2] = {W.w.x, W.w.y}, hw[2] = {h2.x, h2.y};
#pragma unroll
        for (int i = 0; i < 2; i++)
            a[i] = ((kq < 2 ? lw[i] << 2 : lw[i] >> 2) & 0x3C3C3C3Cu) | (((hw[i] << (6 - 2 * kq)) & 0xC0C0C0C0u) ^ 0x80808080u);
    }
    struct Own { uint4 s; float d, f; };
    static __device__ __forceinline__ void own(Own& O, uint32_t at, uint32_t d_at) {
        O.s = lds128(at);
        unsigned short h;
        asm volatile("ld.shared.u16 %0, [%1];" : "=h"(h) : "r"(d_at));
        O.d = __half2float(__ushort_as_half(h)) * 0.25f;
    }
    static __device__ __forceinline__ float scale(const Own& O, int i) {   // of sub-block i
        const uint32_t w = (i & 8) ? ((i & 4) ? O.s.w : O.s.z) : ((i & 4) ? O.s.y : O.s.x);
        return (float)(int8_t)(w >> (8 * (i & 3)));
    }
    static __device__ __forceinline__ float minimum(const Own&, int) { return 0.0f; }
};

// ---- Q4_0 / Q4_1 (quant.rs:570-597): d * d_x * sum((q - 8) * q_x), d * d_x * sum(q * q_x) + m * s_x.
//      A block's 16 bytes hold element j in the low half of byte j and j + 16 in the high half:
//      a lane's 4 bytes give both halves of the MMA's K.  The nibbles go to the high half of
//      their byte - Q4_0 with bit 3 flipped, which makes the byte the int8 value 16 (q - 8) -
//      and the exact 1/16 into the scale.
template <int TY> struct FmtQ4 {
    static constexpr int G = 4, HDR = 8, ODD = 0;
    static constexpr bool MIN = TY == BIVMOE_Q4_1, SIGNED = TY == BIVMOE_Q4_0, HALVES = false, NIBBLE16 = true;
    static constexpr int FACTORS = 0;
    struct Row {};
    static __device__ __forceinline__ void row(Row&, uint32_t) {}
    struct Group { uint32_t w[2]; };
    static __device__ __forceinline__ void group(Group& W, uint32_t at, int j) {
        W.w[0] = lds32(at + (2 * j) * 2048);
        W.w[1] = lds32(at + (2 * j + 1) * 2048);
    }
    static __device__ __forceinline__ void bytes(const Row&, const Group& W, int b, uint32_t (&a)[2]) {
        constexpr uint32_t flip = TY == BIVMOE_Q4_0 ? 0x80808080u : 0u;
        a[0] = ((W.w[b & 1] << 4) & 0xF0F0F0F0u) ^ flip;
        a[1] = (W.w[b & 1] & 0xF0F0F0F0u) ^ flip;
    }
    struct Own { uint4 h, m; float d, f; };
    static __device__ __forceinline__ void own(Own& O, uint32_t at, uint32_t) {
        O.h = lds128(at);
        if (TY == BIVMOE_Q4_1) O.m = lds128(at + 2048);
    }
    static __device__ __forceinline__ float scale(const Own& O, int b) { return half_at(O.h, b) * 0.0625f; }
    static __device__ __forceinline__ float minimum(const Own& O, int b) { return half_at(O.m, b); }
};
template <> struct Fmt<BIVMOE_Q4_0> : FmtQ4<BIVMOE_Q4_0> {};
template <> struct Fmt<BIVMOE_Q4_1> : FmtQ4<BIVMOE_Q4_1> {};

// A warp's shared scales: a float per row and block (Q6_K: half block), [block][g][4 rows g + 8i],
// so that a lane gets those of its four rows in one load and lane l stores those of row l
// (= 8i + g) without conflicts; then the minimums of the rows [2][32 rows][4], and a factor
// per row, [g][4].
template <> struct Fmt<BIVMOE_BF16> { static constexpr int G = 4; };

template <int TY> struct EqScales {
    using F = Fmt<TY>;
    static constexpr bool OVER = TY == BIVMOE_Q5_K;   // no room beside the rings: the minimums follow in the scales' place
    static constexpr int SCALES = 8 * (F::HALVES ? 2 : 1) * 128, MINS = OVER ? 0 : SCALES;
    static constexpr int FACTOR = SCALES + (F::MIN && !OVER ? 1024 : 0);
    static constexpr int BYTES = FACTOR + F::FACTORS * 128;
};

template <> struct EqScales<BIVMOE_BF16> { static constexpr int BYTES = 0; };

// One stage for one warp: its 32 rows (tile 0: places r0 .. of the chunk, tile 1: r1 ..) against the
// tile's tokens.  acc[i][tt]: token 2c + tt of the row at place 8i + g of the 32.
// Summation: block by block, sum = fma(weight scale, d_x * dot, sum) - the types with a factor
// per super-block or a minimum sum a stage by itself, then acc += d * sum - dmin * minimum
// term; the other kernels for the same types keep this order.
// whether a stage is summed by itself first
template <int TY> __host__ __device__ constexpr bool eq_stage_sum() { return Fmt<TY>::MIN || Fmt<TY>::NIBBLE16; }
template <int TY, int NT>
__device__ __forceinline__ void eq_stage(uint32_t w, uint32_t x, uint32_t ss, int r0, int r1, float (*acc)[4][2], int lane) {
    using F = Fmt<TY>;
    using S = EqScales<TY>;
    const int g = lane >> 2, c = lane & 3;
    // the lane's pieces: of rows with the place shift of odd units (swizzled types)
    const int odd = unit_shift(TY, (F::ODD + (c >> 1)) & 1);
    const uint32_t lp = F::NIBBLE16 ? w + g * 16 + 4 * c : w + (c >> 1) * 2048 + (g ^ odd) * 16 + (c & 1) * 8;
    const uint32_t at[2] = {lp + r0 * 16, lp + r1 * 16};     // rows g; rows g + 8 are 128 bytes on
    const int orow = (lane < 16 ? r0 : r1 - 16) + lane;      // the row whose scales this lane unpacks
    typename F::Own O;
    F::own(O, w + F::HDR * 2048 + orow * 16, w + kChunkRows * 208 + orow * 2);
    typename F::Row R[2][2];
#pragma unroll
    for (int mt = 0; mt < 2; mt++)
#pragma unroll
        for (int r = 0; r < 2; r++) F::row(R[mt][r], at[mt] + 128 * r);
    const uint32_t xq = F::NIBBLE16 ? x + g * 16 + 4 * c : x + (c >> 1) * 128 + g * 16 + (c & 1) * 8;
    const uint32_t xd = x + kActOffDx + 8 * c;               // d_x of tokens 2c, 2c + 1
    const uint32_t srow = ss + g * 16;
    const uint32_t sown = ss + ((lane & 7) * 4 + (lane >> 3)) * 4;
#pragma unroll
    for (int i = 0; i < (F::HALVES ? 16 : 8); i++)
        asm volatile("st.shared.f32 [%0], %1;" ::"r"(sown + i * 128), "f"(F::scale(O, i)) : "memory");
    auto put_minimums = [&]() {
#pragma unroll
        for (int i = 0; i < 2; i++)
            sts_f4(ss + S::MINS + i * 512 + lane * 16, F::minimum(O, 4 * i), F::minimum(O, 4 * i + 1), F::minimum(O, 4 * i + 2),
                   F::minimum(O, 4 * i + 3));
    };
    if (F::MIN && !S::OVER) put_minimums();
    if (F::FACTORS > 0) asm volatile("st.shared.f32 [%0], %1;" ::"r"(sown + S::FACTOR), "f"(O.d) : "memory");
    if (F::FACTORS > 1) asm volatile("st.shared.f32 [%0], %1;" ::"r"(sown + S::FACTOR + 128), "f"(O.f) : "memory");
    __syncwarp();
    // the tokens' words and d_x of a block
    auto tokens = [&](int t, int b, uint2& q, f32x2& dx) {
        if (F::NIBBLE16) {   // K values 4c.. and 16 + 4c.. of token g
            q.x = lds32(xq + t * kActTileBytes + b * 256);
            q.y = lds32(xq + t * kActTileBytes + b * 256 + 128);
        } else {             // K values 8c .. 8c + 7
            q = lds64(xq + t * kActTileBytes + b * 256);
        }
        dx = lds_f2(xd + t * kActTileBytes + b * 32);
    };
    auto at4 = [](const uint4& v, int i) { return __uint_as_float(i & 2 ? (i & 1 ? v.w : v.z) : (i & 1 ? v.y : v.x)); };
    constexpr bool STAGE_SUM = eq_stage_sum<TY>();
    float ts[NT][4][2] = {};
    uint4 fd = make_uint4(0, 0, 0, 0);
    if (F::FACTORS > 0) fd = lds128(srow + S::FACTOR);
#pragma unroll
    for (int j = 0; j < 4; j++) {    // two blocks with common bytes
        typename F::Group W[2][2];
#pragma unroll
        for (int mt = 0; mt < 2; mt++)
#pragma unroll
            for (int r = 0; r < 2; r++) F::group(W[mt][r], at[mt] + 128 * r, j);
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int b = F::HALVES ? 4 * (j >> 1) + (j & 1) + 2 * h : 2 * j + h;
            uint2 q[NT];
            f32x2 dx[NT];
#pragma unroll
            for (int t = 0; t < NT; t++) tokens(t, b, q[t], dx[t]);
            uint4 sv[F::HALVES ? 2 : 1];
#pragma unroll
            for (int i = 0; i < (F::HALVES ? 2 : 1); i++) sv[i] = lds128(srow + ((F::HALVES ? 2 * b : b) + i) * 128);
#pragma unroll
            for (int mt = 0; mt < 2; mt++) {
                uint32_t a[2][2];
#pragma unroll
                for (int r = 0; r < 2; r++) F::bytes(R[mt][r], W[mt][r], b, a[r]);
#pragma unroll
                for (int t = 0; t < NT; t++) {
                    f32x2 d[2];
                    if constexpr (F::HALVES) {
                        // the scales cover 16 elements: lanes c < 2 hold the first half of a block's K
                        // values, the others the second, so each half is an MMA whose B is zero in
                        // the other lanes.  sc0 * dot0 + sc1 * dot1 is an integer below 2^24 times
                        // the 4 of the bytes: exact in f32
                        f32x2 o[2];
                        mma_dots<F::SIGNED>(d, a[0][0], a[1][0], a[0][1], a[1][1], c < 2 ? q[t].x : 0u, c < 2 ? q[t].y : 0u);
                        mma_dots<F::SIGNED>(o, a[0][0], a[1][0], a[0][1], a[1][1], c < 2 ? 0u : q[t].x, c < 2 ? 0u : q[t].y);
#pragma unroll
                        for (int r = 0; r < 2; r++) {
                            const float s0 = at4(sv[0], 2 * mt + r), s1 = at4(sv[1], 2 * mt + r);
                            const f32x2 p = mul2(dx[t], fma2(pk(s1, s1), o[r], mul2(pk(s0, s0), d[r])));
                            float (&to)[2] = acc[t][2 * mt + r];
                            to[0] = fmaf(at4(fd, 2 * mt + r), lo_of(p), to[0]);
                            to[1] = fmaf(at4(fd, 2 * mt + r), hi_of(p), to[1]);
                        }
                    } else {
                        mma_dots<F::SIGNED>(d, a[0][0], a[1][0], a[0][1], a[1][1], q[t].x, q[t].y);
#pragma unroll
                        for (int r = 0; r < 2; r++) {
                            const float s = at4(sv[0], 2 * mt + r);
                            const f32x2 p = mul2(dx[t], d[r]);
                            float (&to)[2] = STAGE_SUM ? ts[t][2 * mt + r] : acc[t][2 * mt + r];
                            to[0] = fmaf(s, lo_of(p), to[0]);
                            to[1] = fmaf(s, hi_of(p), to[1]);
                        }
                    }
                }
            }
        }
    }
    if constexpr (STAGE_SUM) {
        uint4 fm = make_uint4(0, 0, 0, 0);
        if (F::FACTORS > 1) fm = lds128(srow + S::FACTOR + 128);
        if (F::MIN && S::OVER) {
            __syncwarp();
            put_minimums();
            __syncwarp();
        }
        float m[2][4];   // minimums: rows g, g + 8 of block c, then of block c + 4
        if constexpr (F::MIN)
#pragma unroll
            for (int mt = 0; mt < 2; mt++)
#pragma unroll
                for (int i = 0; i < 4; i++)
                    m[mt][i] = ldsf(srow + S::MINS + (i >> 1) * 512 + (mt * 16 + (i & 1) * 8) * 16 + c * 4);
#pragma unroll
        for (int t = 0; t < NT; t++) {
            float tm[4][2] = {};
            if constexpr (F::MIN) {
                float sv[4];
#pragma unroll
                for (int i = 0; i < 4; i++) sv[i] = ldsf(x + t * kActTileBytes + kActOffSHi + g * 16 + c * 4 + i * 128);   // hi: blocks c, c + 4; lo
#pragma unroll
                for (int mt = 0; mt < 2; mt++) {
                    // sum_b m[row][b] * s[token][b], a 16x8x8 product
                    float v[4] = {};
                    mma_tf32_k8(v, m[mt], sv[0], sv[1]);
                    mma_tf32_k8(v, m[mt], sv[2], sv[3]);
#pragma unroll
                    for (int i = 0; i < 4; i++) tm[2 * mt + (i >> 1)][i & 1] = v[i];
                }
            }
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int tt = 0; tt < 2; tt++)
                    acc[t][i][tt] = __fadd_rn(acc[t][i][tt], F::FACTORS > 1 ? fmaf(at4(fd, i), ts[t][i][tt], -__fmul_rn(at4(fm, i), tm[i][tt]))
                                                                            : __fadd_rn(ts[t][i][tt], tm[i][tt]));
        }
    }
    __syncwarp();    // this warp is done with the slot, and with its shared scales
}

// BF16: fragments come by ldmatrix, whose 8 rows of 16 bytes are what lies contiguous in the
// weights and in the records.  The stage is summed by itself (the terms from lo to hi), so the
// tensor core's own accumulation never runs longer than twelve products of 16.
__device__ __forceinline__ void ldmatrix4(uint32_t (&v)[4], uint32_t a) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(a));
}
__device__ __forceinline__ void eq_stage_bf16(uint32_t w, uint32_t x, int r0, int r1, float (&acc)[4][2], int lane) {
    // lane l gives the address of row l % 8 of matrix l / 8: weights (rows 0-7, 8-15) x (two units), tokens four units
    const uint32_t wl = w + (lane >> 4) * 2048 + (lane & 15) * 16, xl = x + (lane >> 3) * 128 + (lane & 7) * 16;
    uint32_t b[3][2][4];   // [term][half of the K-slice]: units 4 half .. + 3, the two of K step 2 half, then of the next
#pragma unroll
    for (int t = 0; t < 3; t++)
#pragma unroll
        for (int i = 0; i < 2; i++) ldmatrix4(b[t][i], xl + t * kAct3Term + i * 512);
#pragma unroll
    for (int mt = 0; mt < 2; mt++) {
        uint32_t a[4][4];
#pragma unroll
        for (int k = 0; k < 4; k++) ldmatrix4(a[k], wl + k * 4096 + (mt ? r1 : r0) * 16);
        float v[4] = {};
#pragma unroll
        for (int t = 2; t >= 0; t--)
#pragma unroll
            for (int k = 0; k < 4; k++)
                asm volatile(
                    "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
                    "{%0,%1,%2,%3};"
                    : "+f"(v[0]), "+f"(v[1]), "+f"(v[2]), "+f"(v[3])
                    : "r"(a[k][0]), "r"(a[k][1]), "r"(a[k][2]), "r"(a[k][3]), "r"(b[t][k >> 1][2 * (k & 1)]),
                      "r"(b[t][k >> 1][2 * (k & 1) + 1]));
#pragma unroll
        for (int i = 0; i < 4; i++) acc[2 * mt + (i >> 1)][i & 1] = __fadd_rn(acc[2 * mt + (i >> 1)][i & 1], v[i]);
    }
    __syncwarp();    // this warp is done with the slot
}

template <int TY, int NT> __host__ __device__ constexpr int eq_stage_bytes() { return slice_stage_bytes(TY) + eq_x_bytes<TY, NT>(); }
// consumer groups: one less where a tile has two records (shared memory, and the registers for
// twice the sums)
template <int TY, int NT> __host__ __device__ constexpr int eq_groups() { return Fmt<TY>::G - (NT - 1); }
template <int TY, int NT> __host__ __device__ constexpr int eq_smem() {
    constexpr int G = eq_groups<TY, NT>();
    return EQ_HEAD + G * NT * EQ_TT * 64 * 4 + G * EQ_SLOTS * eq_stage_bytes<TY, NT>() + 4 * G * EqScales<TY>::BYTES;
}

struct EqStage {        // what the producer tells a group about a stage
    int pos0, tc;       // the tile: first position, tokens
    int chunk, rows;    // chunk of the expert's matrix; its rows (down: the stride of the output rows)
    int flags;          // EQ_*
    int part;
    uint32_t mask;      // the tile's tokens whose rows are wanted
    int pad;
};
enum { EQ_FIRST = 1, EQ_LAST = 2, EQ_END = 4 };
// which bounded wait gave up (status word 2, for the error text)
enum { EQ_SITE_PRODUCER = 11, EQ_SITE_STAGE = 12 };

struct EqItem {         // a decoded work item: a token tile x a chunk
    int chunk, nsl;     // end of its K-slices (none when the matrix has no such chunk)
    int pos0, tc, rows, part;
    uint32_t mask;
    const uint8_t* src; // K-slice 0 of the chunk; the slices follow each other
};

// One look, without blocking: has the phase of parity `parity` completed?
__device__ __forceinline__ bool eq_test_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(pf_smem(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ void group_sync(int grp) {   // the 128 threads of one consumer group
    asm volatile("bar.sync %0, 128;" ::"r"(grp + 1) : "memory");
}
// A consumer warp that gave up arrives at its group's meetings for the others, which leave at their next
// wait: for some 65 ms.  (Counting those that have left took 1 to 5 % of passes of a few tokens.)
__device__ __forceinline__ void group_abandon(int grp) { arrive_until_all_left(PfMeetingForAWhile{grp + 1, 128}, 1u << 16); }

// SwiGLU of a thread's gate rows (places p, p + 8 of the chunk) and up rows into the staging tile [token][64 rows of the chunk]
template <int TY, int NT>
__device__ __forceinline__ void swiglu_tile(const float (&acc)[NT][4][2], float* s_mid, int tc, int p, int c) {
    const int r = row_of_place(TY, p);
    constexpr int NEXT = row_of_place(TY, 8);
#pragma unroll
    for (int t = 0; t < NT; t++) {
        if (8 * t >= tc) break;
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
            for (int tt = 0; tt < 2; tt++) {
                // ops.rs:160-167: silu(x) = x * (1 / (1 + exp(-x)))
                const float gt = acc[t][i][tt], u = acc[t][2 + i][tt];
                s_mid[(8 * t + 2 * c + tt) * 64 + r + NEXT * i] = (gt * __fdiv_rn(1.0f, 1.0f + expf(-gt))) * u;
            }
    }
}
// A warp's 32 values `v` of one SwiGLU row (this lane: output row r): the f32 row and its Q8 record, or
// its three-term record
template <int TY>
__device__ __forceinline__ void store_mid_block(float v, float* out, uint8_t* out_t, int act_rows, int r, size_t pos, int lane) {
    out[((size_t)(r / 64) * act_rows + pos) * 64 + r % 64] = v;
    if (TY == BIVMOE_BF16) {
        uint16_t term[3];
        split_bf16_3(v, term);
        uint8_t* rec = out_t + ((size_t)(r / 64) * (act_rows / 8) + pos / 8) * kAct3Rec + act_b_off((int)(pos % 8), r % 64);
#pragma unroll
        for (int i = 0; i < 3; i++) *(uint16_t*)(rec + i * kAct3Term) = term[i];
    } else if (out_t) {
        float dd, sm;
        const int qv = q8_quantize_lane(v, dd, sm);
        uint8_t* rec = out_t + ((size_t)(r / 256) * (act_rows / 8) + pos / 8) * kActTileBytes;
        rec[act_q_off((int)(pos % 8), r % 256)] = (uint8_t)(int8_t)qv;
        if (lane < 4) {
            float shi, slo;
            split_tf32(sm, &shi, &slo);
            const float val = lane == 0 ? dd : lane == 1 ? shi : lane == 2 ? slo : sm;
            *(float*)(rec + act_scale_off(lane, (r % 256) / 32, (int)(pos % 8))) = val;
        }
    }
}

// NT: 8-token records per tile
template <int TY, int MODE, int NT>
__global__ void __launch_bounds__(32 * (4 * eq_groups<TY, NT>() + 1), 1)
experts_quant_kernel(const QuantArgs A) {
    constexpr int G = eq_groups<TY, NT>(), SB = eq_stage_bytes<TY, NT>();
    constexpr uint32_t W_BYTES = slice_stage_bytes(TY);
    constexpr int CH = MODE == EQ_GATEUP ? 64 : 128;   // output rows per chunk
    pdl_launch_dependents();
    extern __shared__ __align__(128) uint8_t smem[];
    uint64_t* full = (uint64_t*)smem;                 // [G][2] a stage has landed
    uint64_t* empty = full + G * EQ_SLOTS;            // [G][2] its four warps are done with it
    int* s_abort = (int*)(smem + 256);
    int* s_next = (int*)(smem + 260);                 // the block's next unclaimed item (index in its list)
    EqStage* s_desc = (EqStage*)(smem + 512);         // [G][2]
    float* s_mid_all = (float*)(smem + EQ_HEAD);      // [G][8 NT][64] SwiGLU staging
    uint8_t* ring = (uint8_t*)(s_mid_all + G * NT * EQ_TT * 64);   // [G][2][SB]
    uint8_t* s_scales = ring + G * EQ_SLOTS * SB;     // [4 G] the warps' shared scales
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

    if (tid == 0) {
        for (int i = 0; i < G * EQ_SLOTS; i++) {
            pf_bar_init(&full[i], 1);
            pf_bar_init(&empty[i], 4);
        }
        *s_abort = 0;
        *s_next = G;   // the first G items of the list are the groups' first items
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    pdl_wait();   // the tile lists and the activation records are the previous kernels'

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
        const int units = (tile_hi - tile_lo) * A.chunks * A.parts;
        // The lanes stay together: every turn of the loop each lane looks once (without
        // blocking) whether its group has a free slot and, if so, issues its next stage, so
        // no group waits for another lane's wait to end.  A turn without progress in any
        // lane sleeps 64 ns; 2^20 such turns in a row (about 70 ms) end the kernel.
        constexpr uint32_t LANES = (1u << G) - 1u;
        uint32_t issued = 0;      // stages this lane has given its group
        EqItem it;
        it.nsl = 0;
        int slice = 0, from = 0;  // next K-slice of the lane's item; its first one
        int first = 1, ending = 0, done = 0;
        uint32_t idle = 0;
        while (true) {
            int progressed = 0;
            if (!done && !ending && slice >= it.nsl) {
                // the block's list: items blockIdx.x, blockIdx.x + gridDim.x, ...; group g
                // starts with entry g, later entries go to whichever group is ready first
                const int entry = first ? lane : atomicAdd(s_next, 1);
                first = 0;
                const int idx = (int)blockIdx.x + entry * (int)gridDim.x;
                if (idx >= units) {
                    ending = 1;
                } else {
                    it.part = idx % A.parts;
                    const int rest = idx / A.parts;
                    it.chunk = rest % A.chunks;
                    const int4 td = A.tile_desc[tile_lo + rest / A.chunks];
                    const bool shared = td.x == A.n_expert;
                    it.pos0 = td.y;
                    it.tc = td.z;
                    it.mask = td.w ? (uint32_t)td.w : 0xffffffffu;
                    const DevTiles& m = shared ? A.sh : A.w;
                    const int nsl = it.chunk < m.chunks ? m.nslices : 0;
                    from = nsl * it.part / A.parts;
                    it.nsl = nsl * (it.part + 1) / A.parts;
                    it.rows = m.rows;
                    it.src = m.stage(shared ? 0 : td.x, min(it.chunk, max(m.chunks - 1, 0)), 0);
                    slice = from;
                }
                progressed = 1;
            }
            if (!done && (ending || slice < it.nsl)) {
                const int bi = lane * EQ_SLOTS + (int)(issued & 1);
                if (eq_test_wait(&empty[bi], ((issued >> 1) & 1) ^ 1)) {
                    EqStage d{};
                    if (ending) {   // the end marker: a stage without data
                        d.flags = EQ_END;
                        s_desc[bi] = d;
                        pf_bar_arrive(&full[bi]);
                        done = 1;
                    } else {
                        d.pos0 = it.pos0; d.tc = it.tc; d.chunk = it.chunk; d.rows = it.rows;
                        d.part = it.part;
                        d.mask = it.mask;
                        d.flags = (slice == from ? EQ_FIRST : 0) | (slice == it.nsl - 1 ? EQ_LAST : 0);
                        s_desc[bi] = d;
                        uint8_t* dst = ring + (size_t)bi * SB;
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the slot was last read through the generic proxy
                        // the tile's records of this K-slice (pos0 is a multiple of 8)
                        const uint32_t x_bytes = NT > 1 && it.tc > 8 ? eq_x_bytes<TY, NT>() : eq_x_bytes<TY>();
                        pf_bar_expect_tx(&full[bi], W_BYTES + x_bytes);
                        pf_bulk_g2s(dst, it.src + (size_t)slice * W_BYTES, W_BYTES, &full[bi]);
                        pf_bulk_g2s(dst + W_BYTES, A.x_t + ((size_t)slice * (A.act_rows / 8) + it.pos0 / 8) * kActTileBytes,
                                    x_bytes, &full[bi]);
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
                if (lane == 0) give_up(EQ_SITE_PRODUCER);
                break;
            } else {
                __nanosleep(64);
            }
        }
        // leave no copy in flight behind, whoever gave up on it: the last two stages this lane issued, or
        // the last one (the end marker took the other's slot)
        for (uint32_t in_flight = done ? 1 : 2, q = issued > in_flight ? issued - in_flight : 0; q < issued; q++)
            pf_bar_wait(&full[lane * EQ_SLOTS + (q & 1)], (q >> 1) & 1);
        return;
    }

    // ---------------------------------------------------------------- consumer groups
    const int grp = warp >> 2, wig = warp & 3;
    const int g = lane >> 2, c = lane & 3;
    const uint32_t ring_a = pf_smem(ring);
    float* s_mid = s_mid_all + grp * NT * EQ_TT * 64;
    const uint32_t ss = pf_smem(s_scales + warp * EqScales<TY>::BYTES);
    // the first places of this warp's two 16-row MMA tiles: GATEUP gate rows' 16w .. and the
    // same up rows' (64 further), DOWN 32w ..
    const int r0 = MODE == EQ_GATEUP ? 16 * wig : 32 * wig, r1 = MODE == EQ_GATEUP ? 64 + r0 : r0 + 16;
    float acc[NT][4][2] = {};   // [t][i][tt]: token 8t + 2c + tt of the row at place 8i + g of the warp's 32
    for (uint32_t q = 0;; q++) {
        const int bi = grp * EQ_SLOTS + (int)(q & 1);
        if (!pf_bar_wait(&full[bi], (q >> 1) & 1, s_abort)) {
            give_up(EQ_SITE_STAGE);
            if (MODE == EQ_GATEUP) group_abandon(grp);   // (down has no meetings)
            return;
        }
        const EqStage d = s_desc[bi];
        if (d.flags & EQ_END) return;
        if (d.flags & EQ_FIRST) {
#pragma unroll
            for (int i = 0; i < 8 * NT; i++) (&acc[0][0][0])[i] = 0.0f;
        }
        const uint32_t sta = ring_a + (uint32_t)bi * SB;
        if constexpr (TY == BIVMOE_BF16) eq_stage_bf16(sta, sta + W_BYTES, r0, r1, acc[0], lane);
        else if (NT > 1 && d.tc > 8) eq_stage<TY, NT>(sta, sta + W_BYTES, ss, r0, r1, acc, lane);
        else eq_stage<TY, 1>(sta, sta + W_BYTES, ss, r0, r1, acc, lane);
        if (lane == 0) pf_bar_arrive(&empty[bi]);
        if (!(d.flags & EQ_LAST)) continue;

        // ---- the chunk is complete
        if (MODE == EQ_DOWN || A.parts > 1) {
            // The sums, or a part's for the kernel that adds the parts; of gate+up the gate row, then
            // the up row that the up matrix has in that place.
            constexpr int NEXT = row_of_place(TY, 8);
            const size_t stride = (MODE == EQ_GATEUP ? 2 : 1) * d.rows;
            float* first = A.out + ((size_t)d.part * A.part_rows + d.pos0 + 2 * c) * stride + d.chunk * CH + row_of_place(TY, r0 + g);
#pragma unroll
            for (int t = 0; t < NT; t++)
#pragma unroll
                for (int tt = 0; tt < 2; tt++) {
                    const int tok = 8 * t + 2 * c + tt;
                    if (tok >= d.tc || !(d.mask >> tok & 1)) continue;
                    float* o = first + (8 * t + tt) * stride;
                    const float v[4] = {acc[t][0][tt], acc[t][1][tt], acc[t][2][tt], acc[t][3][tt]};
                    if constexpr (MODE == EQ_DOWN && NEXT == 1) {
                        *(float4*)o = make_float4(v[0], v[1], v[2], v[3]);
                    } else if constexpr (NEXT == 1) {
                        *(float2*)o = make_float2(v[0], v[1]);
                        *(float2*)(o + d.rows) = make_float2(v[2], v[3]);
                    } else {
#pragma unroll
                        for (int i = 0; i < 4; i++) o[MODE == EQ_GATEUP ? (i >> 1) * d.rows + NEXT * (i & 1) : NEXT * i] = v[i];
                    }
                }
        } else {
            swiglu_tile<TY, NT>(acc, s_mid, d.tc, 16 * wig + g, c);
            group_sync(grp);
            // rows of mid: f32 (slice-major by 64) and, for quantised down types, the
            // Q8Act of each 32-row block (quant.rs:368-394); one warp per (token, block)
            for (int p = wig; p < 2 * d.tc; p += 4)
                store_mid_block<TY>(s_mid[(p >> 1) * 64 + 32 * (p & 1) + lane], A.out, A.out_t, A.act_rows, d.chunk * CH + 32 * (p & 1) + lane,
                                    (size_t)d.pos0 + (p >> 1), lane);
            group_sync(grp);   // the staging tile is free for the group's next chunk
        }
    }
}

// ---------------------------------------------------------------------------
// A few tokens (up to 8): top-k, the lists, the quantiser and the gate+up product in one launch.
// With the router's logits there every block finds the selected experts by itself, a warp per
// token, while the other warps quantise the rows into the block's own shared memory - one record
// per K-slice for all tokens.  An expert's tile is all the tokens, whichever of them selected
// it: the products cost the same, nothing has to be sorted, gathered or laid out, and only the
// wanted rows are stored.  Positions: expert number s of the list has 8 s + token (after the shared
// expert's eight).  Block 0 leaves the routing result and the tile list for the kernels that follow
// and for the taps.
// What bounds it: a chain of latencies - top-k, then the weights' way from HBM.  One token of 2048 /
// 512, 256 experts, Q4_K: with top-k and sort, dispatch and gate+up as three launches a pass took
// 28.7 us, with this kernel 24.0, with an item's K-slices dealt to the groups (below) 20.9.
constexpr int FEW_TOKENS = 8, FEW_EXPERTS = 256, FEW_K = 32;
constexpr int FEW_SLOTS_MAX = FEW_TOKENS * FEW_K + 1;

struct FewArgs {
    DevTiles w, sh;
    Workspace ws;
    const float* norm_w;   // the rows are the residual: h = x * (row_scale * w), rms_norm on the fly
    int n, k, e, n_expert, has_shared, chunks;
};

template <int TY> __host__ __device__ constexpr int few_ring_bytes() { return Fmt<TY>::G * EQ_SLOTS * slice_stage_bytes(TY); }
constexpr int few_x_bytes(int e) { return e / 256 * kActOffS; }
constexpr int FEW_SMEM_MAX = 227 * 1024 - 2560;   // the lists are static
template <int TY> constexpr int few_smem(int e) {
    return EQ_HEAD + few_ring_bytes<TY>() + 4 * Fmt<TY>::G * EqScales<TY>::BYTES + few_x_bytes(e);
}

template <int TY>
__global__ void __launch_bounds__(32 * (4 * Fmt<TY>::G + 1), 1)
experts_few_kernel(const float* __restrict__ h, const FewArgs A) {
    constexpr int G = Fmt<TY>::G, THREADS = 32 * (4 * G + 1);
    constexpr uint32_t W_BYTES = slice_stage_bytes(TY);
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ uint16_t s_slot_expert[FEW_SLOTS_MAX];
    __shared__ uint8_t s_slot_mask[FEW_SLOTS_MAX];
    __shared__ uint32_t s_mask[FEW_EXPERTS];          // an expert's tokens
    __shared__ uint16_t s_ids[FEW_TOKENS * FEW_K];
    __shared__ int s_count[FEW_EXPERTS / 32], s_slots, s_unit;
    uint64_t* full = (uint64_t*)smem;                 // [G][2] a stage has landed
    uint64_t* empty = full + G * EQ_SLOTS;            // [G][2] its four warps are done with it
    int* s_abort = (int*)(smem + 256);
    int* s_next = (int*)(smem + 260);
    EqStage* s_desc = (EqStage*)(smem + 512);         // [G][2]
    uint8_t* ring = smem + EQ_HEAD;                   // [G][2][W_BYTES]; until the products start the tokens' probabilities
    uint8_t* s_scales = ring + few_ring_bytes<TY>();
    uint8_t* s_x = s_scales + 4 * G * EqScales<TY>::BYTES;         // [e / 256] records, without their last part
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const Workspace& ws = A.ws;
    pdl_launch_dependents();
    if (tid == 0) {
        for (int i = 0; i < G * EQ_SLOTS; i++) {
            pf_bar_init(&full[i], 1);
            pf_bar_init(&empty[i], 4);
        }
        *s_abort = 0;
        *s_next = G;
        s_unit = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int i = tid; i < FEW_EXPERTS; i += THREADS) s_mask[i] = 0;
    __syncthreads();
    pdl_wait();
    if (warp < A.n) {   // a token a warp
        int id;
        float w;
        topk_token<FEW_EXPERTS / 32>(ws.logits + (size_t)warp * (A.n_expert + 1), (float*)ring + warp * FEW_EXPERTS, A.n_expert, A.k,
                                     lane, id, w);
        if (lane < A.k) {
            s_ids[warp * A.k + lane] = (uint16_t)id;
            atomicOr(&s_mask[id], 1u << warp);
            if (blockIdx.x == 0) {
                ws.ids[warp * A.k + lane] = id;
                ws.weights[warp * A.k + lane] = w;
            }
        }
        __syncwarp();
    }
    // the rows, one K-slice of a token at a time, by whichever warp is free
    const int units = A.n * (A.e / 256);
    while (true) {
        int u = lane == 0 ? atomicAdd(&s_unit, 1) : 0;
        u = __shfl_sync(0xffffffffu, u, 0);
        if (u >= units) break;
        const int t = u % A.n, sl = u / A.n, el = 8 * lane;
        const float* x = h + (size_t)t * A.e + sl * 256 + el;
        float4 a = *(const float4*)x, b = *(const float4*)(x + 4);
        if (A.norm_w) {
            const float s = ws.row_scale[t];
            const float4 wa = *(const float4*)(A.norm_w + sl * 256 + el), wb = *(const float4*)(A.norm_w + sl * 256 + el + 4);
            a.x = __fmul_rn(a.x, __fmul_rn(s, wa.x)); a.y = __fmul_rn(a.y, __fmul_rn(s, wa.y));
            a.z = __fmul_rn(a.z, __fmul_rn(s, wa.z)); a.w = __fmul_rn(a.w, __fmul_rn(s, wa.w));
            b.x = __fmul_rn(b.x, __fmul_rn(s, wb.x)); b.y = __fmul_rn(b.y, __fmul_rn(s, wb.y));
            b.z = __fmul_rn(b.z, __fmul_rn(s, wb.z)); b.w = __fmul_rn(b.w, __fmul_rn(s, wb.w));
        }
        const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        uint32_t w0, w1;
        float dd, ss, shi, slo;
        quantize_eight(v, w0, w1, dd, ss);
        split_tf32(ss, &shi, &slo);
        uint8_t* rec = s_x + sl * kActOffS;
        *(uint2*)(rec + act_q_off(t, el)) = make_uint2(w0, w1);
        const int which = lane & 3;
        const float val = which == 0 ? dd : which == 1 ? shi : which == 2 ? slo : ss;
        if (which < 3) *(float*)(rec + act_scale_off(which, el / 32, t)) = val;
        if (blockIdx.x == 0) {
            uint8_t* keep = ws.act_t + (size_t)sl * (ws.act_rows / 8) * kActTileBytes;
            *(uint2*)(keep + act_q_off(t, el)) = make_uint2(w0, w1);
            *(float*)(keep + act_scale_off(which, el / 32, t)) = val;
        }
    }
    __syncthreads();
    // the selected experts in ascending order, after the shared one
    const int g_sh = A.has_shared;
    uint32_t mask = 0, vote = 0;
    if (warp < FEW_EXPERTS / 32) {
        mask = s_mask[tid];
        vote = __ballot_sync(0xffffffffu, mask != 0);
        if (lane == 0) s_count[warp] = __popc(vote);
    }
    __syncthreads();
    if (warp < FEW_EXPERTS / 32) {
        int slot = g_sh + __popc(vote & ((1u << lane) - 1u));
        for (int i = 0; i < warp; i++) slot += s_count[i];
        if (mask) {
            s_slot_expert[slot] = (uint16_t)tid;
            s_slot_mask[slot] = (uint8_t)mask;
        }
        if (tid == FEW_EXPERTS - 1) s_slots = slot + (mask != 0);
        if (tid == 0 && g_sh) {
            s_slot_expert[0] = (uint16_t)A.n_expert;
            s_slot_mask[0] = (uint8_t)((1u << A.n) - 1u);
        }
        if (blockIdx.x == 0) {
            if (tid < A.n_expert) {
                ws.counts[tid] = __popc(mask);
                ws.offsets[tid] = 8 * slot;
            }
            if (mask) ws.tile_desc[slot] = make_int4(tid, 8 * slot, A.n, (int)mask);
            for (uint32_t m = mask, r = 0; m; m &= m - 1, r++) {   // the pairs in ascending order: their tokens
                const int t = __ffs(m) - 1;
                for (int j = 0; j < A.k; j++)
                    if (s_ids[t * A.k + j] == tid) {
                        ws.order[8 * slot + r] = t * A.k + j;
                        ws.pos_of[t * A.k + j] = 8 * slot + t;
                    }
            }
            if (tid == FEW_EXPERTS - 1) {
                const int all = slot + (mask != 0);
                ws.offsets[A.n_expert] = 8 * all;
                *ws.n_groups = all;
                ws.n_tiles[0] = all;
                ws.n_tiles[1] = g_sh;
                ws.n_ptiles[0] = ws.n_ptiles[1] = 0;
                *ws.big_min = 0;
                if (g_sh) ws.tile_desc[0] = make_int4(A.n_expert, 0, A.n, (int)((1u << A.n) - 1u));
            }
        }
    }
    __syncthreads();

    auto give_up = [&](int site) {
        if (atomicExch(ws.status, BIVMOE_ERR_TIMEOUT) == 0) atomicExch(ws.status + 2, site);
        atomicExch(s_abort, 1);
    };
    const int total = s_slots * A.chunks;
    // With no more items than blocks an item is its block's alone: the groups take its K-slices in
    // turn, each of which is summed by itself anyway, leave the sums where the slice's weights were,
    // and all threads add them up in the slices' order - the same bits as one group by itself.
    constexpr bool CAN_SPLIT = G == 4 && eq_stage_sum<TY>();
    if constexpr (CAN_SPLIT) {
        if (total <= (int)gridDim.x && A.w.nslices <= G * EQ_SLOTS) {
            const int slot = (int)blockIdx.x / A.chunks, chunk = (int)blockIdx.x % A.chunks;
            if ((int)blockIdx.x >= total) return;
            const bool shared = g_sh && slot == 0;
            const DevTiles& m = shared ? A.sh : A.w;
            if (chunk >= m.chunks) return;
            const int nsl = m.nslices;   // of both: the rows' width
            if (warp == 4 * G) {
                if (lane < nsl) {        // slice s: group s % G, its slot s / G
                    const int bi = lane % G * EQ_SLOTS + lane / G;
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the ring held the probabilities
                    pf_bar_expect_tx(&full[bi], W_BYTES);
                    pf_bulk_g2s(ring + (size_t)bi * W_BYTES, m.stage(shared ? 0 : s_slot_expert[slot], chunk, lane), W_BYTES, &full[bi]);
                }
                return;
            }
            const int grp = warp >> 2, wig = warp & 3, g = lane >> 2, c = lane & 3;
            const uint32_t ss = pf_smem(s_scales + warp * EqScales<TY>::BYTES);
            const int r0 = 16 * wig, r1 = 64 + r0;
            bool ok = true;
            for (int i = 0; grp + i * G < nsl; i++) {
                const int bi = grp * EQ_SLOTS + i;
                // (after a wait that gave up the sums are still met for, and thrown away; the copy is waited for
                // once more, so that none is in flight when the block ends)
                if (!pf_bar_wait(&full[bi], 0)) {
                    ok = false;
                    pf_bar_wait(&full[bi], 0);
                }
                float acc[1][4][2] = {};
                eq_stage<TY, 1>(pf_smem(ring) + (uint32_t)bi * W_BYTES, pf_smem(s_x) + (grp + i * G) * kActOffS, ss, r0, r1, acc, lane);
                group_sync(grp);         // the group is done with the weights
                float* part = (float*)(ring + (size_t)bi * W_BYTES) + 2 * c;   // [128 places][8 tokens]
#pragma unroll
                for (int j = 0; j < 4; j++)
                    *(float2*)(part + ((j < 2 ? r0 : r1) + 8 * (j & 1) + g) * 8) = make_float2(acc[0][j][0], acc[0][j][1]);
            }
            if (!ok) give_up(EQ_SITE_STAGE);
            asm volatile("bar.sync %0, %1;" ::"n"(G + 1), "n"(128 * G) : "memory");
            if (*(volatile int*)s_abort) return;
            float* s_mid = (float*)s_scales;   // [8][64]
            {
                const int t = tid & 7, r = tid >> 3;
                float gt = 0.0f, u = 0.0f;
                for (int s = 0; s < nsl; s++) {
                    const float* part = (const float*)(ring + (size_t)(s % G * EQ_SLOTS + s / G) * W_BYTES) + tid;
                    gt = __fadd_rn(gt, part[0]);
                    u = __fadd_rn(u, part[64 * 8]);
                }
                if (t < A.n) s_mid[t * 64 + row_of_place(TY, r)] = (gt * __fdiv_rn(1.0f, 1.0f + expf(-gt))) * u;   // ops.rs:160-167
            }
            asm volatile("bar.sync %0, %1;" ::"n"(G + 1), "n"(128 * G) : "memory");
            static_assert(4 * G >= 2 * FEW_TOKENS, "a warp per token and 32-row block");
            if (warp < 2 * A.n && (s_slot_mask[slot] >> (warp >> 1) & 1))
                store_mid_block<TY>(s_mid[(warp >> 1) * 64 + 32 * (warp & 1) + lane], ws.mid, ws.mid_t,
                                    ws.act_rows, chunk * 64 + 32 * (warp & 1) + lane, (size_t)8 * slot + (warp >> 1), lane);
            return;
        }
    }
    if (warp == 4 * G) {
        // ------------------------------------------------------------ producer warp, as above
        if (lane >= G) return;
        constexpr uint32_t LANES = (1u << G) - 1u;
        uint32_t issued = 0, idle = 0;
        int slice = 0, nsl = 0, first = 1, ending = 0, done = 0;
        EqStage it{};
        const uint8_t* src = nullptr;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the ring held the probabilities
        while (true) {
            int progressed = 0;
            if (!done && !ending && slice >= nsl) {
                const int entry = first ? lane : atomicAdd(s_next, 1);
                first = 0;
                const int idx = (int)blockIdx.x + entry * (int)gridDim.x;
                if (idx >= total) {
                    ending = 1;
                } else {
                    const int slot = idx / A.chunks;
                    it.chunk = idx % A.chunks;
                    const bool shared = g_sh && slot == 0;
                    const DevTiles& m = shared ? A.sh : A.w;
                    nsl = it.chunk < m.chunks ? m.nslices : 0;
                    it.pos0 = 8 * slot;
                    it.mask = s_slot_mask[slot];
                    src = m.stage(shared ? 0 : s_slot_expert[slot], min(it.chunk, max(m.chunks - 1, 0)), 0);
                    slice = 0;
                }
                progressed = 1;
            }
            if (!done && (ending || slice < nsl)) {
                const int bi = lane * EQ_SLOTS + (int)(issued & 1);
                if (eq_test_wait(&empty[bi], ((issued >> 1) & 1) ^ 1)) {
                    if (ending) {
                        EqStage d{};
                        d.flags = EQ_END;
                        s_desc[bi] = d;
                        pf_bar_arrive(&full[bi]);
                        done = 1;
                    } else {
                        it.flags = (slice == 0 ? EQ_FIRST : 0) | (slice == nsl - 1 ? EQ_LAST : 0);
                        it.part = slice;
                        s_desc[bi] = it;
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the slot was last read through the generic proxy
                        pf_bar_expect_tx(&full[bi], W_BYTES);
                        pf_bulk_g2s(ring + (size_t)bi * W_BYTES, src + (size_t)slice * W_BYTES, W_BYTES, &full[bi]);
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
                if (lane == 0) give_up(EQ_SITE_PRODUCER);
                break;
            } else {
                __nanosleep(64);
            }
        }
        for (uint32_t in_flight = done ? 1 : 2, q = issued > in_flight ? issued - in_flight : 0; q < issued; q++)
            pf_bar_wait(&full[lane * EQ_SLOTS + (q & 1)], (q >> 1) & 1);
        return;
    }
    // ---------------------------------------------------------------- consumer groups
    const int grp = warp >> 2, wig = warp & 3;
    const int g = lane >> 2, c = lane & 3;
    const uint32_t ring_a = pf_smem(ring), x_a = pf_smem(s_x);
    float* s_mid = (float*)(s_scales + 4 * grp * EqScales<TY>::BYTES);   // [8][64] SwiGLU staging, where the group's scales were
    static_assert(4 * EqScales<TY>::BYTES >= EQ_TT * 64 * 4, "the staging tile");
    const uint32_t ss = pf_smem(s_scales + warp * EqScales<TY>::BYTES);
    const int r0 = 16 * wig, r1 = 64 + r0;
    float acc[1][4][2] = {};
    for (uint32_t q = 0;; q++) {
        const int bi = grp * EQ_SLOTS + (int)(q & 1);
        if (!pf_bar_wait(&full[bi], (q >> 1) & 1, s_abort)) {
            give_up(EQ_SITE_STAGE);
            group_abandon(grp);
            return;
        }
        const EqStage d = s_desc[bi];
        if (d.flags & EQ_END) return;
        if (d.flags & EQ_FIRST) {
#pragma unroll
            for (int i = 0; i < 8; i++) (&acc[0][0][0])[i] = 0.0f;
        }
        eq_stage<TY, 1>(ring_a + (uint32_t)bi * W_BYTES, x_a + d.part * kActOffS, ss, r0, r1, acc, lane);
        if (lane == 0) pf_bar_arrive(&empty[bi]);
        if (!(d.flags & EQ_LAST)) continue;
        group_sync(grp);
        swiglu_tile<TY, 1>(acc, s_mid, A.n, 16 * wig + g, c);
        group_sync(grp);
        for (int p = wig; p < 2 * A.n; p += 4)
            if (d.mask >> (p >> 1) & 1)
                store_mid_block<TY>(s_mid[(p >> 1) * 64 + 32 * (p & 1) + lane], ws.mid, ws.mid_t, ws.act_rows,
                                    d.chunk * 64 + 32 * (p & 1) + lane, (size_t)d.pos0 + (p >> 1), lane);
        group_sync(grp);   // the staging tile is free for the group's next chunk
    }
}

// ---------------------------------------------------------------------------
// host side

template <int TY, int MODE, int NT = 1>
static cudaError_t launch_quant_one(const LaunchCfg& c, const QuantArgs& A) {
    if constexpr (NT == 1 && (TY == BIVMOE_Q4_K || TY == BIVMOE_Q5_K || TY == BIVMOE_Q6_K))
        if (c.tile_rows > kQuantTile) return launch_quant_one<TY, MODE, 2>(c, A);
    constexpr int smem = eq_smem<TY, NT>();
    static_assert(smem <= 227 * 1024, "the block must fit in shared memory");
    static std::atomic<uint64_t> attr_set{0};
    if (cudaError_t e = ensure_dynamic_smem(experts_quant_kernel<TY, MODE, NT>, smem, attr_set)) return e;
    constexpr int threads = 32 * (4 * eq_groups<TY, NT>() + 1);
    count_launch();
    // the down product may be scheduled while gate+up's last blocks drain: their blocks have the same
    // size, so one only gets an SM that has nothing left to do
    return launch_with(pdl_mode() == 1 || (pdl_mode() != 0 && MODE == EQ_DOWN && c.n < kEarlyTokens), c.stream, experts_quant_kernel<TY, MODE, NT>, dim3(c.sm_count), dim3(threads), smem, A);
}
template <int MODE>
static cudaError_t launch_quant_mode(int ty, const LaunchCfg& c, const QuantArgs& A) {
    switch (ty) {
        case BIVMOE_BF16: return launch_quant_one<BIVMOE_BF16, MODE>(c, A);
        case BIVMOE_Q8_0: return launch_quant_one<BIVMOE_Q8_0, MODE>(c, A);
        case BIVMOE_Q4_0: return launch_quant_one<BIVMOE_Q4_0, MODE>(c, A);
        case BIVMOE_Q4_1: return launch_quant_one<BIVMOE_Q4_1, MODE>(c, A);
        case BIVMOE_Q4_K: return launch_quant_one<BIVMOE_Q4_K, MODE>(c, A);
        case BIVMOE_Q5_K: return launch_quant_one<BIVMOE_Q5_K, MODE>(c, A);
        case BIVMOE_Q6_K: return launch_quant_one<BIVMOE_Q6_K, MODE>(c, A);
        default: return cudaErrorInvalidValue;
    }
}

// one product (gate+up, or down) over the tile list's groups; `tiles_mode` as in QuantArgs
cudaError_t launch_experts_quant(const LaunchCfg& c, bool down, int ty, const DevTiles& w, const DevTiles& sh,
                                 const Workspace& ws, bool quant_mid, int tiles_mode) {
    QuantArgs A{};
    A.w = w;
    A.sh = sh;
    const bool terms = ty == BIVMOE_BF16;
    A.x_t = terms ? (down ? ws.mid_3 : ws.act_3) : down ? ws.mid_t : ws.act_t;
    A.act_rows = ws.act_rows;
    A.out = down ? ws.pair_out : ws.mid;
    A.out_t = down ? nullptr : terms ? ws.mid_3 : quant_mid ? ws.mid_t : nullptr;
    A.tile_desc = ws.tile_desc;
    A.n_tiles = ws.n_tiles;
    A.status = ws.status;
    A.n_expert = c.n_expert;
    A.tiles_mode = tiles_mode;
    A.chunks = std::max(w.chunks, sh.chunks);
    A.parts = down ? c.down_parts : c.gateup_parts;
    A.part_rows = c.n;
    if (A.parts > 1) A.out = ws.parts;
    return down ? launch_quant_mode<EQ_DOWN>(ty, c, A) : launch_quant_mode<EQ_GATEUP>(ty, c, A);
}

// Whether a pass runs through experts_few_kernel: up to eight tokens, quantised gate and up of one
// type with the shared expert's (or none), and rows that fit in shared memory beside the rings.
template <int TY> static bool few_fits(int e) { return few_smem<TY>(e) <= FEW_SMEM_MAX; }
bool few_supported(int n, int k, int e, int n_expert, int ty) {
    if (n < 1 || n > FEW_TOKENS || k > FEW_K || n_expert > FEW_EXPERTS) return false;
    switch (ty) {
        case BIVMOE_Q8_0: return few_fits<BIVMOE_Q8_0>(e);
        case BIVMOE_Q4_0: return few_fits<BIVMOE_Q4_0>(e);
        case BIVMOE_Q4_1: return few_fits<BIVMOE_Q4_1>(e);
        case BIVMOE_Q4_K: return few_fits<BIVMOE_Q4_K>(e);
        case BIVMOE_Q5_K: return few_fits<BIVMOE_Q5_K>(e);
        case BIVMOE_Q6_K: return few_fits<BIVMOE_Q6_K>(e);
        default: return false;
    }
}
template <int TY>
static cudaError_t launch_few_one(const LaunchCfg& c, const float* h, const FewArgs& A) {
    static std::atomic<uint64_t> attr_set{0};
    if (cudaError_t e = ensure_dynamic_smem(experts_few_kernel<TY>, FEW_SMEM_MAX, attr_set)) return e;
    count_launch();
    return launch_early(c.n, c.stream, experts_few_kernel<TY>, dim3(c.sm_count), dim3(32 * (4 * Fmt<TY>::G + 1)),
                        (size_t)few_smem<TY>(c.e), h, A);
}
cudaError_t launch_experts_few(const LaunchCfg& c, const float* h, const DevTiles& w, const DevTiles& sh, const Workspace& ws,
                               const RowNorm* norm) {
    const FewArgs A{w, sh, ws, norm ? norm->w : nullptr, c.n, c.k, c.e, c.n_expert, c.has_shared, std::max(w.chunks, sh.chunks)};
    if (!few_supported(c.n, c.k, c.e, c.n_expert, w.ty)) return cudaErrorInvalidValue;
    switch (w.ty) {
        case BIVMOE_Q8_0: return launch_few_one<BIVMOE_Q8_0>(c, h, A);
        case BIVMOE_Q4_0: return launch_few_one<BIVMOE_Q4_0>(c, h, A);
        case BIVMOE_Q4_1: return launch_few_one<BIVMOE_Q4_1>(c, h, A);
        case BIVMOE_Q4_K: return launch_few_one<BIVMOE_Q4_K>(c, h, A);
        case BIVMOE_Q5_K: return launch_few_one<BIVMOE_Q5_K>(c, h, A);
        case BIVMOE_Q6_K: return launch_few_one<BIVMOE_Q6_K>(c, h, A);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace bivmoe
