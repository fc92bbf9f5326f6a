// Device-side decoding of the weight block formats (device row layouts are
// described in common.cuh) and the Q8 activation quantiser.  Shared by the
// expert kernels and by the int32 block-dot tap so both see the same integers.
// Reference: engine/src/quant.rs:144-153 (scale_min_k4), 368-394 (quantiser),
// 599-686 (scalar dots: the definition of each block's integers).
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

namespace bivmoe {

// The 6-bit scales and mins of a Q4_K / Q5_K super-block, from its 12 packed
// bytes held as three little-endian words: byte j of sc_lo/m_lo is sub-block j
// (j < 4), byte j of sc_hi/m_hi is sub-block 4 + j.
struct K4Scales { uint32_t sc_lo, sc_hi, m_lo, m_hi; };
__device__ __forceinline__ K4Scales unpack_k4_scales(uint32_t w0, uint32_t w1, uint32_t w2) {
    K4Scales s;
    s.sc_lo = w0 & 0x3F3F3F3Fu;
    s.m_lo = w1 & 0x3F3F3F3Fu;
    s.sc_hi = (w2 & 0x0F0F0F0Fu) | ((w0 >> 2) & 0x30303030u);
    s.m_hi = ((w2 >> 4) & 0x0F0F0F0Fu) | ((w1 >> 2) & 0x30303030u);
    return s;
}

// The three bf16 terms of an f32: hi + mid + lo is the value itself (3 x 8 significant bits,
// short of terms below the smallest bf16, 2^-133).  A value that rounds past the largest bf16
// is truncated instead, and an infinity is hi alone: as a second term, inf - inf would make a
// NaN of a product that is infinite.
__device__ __forceinline__ void split_bf16_3(float v, uint16_t (&t)[3]) {
#pragma unroll
    for (int i = 0; i < 3; i++) {
        __nv_bfloat16 b = __float2bfloat16_rn(v);
        if (i == 0 && isinf(__bfloat162float(b))) b = __float2bfloat16_rz(v);
        t[i] = __bfloat16_as_ushort(b);
        v = i == 0 && isinf(v) ? 0.0f : v - __bfloat162float(b);
    }
}

// One Q8 block (32 values) held by the 32 lanes of a warp: returns the int8
// value of this lane; d and s are the block's scale and d * sum(q).
// quant.rs:380-393: d = amax/127, id = 1/d (0 when d is 0), q = round(v*id)
// with halves away from zero, s = d * (float)sum.
__device__ __forceinline__ int q8_quantize_lane(float v, float& d, float& s) {
    float amax = fabsf(v);
#pragma unroll
    for (int o = 16; o; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    d = __fdiv_rn(amax, 127.0f);
    const float id = d != 0.0f ? __fdiv_rn(1.0f, d) : 0.0f;
    const int q = (int)roundf(__fmul_rn(v, id));
    int sum = q;
#pragma unroll
    for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    s = __fmul_rn(d, (float)sum);
    return q;
}

// Quantised rows.  A thread owns 8 consecutive values, four threads a 32-value block:
// the block's amax and sum(q) take two shuffle steps, two neighbouring threads make one
// 16-byte unit of int8, and one thread of the four stores the block's scales.  (One lane
// per value - a warp per block, five shuffle steps per reduction - cost eight times the
// instructions and took 0.18 ms for 4096 rows.)  The quantiser's arithmetic is
// q8_quantize_lane's: max and the integer sum do not depend on the order.
__device__ __forceinline__ void quantize_eight(const float (&v)[8], uint32_t& w0, uint32_t& w1, float& dd, float& ss) {
    // quant.rs:380-393: d = amax/127, id = 1/d (0 when d is 0), q = round(v*id) with
    // halves away from zero, s = d * (float)sum
    float amax = fabsf(v[0]);
#pragma unroll
    for (int j = 1; j < 8; j++) amax = fmaxf(amax, fabsf(v[j]));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
    dd = __fdiv_rn(amax, 127.0f);
    const float id = dd != 0.0f ? __fdiv_rn(1.0f, dd) : 0.0f;
    int sum = 0;
    w0 = w1 = 0;
#pragma unroll
    for (int j = 0; j < 8; j++) {
        const int q = (int)roundf(__fmul_rn(v[j], id));
        sum += q;
        if (j < 4) w0 |= ((uint32_t)q & 0xffu) << (8 * j);
        else w1 |= ((uint32_t)q & 0xffu) << (8 * (j - 4));
    }
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    ss = __fmul_rn(dd, (float)sum);
}

// Eight int8 values, as two words, as the f16 numbers of a unit of an f16 record (common.cuh: every
// four in the order 0 2 1 3): a byte as the low mantissa bits of 1024, less 1024 + 128.
__device__ __forceinline__ uint4 half_unit(uint32_t w0, uint32_t w1) {
    const uint32_t x0 = w0 ^ 0x80808080u, x1 = w1 ^ 0x80808080u;
    uint32_t r[4] = {__byte_perm(x0, 0x64646464u, 0x4240), __byte_perm(x0, 0x64646464u, 0x4341),
                     __byte_perm(x1, 0x64646464u, 0x4240), __byte_perm(x1, 0x64646464u, 0x4341)};
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const __half2 h = __hadd2(*(__half2*)&r[i], __half2half2(__ushort_as_half(0xE480)));
        r[i] = *(const uint32_t*)&h;
    }
    return make_uint4(r[0], r[1], r[2], r[3]);
}
// Eight quantised values of a thread as what it stores of them in every record they go to: an even thread a
// 16-byte unit (with its neighbour's eight), each of a block's four threads one of its scales; HALF: an f16 record.
struct Q8Unit { uint4 unit; float val, dd, ss; };
__device__ __forceinline__ Q8Unit q8_unit(const float (&v)[8], int lane, bool half) {
    Q8Unit u;
    uint32_t w0, w1;
    quantize_eight(v, w0, w1, u.dd, u.ss);
    if (half) {
        u.unit = half_unit(w0, w1);
        return u;
    }
    // the neighbour's 8 bytes: an even thread holds the low half of a 16-byte unit
    const uint32_t p0 = __shfl_down_sync(0xffffffffu, w0, 1), p1 = __shfl_down_sync(0xffffffffu, w1, 1);
    u.unit = make_uint4(w0, w1, p0, p1);
    float shi, slo;
    split_tf32(u.ss, &shi, &slo);
    const int which = lane & 3;
    u.val = which == 0 ? u.dd : which == 1 ? shi : which == 2 ? slo : u.ss;
    return u;
}
// A thread's eight values of a block into an f16 record: their unit, and one of the block's four
// scales (`which`: the thread's place among the block's four).
__device__ __forceinline__ void put_half_record(uint8_t* rec, int tk, int el, int which, const uint4& unit, float dd, float ss) {
    *(uint4*)(rec + half_q_off(tk, el)) = unit;
    float shi, slo;
    split_tf32(ss, &shi, &slo);
    *(float*)(rec + half_scale_off(which, el / 32, tk)) = which == 0 ? dd : which == 1 ? shi : which == 2 ? slo : ss;
}

// values i0 .. i0 + 7 of the row at position pos; R positions in all
__device__ __forceinline__ void put_q8_unit(uint8_t* act_t, int R, int pos, int i0, int lane, bool half, const Q8Unit& u) {
    const int sl = i0 / 256, el = i0 % 256;       // K-slice, element within it
    if (half) {
        put_half_record(act_t + ((size_t)sl * (R / 8) + pos / 8) * kHalfRec, pos % 8, el, lane & 3, u.unit, u.dd, u.ss);
        return;
    }
    uint8_t* rec = act_t + ((size_t)sl * (R / 8) + pos / 8) * kActTileBytes;
    if (!(lane & 1)) *(uint4*)(rec + act_q_off(pos % 8, el)) = u.unit;
    *(float*)(rec + act_scale_off(lane & 3, el / 32, pos % 8)) = u.val;
}

// A row by the threads of a block, e % 256 == 0 (whole warps): quantised, [e] int8 and [e / 32] (d, s) ...
__device__ __forceinline__ void quantize_row(const float* __restrict__ x, int8_t* __restrict__ q, float2* __restrict__ s, int e) {
    for (int i0 = threadIdx.x * 8; i0 < e; i0 += blockDim.x * 8) {
        const float4 a = *(const float4*)(x + i0), b = *(const float4*)(x + i0 + 4);
        const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        uint32_t w0, w1;
        float dd, ss;
        quantize_eight(v, w0, w1, dd, ss);
        *(uint2*)(q + i0) = make_uint2(w0, w1);
        if ((threadIdx.x & 3) == 0) s[i0 / 32] = make_float2(dd, ss);
    }
}
// ... or as two bf16 terms, [K / 64][hi 64 | lo 64]; with norm_w the row is x * (scale * w), rms_norm on the fly.
__device__ __forceinline__ void split_row(const float* __restrict__ x, uint8_t* __restrict__ to, int e, const float* norm_w = nullptr,
                                          float nscale = 1.0f) {
    for (int i0 = threadIdx.x * 8; i0 < e; i0 += blockDim.x * 8) {
        float4 a = *(const float4*)(x + i0), b = *(const float4*)(x + i0 + 4);
        if (norm_w) {
            const float4 wa = *(const float4*)(norm_w + i0), wb = *(const float4*)(norm_w + i0 + 4);
            a.x = __fmul_rn(a.x, __fmul_rn(nscale, wa.x)); a.y = __fmul_rn(a.y, __fmul_rn(nscale, wa.y));
            a.z = __fmul_rn(a.z, __fmul_rn(nscale, wa.z)); a.w = __fmul_rn(a.w, __fmul_rn(nscale, wa.w));
            b.x = __fmul_rn(b.x, __fmul_rn(nscale, wb.x)); b.y = __fmul_rn(b.y, __fmul_rn(nscale, wb.y));
            b.z = __fmul_rn(b.z, __fmul_rn(nscale, wb.z)); b.w = __fmul_rn(b.w, __fmul_rn(nscale, wb.w));
        }
        const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        uint32_t hi[4], lo[4];
#pragma unroll
        for (int p = 0; p < 4; p++) {
            const __nv_bfloat16 h0 = __float2bfloat16_rn(v[2 * p]), h1 = __float2bfloat16_rn(v[2 * p + 1]);
            const __nv_bfloat16 l0 = __float2bfloat16_rn(v[2 * p] - __bfloat162float(h0));
            const __nv_bfloat16 l1 = __float2bfloat16_rn(v[2 * p + 1] - __bfloat162float(h1));
            hi[p] = (uint32_t)__bfloat16_as_ushort(h0) | ((uint32_t)__bfloat16_as_ushort(h1) << 16);
            lo[p] = (uint32_t)__bfloat16_as_ushort(l0) | ((uint32_t)__bfloat16_as_ushort(l1) << 16);
        }
        uint8_t* rec = to + (size_t)(i0 / 64) * kTokBRec + (i0 % 64) * 2;
        *(uint4*)rec = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        *(uint4*)(rec + kTokBLo) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    }
}

}  // namespace bivmoe
