// Inline-PTX helpers of the tcgen05 kernels: mbarriers with bounded waits, bulk
// copies, shared-memory matrix descriptors, MMA issue and commit, tensor-memory
// loads, packed f32x2 arithmetic.
#pragma once
#include <stdint.h>

#include "bounded_wait.h"

namespace bivmoe {

__device__ __forceinline__ uint32_t pf_smem(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
// One lane of the warp, which has to be together here.  Where the branch to what one lane does is
// this, and not a comparison of lane numbers, the compiler knows that a single lane is active and
// keeps the operands of tensor-core instructions in uniform registers: an MMA 128 x 16 x 16 issues
// in 9 to 16 clocks that way, in 45 the other (a probe that issues nothing else).
__device__ __forceinline__ bool pf_elect() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ void pf_bar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(pf_smem(bar)), "r"(count));
}
__device__ __forceinline__ void pf_bar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(pf_smem(bar)) : "memory");
}
__device__ __forceinline__ void pf_bar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(pf_smem(bar)),
                 "r"(bytes)
                 : "memory");
}
// One try: the hardware suspends the warp until the phase completes, for a time of its own
// choosing.  (With a suspend time the waits of the warp-MMA kernel, a stage or less long, ended
// late: 64 tokens Q4_K 85 -> 81 us without.)
__device__ __forceinline__ bool pf_bar_try(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(pf_smem(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ uint64_t pf_now_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// What bounded_wait waits with: an mbarrier's phase, until `*abort` (a block-wide flag in shared memory)
// is set.  CLOCK: or until kWaitNs have passed, for the role of a block that raises the flag when the
// block does not get on; the others give up by themselves only after 2^14 looks.
template <bool CLOCK = false, bool SLEEP = false> struct PfWait {
    uint64_t* bar;
    uint32_t parity;
    const volatile int* abort;
    uint64_t t0 = 0;
    __device__ __forceinline__ bool ready() const { return pf_bar_try(bar, parity); }
    __device__ __forceinline__ bool late(uint32_t look) {
        if (CLOCK) {
            const uint64_t t = pf_now_ns();
            if (look == 1) t0 = t;
            return *abort || t - t0 >= kWaitNs;
        }
        return *abort || (look >> 14) != 0;
    }
    __device__ __forceinline__ void pause() const { if (SLEEP) __nanosleep(32); }
    __device__ __forceinline__ bool all(bool v) const { return __all_sync(0xffffffffu, v); }
};
// For arrive_until_all_left: a named barrier of `threads`, and an mbarrier that every warp which meets
// there arrives at when it leaves its loop.
struct PfMeeting {
    int id, threads;
    uint64_t* left;
    __device__ __forceinline__ bool all_left() const { return __any_sync(0xffffffffu, pf_bar_try(left, 0)); }
    __device__ __forceinline__ void arrive() const { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
};
constexpr uint32_t kLeaveTurns = 1u << 16;
// The same where nobody counts who has left: a turn takes a microsecond.
struct PfMeetingForAWhile {
    int id, threads;
    __device__ __forceinline__ bool all_left() const { __nanosleep(1000); return false; }
    __device__ __forceinline__ void arrive() const { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
};
constexpr uint64_t PF_WAIT_NS = kWaitNs;
// Bounded wait for the phase of parity `parity`; false when it gave up: after PF_WAIT_NS, or
// once `*abort` (when given, a block-wide flag in shared memory) is set.
__device__ __forceinline__ bool pf_bar_wait(uint64_t* bar, uint32_t parity, const volatile int* abort = nullptr) {
    if (pf_bar_try(bar, parity)) return true;
    const uint64_t t0 = pf_now_ns();
    do {
        if (pf_bar_try(bar, parity)) return true;
        if (abort && *abort) return false;
    } while (pf_now_ns() - t0 < PF_WAIT_NS);
    return false;
}
// The same with a suspend time, for waits of many stages: the warps that wait then take fewer issue
// slots and less of the power that the tensor cores run on.  BF16 tcgen05 kernels, with the wait
// above and with this one, passes 150 ms apart / back to back: 1536 rows, 8 experts of 4096 / 14336,
// 2844 -> 2794 / 3433 -> 3301 us; 16384 rows of 2048 / 512 2313 -> 2293 / 2541 -> 2541.  Gives up
// after 2^16 tries.
__device__ __forceinline__ bool pf_bar_wait_long(uint64_t* bar, uint32_t parity) {
    for (uint32_t i = 0; i < (1u << 16); i++) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(pf_smem(bar)), "r"(parity), "r"(20000u)   // ns
            : "memory");
        if (ok) return true;
    }
    return false;
}
// What one lane of a warp got of a wait, for all of them: they go on, or leave, together (bounded_wait.h).
__device__ __forceinline__ bool pf_together(bool ok) { return __all_sync(0xffffffffu, ok); }
__device__ __forceinline__ void pf_bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
            "r"(pf_smem(dst)),
        "l"(src), "r"(bytes), "r"(pf_smem(bar))
        : "memory");
}
// The same way out, in the thread's own order of groups; the thread waits until what its groups copy has
// been read, or has been written.
__device__ __forceinline__ void pf_bulk_s2g(void* dst, const void* src, uint32_t bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(pf_smem(src)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void pf_bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void pf_bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void pf_bulk_wait() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
// Shared-memory matrix descriptor, K-major, no swizzle: 8 rows x 16 bytes are
// contiguous; `sbo` bytes from one 8-row group to the next, `lbo` bytes from
// one 16-byte K step to the next.
__device__ __forceinline__ uint64_t pf_desc(uint32_t smem_addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo >> 4) << 16) |
           ((uint64_t)(sbo >> 4) << 32) | (1ull << 46);
}
// The same for the 128-byte swizzle, K-major: a row is 128 contiguous bytes (64 bf16),
// 8 rows make a 1024-byte atom (1024-byte aligned), and the 16-byte piece c of row r of
// an atom sits at piece position c ^ r.  `sbo` = 1024 from one 8-row group to the next;
// a K step of 16 bf16 advances the start address by 32 bytes.
__device__ __forceinline__ uint64_t pf_desc_sw128(uint32_t smem_addr) {
    return (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) |
           (1ull << 46) | (2ull << 61);
}
// kind::i8 instruction descriptor: s32 accumulator, signed 8-bit A and B, both K-major
__device__ __forceinline__ uint32_t pf_idesc(int m, int n) {
    return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
__device__ __forceinline__ void pf_mma_i8(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, 0, 0;\n\t"   // overwrite the buffer: a block dot is not accumulated
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc)
        : "memory");
}
// kind::f16 instruction descriptor: f32 accumulator, bf16 A and B, both K-major
__device__ __forceinline__ uint32_t pf_idesc_bf16(int m, int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
// The same of two MMAs in a row with one A: the first leaves A in the collector buffer, the second takes
// it from there instead of from shared memory.
template <bool FIRST>
__device__ __forceinline__ void pf_mma_bf16_pair(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                                 uint32_t accumulate) {
    if (FIRST)
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16.collector::a::fill [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
            "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
            : "memory");
    else
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16.collector::a::lastuse [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
            "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
            : "memory");
}
// D (+)= A * B, 16 bf16 values of K per instruction
__device__ __forceinline__ void pf_mma_bf16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                            uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void pf_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                     pf_smem(bar))
                 : "memory");
}
__device__ __forceinline__ void pf_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void pf_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// 32 consecutive columns of this warp's 32 lanes of tensor memory
__device__ __forceinline__ void pf_tmem_ld32(uint32_t taddr, int (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
          "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
          "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]),
          "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]),
          "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void pf_tmem_ld16(uint32_t taddr, int (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
          "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
          "=r"(v[14]), "=r"(v[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void pf_tmem_ld8(uint32_t taddr, int (&v)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr) : "memory");
}
// 16 lanes x 8 N consecutive columns, N = 1, 2 or 4, of this warp's 32 lanes (`taddr`: the first
// of the 16): register 4 j + 2 i + t of lane l is lane l / 4 + 8 i, column 8 j + 2 (l % 4) + t
template <int N>
__device__ __forceinline__ void pf_tmem_ld_16x8(uint32_t taddr, int* v) {
    if constexpr (N == 1)
        asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0,%1,%2,%3}, [%4];"
                     : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(taddr) : "memory");
    else if constexpr (N == 2)
        asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                     : "r"(taddr) : "memory");
    else
        asm volatile(
            "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
              "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
            : "r"(taddr) : "memory");
}
__device__ __forceinline__ void pf_tmem_wait_ld() {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// loads from shared memory by their 32-bit address
__device__ __forceinline__ uint32_t lds32(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
// two f32 lanes per instruction (sm_100): d = a * b + c, d = a + b, d = a * b
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 lds_f2(uint32_t a) {
    f32x2 v;
    asm volatile("ld.shared.b64 %0, [%1];" : "=l"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ uint4 lds128(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ f32x2 pk(float lo, float hi) {
    return (f32x2)__float_as_uint(lo) | ((f32x2)__float_as_uint(hi) << 32);
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ float lo_of(f32x2 v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float hi_of(f32x2 v) { return __uint_as_float((uint32_t)(v >> 32)); }
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

}  // namespace bivmoe
