// The bounded wait of the expert kernels' roles for one another.  Plain C++, without the CUDA
// headers, so that the rule can be tested where there is no GPU.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define BIV_WAIT_FN __device__ __forceinline__
#else
#define BIV_WAIT_FN inline
#endif

namespace bivmoe {

constexpr uint64_t kWaitNs = 2000000000ull;

// Waits until ready; false when it gave up.
//   w.ready()   one try           w.pause()   between two tries
//   w.late(k)   the k-th look, once in EVERY tries, at whether to give up
template <int EVERY, class W>
BIV_WAIT_FN bool bounded_wait(W w) {
    for (uint32_t i = 1; !w.ready(); i++) {
        if (i % EVERY == 0 && w.late(i / EVERY)) return false;
        w.pause();
    }
    return true;
}

// The same for the lanes of a warp, which go on, or leave, together: w.all(v) whether v holds for all
// of them.  A lane that sees another role's flag one turn before the others would by itself leave for
// the end of the kernel, and they would go on without it to what a whole warp has to execute
// (tensor-memory loads and stores, matrix instructions, shuffles).
template <int EVERY, class W>
BIV_WAIT_FN bool bounded_wait_together(W w) {
    const bool here = bounded_wait<EVERY>(w);
    return w.all(here);
}

// What a warp does that gave up on a wait while others may meet at a barrier that counts it: it arrives
// there for them (m.arrive()) until all have left (m.all_left()), each at its next wait; `turns` bounds
// that.  An arrival too many only ends a meeting early, which spoils nothing but results that the
// status disowns.  (Meetings at mbarriers, which a bounded wait could leave, cost the kernels 1 to 5 %.)
template <class M>
BIV_WAIT_FN void arrive_until_all_left(M m, uint32_t turns) {
    for (uint32_t i = 0; i < turns && !m.all_left(); i++) m.arrive();
}

}  // namespace bivmoe
