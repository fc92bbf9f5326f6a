// Kernel launches with programmatic dependent launch: the kernel may be scheduled while
// the previous kernel of the stream is still draining, so that its launch latency and its
// prologue (barrier set-up, shared-memory carving) overlap the predecessor's tail.  Every
// kernel launched this way calls pdl_wait() before it touches anything an earlier kernel
// of the stream wrote - in every thread, before any early return - which is what keeps
// the chain of dependencies intact: a kernel that has passed its wait knows that its
// predecessor, and through the predecessor's own wait everything before it, is complete.
#pragma once
#include <cuda_runtime.h>

#include <cstdlib>
#include <type_traits>
#include <vector>

namespace bivmoe {

// Which launches of a captured pass were given the caller's rows or the caller's output, as they
// were made: what the nodes of its graph have to be rewritten by when a call brings other buffers.
// Filled by every launch of the thread while `launch_watch()` points at one.
struct LaunchWatch {
    const void *h = nullptr, *out = nullptr;
    struct Seen { const void* kernel; int args; std::vector<int> h_at, out_at; };   // argument positions
    std::vector<Seen> seen;
};
inline LaunchWatch*& launch_watch() {
    static thread_local LaunchWatch* w = nullptr;
    return w;
}
// The rows are read through pointers to const, the output is written through others: that tells
// them apart in a call that works in place.
template <class T>
inline void watch_value(LaunchWatch::Seen& s, const LaunchWatch& w, int at, const T& v) {
    if constexpr (std::is_pointer_v<T>) {
        constexpr bool reads = std::is_const_v<std::remove_pointer_t<T>>;
        if (reads && (const void*)v == w.h) s.h_at.push_back(at);
        if (!reads && (const void*)v == w.out) s.out_at.push_back(at);
    }
}
template <class... KArgs>
inline void watch_launch(const void* kernel, KArgs... args) {
    LaunchWatch* w = launch_watch();
    if (!w) return;
    LaunchWatch::Seen s{kernel, (int)sizeof...(KArgs), {}, {}};
    int at = 0;
    (watch_value(s, *w, at++, args), ...);
    if (!s.h_at.empty() || !s.out_at.empty()) w->seen.push_back(s);
}

__device__ __forceinline__ void pdl_wait() {
    // without the launch attribute this is a no-op
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
// Lets the next kernel of the stream be scheduled once every block of this one has got
// here (or exited): placed at the top of a kernel, the successor's blocks fill in as this
// kernel's last wave drains, and then sit in their own pdl_wait().
__device__ __forceinline__ void pdl_launch_dependents() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
// both, for kernels with nothing to do before their inputs are ready
__device__ __forceinline__ void pdl_enter() {
    pdl_launch_dependents();
    pdl_wait();
}

template <class... KArgs, class... Args>
inline cudaError_t launch_with(bool overlap, cudaStream_t stream, void (*kernel)(KArgs...), dim3 grid, dim3 block,
                               size_t smem, Args... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = overlap ? 1 : 0;
    watch_launch<KArgs...>((const void*)kernel, KArgs(args)...);
    return cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
}
// BIVMOE_PDL: 1 every launch may overlap its predecessor, 0 none, unset those of launch_early
inline int pdl_mode() {
    static const int mode = [] { const char* e = getenv("BIVMOE_PDL"); return e ? atoi(e) : -1; }();
    return mode;
}
template <class... KArgs, class... Args>
inline cudaError_t launch_after(cudaStream_t stream, void (*kernel)(KArgs...), dim3 grid, dim3 block,
                                size_t smem, Args... args) {
    return launch_with(pdl_mode() == 1, stream, kernel, grid, block, smem, args...);
}
// For the small kernels between the router product and the expert products, which follow one
// another: with few tokens their launch latencies overlap (one token 30.9 -> 28.3 us a pass, 64
// tokens 75.3 -> 71.3, 33 BF16 tokens 203 -> 201; 509 tokens 274 -> 279, so not from 256 tokens
// on).  A kernel that follows the expert products only takes their room when it is scheduled
// early: with the combine and the norm early a stack of four layers and 160 tokens went from
// 646 to 652 us, with every launch to 686.
// So does the down product of the small groups (experts_quant.cu: 160 tokens, four layers 645 -> 638 us,
// one token 24.0 -> 23.4), and for a few tokens, whose blocks are few, the combine (-> 23.0).
constexpr int kEarlyTokens = 256, kEarlyCombine = 8;
template <class... KArgs, class... Args>
inline cudaError_t launch_early(int n, cudaStream_t stream, void (*kernel)(KArgs...), dim3 grid, dim3 block,
                                size_t smem, Args... args) {
    return launch_with(pdl_mode() == 1 || (pdl_mode() != 0 && n < kEarlyTokens), stream, kernel, grid, block, smem, args...);
}

}  // namespace bivmoe
