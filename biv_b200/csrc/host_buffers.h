// Which of a caller's host buffers the device may reach by itself.  Plain C++, without the
// CUDA headers, so that the rules can be tested where there is no GPU.
#pragma once
#include <stddef.h>
#include <stdint.h>

namespace bivmoe {

// The page-locked range that an address lies in, as the driver describes it: the device's
// address of the address asked for, the range's first device address, its bytes (0: the
// address is not page-locked), and whether the device may write there.
struct LockedRange {
    uintptr_t dev = 0, start = 0;
    size_t bytes = 0;
    bool writable = false;
};

// The device's address of `bytes` bytes at `p`, or 0 unless all of them lie in one page-locked
// range (and the device may write there, if it has to).  `look`: const void* -> LockedRange.
template <class Look>
inline uintptr_t locked_view(const void* p, size_t bytes, bool write, Look&& look) {
    const LockedRange r = look(p);
    if (r.bytes == 0 || r.dev < r.start || (write && !r.writable)) return 0;
    const uintptr_t off = r.dev - r.start;
    return off <= r.bytes && r.bytes - off >= bytes ? r.dev : 0;
}

// A host-buffer call's two buffers.  What was captured for one call may be replayed for another
// only when all of this is equal: a buffer at the same address need not be page-locked any more.
struct HostBuffers {
    const float* h = nullptr;
    float* out = nullptr;
    int n = -1;
    uintptr_t h_dev = 0, out_dev = 0;   // the device's addresses; 0: not page-locked
    bool operator==(const HostBuffers& o) const {
        return h == o.h && out == o.out && n == o.n && h_dev == o.h_dev && out_dev == o.out_dev;
    }
    bool locked() const { return h_dev && out_dev; }
    // whether kernels may read and write them in place (16 bytes at a time)
    bool direct() const { return locked() && h_dev % 16 == 0 && out_dev % 16 == 0; }
};
template <class Look>
inline HostBuffers host_buffers(const float* h, float* out, int n, size_t row_bytes, Look&& look) {
    const size_t bytes = (size_t)n * row_bytes;
    return HostBuffers{h, out, n, locked_view(h, bytes, false, look), locked_view(out, bytes, true, look)};
}

}  // namespace bivmoe
