"""The rules by which a host-buffer call lets the device reach the caller's memory
(csrc/host_buffers.h), on tables of page-locked ranges: no GPU, no page-locked memory."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <vector>
#include "host_buffers.h"
using namespace bivmoe;
struct Range { uintptr_t at; size_t bytes; bool writable; };
static std::vector<Range> ranges;      // host and device addresses are the same here
static LockedRange look(const void* p) {
    for (const Range& r : ranges)
        if ((uintptr_t)p >= r.at && (uintptr_t)p < r.at + r.bytes) return {(uintptr_t)p, r.at, r.bytes, r.writable};
    return {};
}
static int bad = 0;
#define CHECK(x) do { if (!(x)) { printf("line %d: %s\n", __LINE__, #x); bad = 1; } } while (0)
int main() {
    const size_t row = 1024;
    float *h = (float*)0x100000, *out = (float*)0x200000;
    const int n = 64;                  // 64 KiB each
    auto call = [&](float* a, float* b, int m) { return host_buffers(a, b, m, row, look); };
    // nothing page-locked; one of the two only
    CHECK(!call(h, out, n).locked());
    ranges = {{0x100000, 0x10000, true}};
    CHECK(!call(h, out, n).locked() && call(h, out, n).h_dev == 0x100000);
    ranges = {{0x200000, 0x10000, true}};
    CHECK(!call(h, out, n).locked());
    // both, exactly
    ranges = {{0x100000, 0x10000, true}, {0x200000, 0x10000, true}};
    const HostBuffers both = call(h, out, n);
    CHECK(both.locked() && both.direct());
    // the range ends 16 bytes, or a row, early; starts late; is two ranges side by side
    ranges = {{0x100000, 0x10000 - 16, true}, {0x200000, 0x10000, true}};
    CHECK(!call(h, out, n).locked() && call(h, out, n - 1).locked());
    ranges = {{0x100000, 0x10000, true}, {0x200000, 0x10000 - row, true}};
    CHECK(!call(h, out, n).locked() && call(h, out, n - 1).locked());
    ranges = {{0x100010, 0x10000, true}, {0x200000, 0x10000, true}};
    CHECK(!call(h, out, n).locked() && call(h + 4, out, n).locked());
    ranges = {{0x100000, 0x8000, true}, {0x108000, 0x8000, true}, {0x200000, 0x10000, true}};
    CHECK(!call(h, out, n).locked());
    // part of a larger range; 16-byte alignment decides for the kernels only
    ranges = {{0x100000, 0x20000, true}, {0x200000, 0x20000, true}};
    CHECK(call(h + 1, out, n).locked() && !call(h + 1, out, n).direct());
    CHECK(call(h, out + 2, n).locked() && !call(h, out + 2, n).direct());
    CHECK(call(h + 4, out + 8, n).direct());
    // rows may be read from, but not written to, memory that is read-only for the device
    ranges = {{0x100000, 0x10000, false}, {0x200000, 0x10000, true}};
    CHECK(call(h, out, n).direct());
    ranges = {{0x100000, 0x10000, true}, {0x200000, 0x10000, false}};
    CHECK(!call(h, out, n).locked());
    // what was captured may be replayed only while all of it is as it was
    ranges = {{0x100000, 0x10000, true}, {0x200000, 0x10000, true}};
    CHECK(call(h, out, n) == both);
    CHECK(!(call(h, out, n - 1) == both));
    ranges = {{0x100000, 0x10000, true}};                          // the output was unpinned
    CHECK(!(call(h, out, n) == both));
    ranges = {{0x100000, 0x10000 - 16, true}, {0x200000, 0x10000, true}};   // and pinned again, shorter
    CHECK(!(call(h, out, n) == both));
    return bad;
}
"""


def test_host_buffers_rules(tmp_path):
    src = tmp_path / "t.cpp"
    src.write_text(PROGRAM)
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", os.path.join(ROOT, "biv_b200", "csrc"), str(src),
                    "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


@pytest.mark.gpu
def test_a_buffer_that_is_no_longer_page_locked_is_copied():
    # the graph captured for page-locked buffers must not be replayed once one of them, at the
    # same address, is ordinary memory; pinned again, it is used in place again
    import numpy as np
    import torch
    from biv_b200 import workloads as W
    from biv_b200.moe import Moe
    rt = torch.cuda.cudart()
    wl = W.decode_q4k(n=40, **W.SMALL)
    m = Moe(wl.layer, wl.n)

    def pages(a):   # page-aligned rows: registering them pins nothing else
        raw = np.empty(a.nbytes + 8192, np.uint8)
        at = -raw.ctypes.data % 4096
        out = raw[at:at + a.nbytes].view(np.float32).reshape(a.shape)
        out[:] = a
        return out

    try:
        want = m.moe_host(wl.h)
        h, out = pages(wl.h), pages(np.zeros_like(wl.h))
        for unpin in (h, out):
            for a in (h, out):
                assert int(rt.cudaHostRegister(a.ctypes.data, a.nbytes, 0)) == 0
            for _ in range(3):
                out[:] = 0
                m.moe_host(h, out)
                assert np.array_equal(out, want)
            assert int(rt.cudaHostUnregister(unpin.ctypes.data)) == 0
            for _ in range(3):
                out[:] = 0
                m.moe_host(h, out)
                assert np.array_equal(out, want)
            other = out if unpin is h else h
            assert int(rt.cudaHostUnregister(other.ctypes.data)) == 0
        m.status()
    finally:
        m.close()
