"""Which groups go to the tcgen05 kernels (csrc/big_groups.h): the rule's bound on any routing, and
the sides of its line that were measured; on a GPU, the groups a pass gives those kernels."""
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <algorithm>
#include <cstdio>
#include <random>
#include <vector>
#include "big_groups.h"
using namespace bivmoe;
static int bad = 0;
#define CHECK(x) do { if (!(x)) { printf("line %d: %s\n", __LINE__, #x); bad = 1; } } while (0)
static BigGroups rule(bool bf16, int e, int ff) {
    const long long bytes = bf16 ? 6ll * e * ff : 3ll * e * ff * 34 / 32;
    return {bf16 ? 9 : 17, big_worth(bf16, e, ff, bytes), bytes, bytes};
}
int main() {
    // no routing reaches more than the bound: groups of any sizes up to n that add up to n * k
    std::mt19937 rng(1);
    for (int i = 0; i < 20000; i++) {
        const int n = 1 + rng() % 400, k = 1 + rng() % 8, shared = rng() % 2;
        BigGroups b{9, 0, 1000, 700};
        long long left = (long long)n * k, again = 0;
        const int most = 1 + rng() % n;
        while (left > 0) {
            // sizes one above a multiple of a tile make the most tiles to read again
            long long r = std::min<long long>(left, std::min<long long>(n, rng() % 2 ? most : most / 8 * 8 + 1));
            if (r >= b.min) again += (r - 1) / kSmallTile;
            left -= r;
        }
        const long long bytes = again * b.tile_bytes + (shared && n >= b.min ? (n - 1) / kSmallTile * b.sh_tile_bytes : 0);
        CHECK(bytes <= big_reach(b, n, k, shared));
    }
    // 160 rows, 8 each and a shared expert: eight groups of 153 and one of 56 and the rows themselves
    CHECK(big_reach({17, 0, 1, 1}, 160, 8, 1) >= 8 * 19 + 6 + 19);
    // passes of which both kernels were timed: the sums of tiles read again, and which was faster
    struct { bool bf16; int e, ff, again; bool big; } seen[] = {
        {false, 2048, 512, 87, false}, {false, 2048, 512, 203, true}, {false, 4096, 1536, 55, false}, {false, 4096, 1536, 61, true},
        {false, 4096, 14336, 4, false}, {false, 4096, 14336, 29, true}, {false, 4096, 14336, 139, true},
        {false, 512, 256, 139, false}, {false, 512, 256, 570, true}, {false, 1024, 512, 154, false},
        {false, 1024, 512, 301, true}, {true, 2048, 512, 63, false},
        {true, 2048, 512, 91, true}, {true, 2048, 512, 114, true}, {true, 4096, 1536, 15, false}, {true, 4096, 1536, 82, true},
        {true, 4096, 14336, 2, false}, {true, 4096, 14336, 10, true}, {true, 4096, 14336, 139, true},
        {true, 512, 256, 70, false}, {true, 512, 256, 573, true}};
    for (auto& s : seen) {
        const BigGroups b = rule(s.bf16, s.e, s.ff);
        if ((s.again * b.tile_bytes >= b.worth) != s.big) {
            printf("%s %d / %d, %d tiles\n", s.bf16 ? "BF16" : "Q8_0", s.e, s.ff, s.again);
            bad = 1;
        }
    }
    struct { int e, ff, tiles; bool bf16, big; } alone[] = {
        {2048, 512, 49, false, false}, {2048, 512, 124, false, true}, {4096, 1536, 49, false, true},
        {4096, 14336, 2, false, false}, {4096, 14336, 7, false, true}, {2048, 512, 19, true, false},
        {2048, 512, 49, true, true}, {4096, 1536, 7, true, false}, {4096, 1536, 19, true, true},
        {4096, 14336, 7, true, true}};
    for (auto& s : alone) {
        BigGroups b = rule(s.bf16, s.e, s.ff);
        b.worth = big_worth_alone(s.e, s.ff);
        if ((big_for(b, 8 * s.tiles + 1, 0, 1).min > 0) != s.big) {
            printf("alone %s %d / %d, %d tiles\n", s.bf16 ? "BF16" : "Q8_0", s.e, s.ff, s.tiles);
            bad = 1;
        }
    }
    // a pass without rows for a single group, or that cannot reach the worth, asks for none
    CHECK(big_for(rule(true, 2048, 512), 8, 8, 1).min == 0);
    CHECK(big_for(rule(true, 2048, 512), 64, 8, 1).min == 0);
    CHECK(big_for(rule(true, 2048, 512), 96, 8, 1).min == 9);
    CHECK(big_for({9, 0, 0, 0}, 9, 1, 0).min == 9);
    return bad;
}
"""


def test_big_groups_rule(tmp_path):
    src = tmp_path / "t.cpp"
    src.write_text(PROGRAM)
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I", os.path.join(ROOT, "biv_b200", "csrc"),
                    str(src), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("bf16", [False, True])
def test_groups_of_wide_experts_go_to_the_tensor_core_kernels(bf16):
    # 8 experts of 1024 / 4096, 400 rows to 2 each: 96 tiles to read again are 2.4 GB of BF16
    # weights (Q8_0: 1.3 GB); 40 rows of them, or 100 of experts of 256 / 256, are not worth the start
    import torch
    from biv_b200 import capi, workloads as W
    from biv_b200.moe import Moe
    from test_gpu_parity import run_case
    make = W.ep_bf16 if bf16 else W.parity_q8_0
    wl = make(n=400, n_embd=1024, n_expert=8, k=2, ff=4096, ff_sh=0)
    small = make(n=400, n_embd=256, n_expert=8, k=2, ff=256, ff_sh=0)
    for w, n, first in ((wl, 400, 9 if bf16 else 17), (wl, 40, 0), (small, 100, 0)):
        m = Moe(w.layer, n)
        try:
            m.moe(torch.from_numpy(w.h[:n].copy()).cuda())
            assert m.tap(capi.TAP_BIG_MIN)[0] == first
            if first:
                assert m.tap(capi.TAP_COUNTS).max() >= first
        finally:
            m.close()
    run_case(wl)


@pytest.mark.gpu
@pytest.mark.parametrize("bf16", [False, True])
def test_expert_parallel_steps_weigh_their_groups(bf16):
    # few rows leave the tcgen05 kernels (and for BF16 the kernel that splits rows for them) out
    # of the launches of the shared expert's step and of the owner's; many rows bring them in
    import ctypes as C
    import torch
    from biv_b200 import capi, workloads as W
    from biv_b200.ep import DeviceSteps
    from biv_b200.moe import launch_count
    wl = (W.ep_bf16 if bf16 else W.parity_q8_0)(n=1024, n_embd=1024, n_expert=8, k=2, ff=4096, ff_sh=2048)
    st = DeviceSteps(wl.layer, 1024, 0, 2)
    try:
        def launches(f):
            before = launch_count()
            f()
            torch.cuda.synchronize()
            return launch_count() - before

        seen = {}
        for n in (40, 1024):
            h = torch.from_numpy(wl.h[:n].copy()).cuda()
            send, tags, counts = st.route(h)
            torch.cuda.synchronize()
            m = int(counts[0])
            rows, rtags = send[:m].clone(), tags[:m].clone()
            shared = launches(lambda: capi.check(capi.lib().bivmoe_ep_shared(
                st._h, C.c_void_p(h.data_ptr()), st._stream()), st._h))
            seen[n] = shared, launches(lambda: st.experts(rows, rtags, m))
            st.status()
        assert seen[40][0] == 3                          # dispatch, gate+up, down
        assert seen[1024][0] == 5 + bf16                 # the tcgen05 kernels' two; BF16: the split rows
        assert seen[40][1] == 6                          # localize, sort, dispatch, gate+up, down, combine
        assert seen[1024][1] >= 6 + 2 + 2 + bf16         # the sort in three launches
    finally:
        st.close()
