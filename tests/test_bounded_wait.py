"""The wait of the expert kernels' roles for one another (csrc/bounded_wait.h), on lanes, warps and
barriers that threads of the host play: one answer for all lanes of a warp, and no warp left waiting where
another one gave up."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdio>
#include <mutex>
#include <random>
#include <thread>
#include <vector>
#include "bounded_wait.h"
using namespace bivmoe;
static std::atomic<int> bad{0};
#define CHECK(x) do { if (!(x)) { printf("line %d: %s\n", __LINE__, #x); bad = 1; } } while (0)

// a lane by itself: ready at its ready_at-th try, or told to give up at its late_at-th look
struct One {
    long* tries; long ready_at; long* looks; long late_at;
    bool ready() { return ++*tries >= ready_at; }
    bool late(unsigned look) { CHECK(look == ++*looks); return *looks >= late_at; }
    void pause() {}
};
template <int EVERY> static bool one(long ready_at, long late_at, long* tries, long* looks) {
    *tries = *looks = 0;
    return bounded_wait<EVERY>(One{tries, ready_at, looks, late_at});
}

// lanes of a warp: a vote is complete when every lane has cast its own
struct Vote {
    std::mutex m; std::condition_variable c; int lanes, in = 0; long round = 0; bool all = true, was_all = true;
    bool cast(bool v) {
        std::unique_lock<std::mutex> l(m);
        all = all && v;
        const long r = round;
        if (++in == lanes) { was_all = all; all = true; in = 0; round++; c.notify_all(); }
        else c.wait(l, [&] { return round != r; });
        return was_all;
    }
};
struct Lane : One {
    Vote* vote;
    bool all(bool v) { return vote->cast(v); }
};

// What the warps of a block wait at (a warp is a thread here): an mbarrier's phases, a named barrier
struct Bar {
    std::mutex m; int count, in = 0; unsigned phase = 0;
    void arrive() { std::lock_guard<std::mutex> l(m); if (++in == count) { in = 0; phase++; } }
    bool test(unsigned parity) { std::lock_guard<std::mutex> l(m); return (phase & 1) != parity; }
    unsigned at() { std::lock_guard<std::mutex> l(m); return phase; }
    void sync() {                       // without a bound, as the hardware's
        std::unique_lock<std::mutex> l(m);
        const unsigned p = phase;
        if (++in == count) { in = 0; phase++; return; }
        while (phase == p) { l.unlock(); std::this_thread::yield(); l.lock(); }
    }
};
static uint64_t ms() { return std::chrono::duration_cast<std::chrono::milliseconds>(std::chrono::steady_clock::now().time_since_epoch()).count(); }
struct OnBar {
    Bar* bar; unsigned parity; std::atomic<int>* abort; uint64_t limit_ms = 0, t0 = 0;   // 0: no clock
    bool ready() { return bar->test(parity); }
    bool late(unsigned look) {
        if (limit_ms && look == 1) t0 = ms();
        return abort->load() || (limit_ms && ms() - t0 >= limit_ms);
    }
    void pause() { std::this_thread::yield(); }
};
struct Meeting {
    Bar *met, *left;
    bool all_left() { return left->test(0); }
    void arrive() { met->arrive(); }
};

int main() {
    long tries, looks;
    // at once, after some tries; told to give up: at the first look after that, once in EVERY tries
    CHECK(one<256>(1, 1, &tries, &looks) && tries == 1 && looks == 0);
    CHECK(one<256>(1000, 100, &tries, &looks) && tries == 1000 && looks == 3);
    CHECK(!one<256>(1 << 30, 1, &tries, &looks) && tries == 256);
    CHECK(!one<1>(1 << 30, 7, &tries, &looks) && tries == 7);

    // eight lanes that see their phase, or the flag, at different turns: one answer
    std::mt19937 rng(1);
    for (int run = 0; run < 300; run++) {
        constexpr int LANES = 8;
        Vote vote;
        vote.lanes = LANES;
        long t[LANES] = {}, k[LANES] = {};
        int answer[LANES];
        std::vector<std::thread> lanes;
        for (int l = 0; l < LANES; l++) {
            const long ready_at = 1 + rng() % 40, late_at = run % 2 ? 1 + rng() % 8 : 1 << 30;
            lanes.emplace_back([&, l, ready_at, late_at] {
                answer[l] = bounded_wait_together<4>(Lane{{&t[l], ready_at, &k[l], late_at}, &vote});
            });
        }
        for (auto& l : lanes) l.join();
        for (int l = 0; l < LANES; l++) CHECK(answer[l] == answer[0] && (answer[0] || run % 2));
    }

    // The warps of a block: a feeder fills two slots by its clock, four warps without one work on each
    // stage, meet around a shared tile after every third one, and leave.  One role gives up somewhere, or
    // stops without a word in the middle of its wait; every warp ends.
    for (int run = 0; run < 600; run++) {
        constexpr int WARPS = 4, STAGES = 30;
        std::atomic<int> abort{0}, chunks{0}, tile{0}, ended{0};
        Bar full[2], empty[2], met, left;
        for (int i = 0; i < 2; i++) { full[i].count = 1; empty[i].count = WARPS; }
        met.count = left.count = WARPS;
        const int culprit = run % (WARPS + 2), at = rng() % STAGES;      // the last one: nobody
        const bool silent = run % 20 == 0 && culprit < WARPS, late = run % 3 == 0;
        std::vector<std::thread> roles;
        roles.emplace_back([&] {
            const uint64_t limit = silent ? 20 : 10000;
            bool ok = true;
            for (int q = 0; q < STAGES && ok; q++) {
                ok = !(culprit == WARPS && q == at) && bounded_wait<8>(OnBar{&empty[q & 1], unsigned(((q >> 1) & 1) ^ 1), &abort, limit});
                if (ok) full[q & 1].arrive();
            }
            if (!ok) abort = 1;
            if (!bounded_wait<8>(OnBar{&left, 0, &abort, limit})) abort = 1;   // it stays until they have left
            ended++;
        });
        for (int w = 0; w < WARPS; w++)
            roles.emplace_back([&, w] {
                bool gave_up = true;
                int q = 0;
                for (; q < STAGES; q++) {
                    const bool now = culprit == w && q == at;
                    Bar never;
                    never.count = 2;
                    // the culprit: a wait that nothing ends but the flag; or the flag it raises itself
                    if (now && silent) bounded_wait<8>(OnBar{&never, 0, &abort});
                    if (now || !bounded_wait<8>(OnBar{&full[q & 1], unsigned((q >> 1) & 1), &abort})) break;
                    empty[q & 1].arrive();
                    if (late && culprit == w && abort) std::this_thread::yield();
                    if (q % 3 != 2) continue;
                    tile++;
                    met.sync();
                    CHECK(abort || tile % WARPS == 0);      // the whole tile is there, and nobody writes the next one
                    chunks++;
                    met.sync();
                }
                if (q == STAGES) gave_up = false;
                else abort = 1;
                left.arrive();
                if (gave_up) arrive_until_all_left(Meeting{&met, &left}, 1u << 30);
                ended++;
            });
        for (auto& r : roles) r.join();
        CHECK(ended == WARPS + 1);
        if (culprit > WARPS) CHECK(!abort && chunks == WARPS * STAGES / 3);
        else CHECK(abort);
    }
    printf("done\n");
    return bad;
}
"""


def test_bounded_waits_of_lanes_warps_and_blocks(tmp_path):
    src, exe = tmp_path / "bounded_wait.cpp", tmp_path / "bounded_wait"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-Wall", "-I", os.path.join(ROOT, "biv_b200", "csrc"),
                    "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and "done" in r.stdout, r.stdout + r.stderr
