"""The meeting of warps that share a barrier (csrc/omni_meet.cuh), compiled for the CPU: whichever
warp's wait runs out at whichever item, and whichever warp is held up right behind a barrier while
the others run as far as they can, all leave at the same item and none stays in a barrier.  The four
warps of an epilogue half meet this way; what the softmax warps of the attention do is in
test_attention_schedule_cpu.py."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "cleffa_b200" / "csrc"

PROGRAM = r"""
#include <condition_variable>
#include <cstdio>
#include <mutex>
#include <thread>
#include <vector>
#include "omni_meet.cuh"

enum { WARPS = 4, ITEMS = 5 };

// Barrier over WARPS warps.  A warp that has left never arrives: a meeting that can no longer be
// completed is given up and reported.
struct Half {
    std::mutex m;
    std::condition_variable cv;
    int arrived = 0, generation = 0, left = 0, slow_warp = -1, slow_item = -1;
    bool stuck = false;

    void settle() {                                      // whoever still runs waits in the barrier for warps that never come
        if (left > 0 && arrived + left == WARPS && arrived > 0) { stuck = true; cv.notify_all(); }
    }
    void barrier(int warp, int item) {
        std::unique_lock<std::mutex> l(m);
        const int g = generation;
        if (++arrived == WARPS) { arrived = 0; generation++; }
        settle();
        cv.notify_all();
        cv.wait(l, [&] { return generation != g || stuck; });
        // held up between the barrier and what follows it until all others have left or wait in the next barrier
        if (warp == slow_warp && item == slow_item) cv.wait(l, [&] { return arrived + left == WARPS - 1 || stuck; });
    }
    void leave() {
        std::unique_lock<std::mutex> l(m);
        left++;
        settle();
        cv.notify_all();
    }
};

int main() {
    int bad = 0;
    for (int late = 0; late < WARPS; late++)
        for (int late_item = 0; late_item < ITEMS; late_item++)
            for (int slow = 0; slow < WARPS; slow++)
                for (int slow_item = 0; slow_item < ITEMS; slow_item++) {
                    Half h;
                    h.slow_warp = slow; h.slow_item = slow_item;
                    volatile short quit[2] = {0, 0};
                    int last[WARPS];
                    std::vector<std::thread> t;
                    for (int w = 0; w < WARPS; w++)
                        t.emplace_back([&, w] {
                            int it = 0;
                            auto meet = [&](int item, bool ok) { return warps_meet(quit, item, ok, [&] { h.barrier(w, item); }); };
                            for (; it < ITEMS; it++)
                                if (!meet(it, !(w == late && it == late_item)) || h.stuck) break;
                            last[w] = it;
                            h.leave();
                        });
                    for (auto &x : t) x.join();
                    for (int w = 0; w < WARPS; w++)
                        if (h.stuck || last[w] != late_item) { bad++; break; }
                }
    std::printf("%d\n", bad);
    return bad != 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_all_warps_leave_at_the_same_item(tmp_path):
    src, exe = tmp_path / "meet.cpp", tmp_path / "meet"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-x", "c++", "-I", str(CSRC), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, f"{out.stdout.strip()} schedules leave a warp behind"
