"""The end of a CTA that gave up (csrc/omni_land.cuh), compiled for the CPU: copies in flight are waited for, and whichever of the two
producers of a stage had announced its copies when it all stopped, the time this may take is one limit for the CTA and not
one per stage.  Weights and tokens of a stage share a barrier, so a stage that only one of them announced never completes.  The second
CTA of a pair announces nothing itself: its copies may be in flight with no phase to wait for."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "cleffa_b200" / "csrc"

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "omni_land.cuh"

enum { STAGES = 7, TICK = 100, LIMIT = 50000, SETTLE = 1000 };      // a poll or a look at the clock takes TICK

static uint64_t rnd(uint64_t n) { return (uint64_t)rand() % n; }

int main() {
    int bad = 0;
    for (int run = 0; run < 20000; run++) {
        srand(run);
        volatile int armed[2 * STAGES];
        const bool second = rnd(4) == 0;             // CTA of a pair
        uint64_t at[STAGES], last = rnd(SETTLE);     // when the stage's phase completes; when the last copy lands, announced or not
        bool lost[STAGES], any = false;              // announced by one producer only, or a copy that never comes
        for (int s = 0; s < STAGES; s++) {
            const int phase = (int)rnd(2), who = second ? 0 : (int)rnd(4);
            armed[s] = who & 1 ? phase : -1;
            armed[STAGES + s] = who & 2 ? phase : -1;
            lost[s] = who != 3 || rnd(8) == 0;
            at[s] = rnd(LIMIT * 3 / 4);
            if (who) { any = any || lost[s]; if (!lost[s] && at[s] > last) last = at[s]; }
        }
        uint64_t now = 0;
        bool polled_unarmed = false;
        auto landed = [&](int i, int parity) {
            now += TICK;
            const int s = i % STAGES;
            polled_unarmed |= armed[i] < 0 || parity != armed[i];
            return !lost[s] && now >= at[s];
        };
        copies_land(armed, 2 * STAGES, landed, [&] { now += TICK; return now; }, (uint64_t)LIMIT, (uint64_t)SETTLE);
        const uint64_t slack = SETTLE + (2 * STAGES + 2) * 3 * TICK;
        if (polled_unarmed || now < last || now > (any ? (uint64_t)LIMIT : last) + slack) bad++;
    }
    std::printf("%d\n", bad);
    return bad != 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_copies_are_waited_for_within_one_limit(tmp_path):
    src, exe = tmp_path / "land.cpp", tmp_path / "land"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-x", "c++", "-I", str(CSRC), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, f"{out.stdout.strip()} ends take too long, leave a copy in flight or poll one that was not announced"
