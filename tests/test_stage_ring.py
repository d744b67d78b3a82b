"""The operator's stage ring across 2^32 stages (csrc/stage_ring.h), on the CPU:
producer and consumer positions, the phase a reused slot is waited for with, the
x buffers' guards and the drain of a failed launch, against the stage's number
in exact arithmetic, for tiles of 1 to 23 stages starting below 2^32 and 2^33."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = r"""
#include <cstdio>
#include "stage_ring.h"
using namespace qdfn;
static bool at(const RingPos& p, unsigned __int128 n) {
    return p.slot == (uint32_t)(n % kStages) && p.phase() == (uint32_t)(n / kStages & 1);
}
int main() {
    int bad = 0;
    const uint64_t starts[] = {0, (1ull << 32) - 61, (1ull << 33) - 7};
    for (uint64_t n0 : starts) {
        RingFill f;
        f.filled = n0;
        f.at.slot = (uint32_t)(n0 % kStages);
        f.at.round = (uint32_t)(n0 / kStages);   // (wraps as the count does)
        RingPos take = f.at;
        uint64_t n = n0, last[2] = {0, 0};
        bool any[2] = {false, false};
        for (int tile = 0; tile < 200; ++tile) {
            const int len = 1 + tile * 7 % 23, xb = tile & 1;
            for (int q = 0; q < len; ++q, ++n) {
                bad += !at(f.at, n) || !at(take, n) || f.reused() != (n >= (uint64_t)kStages);
                if (q == 0) {
                    const bool in_use = any[xb] && last[xb] + kStages > n;
                    bad += f.x_in_use(xb) != in_use || (in_use && !at(f.last_at[xb], last[xb]));
                }
                if (q == len - 1) { f.mark_last(xb); last[xb] = n; any[xb] = true; }
                f.advance();
                take.next();
                RingPos back = f.at;
                for (int k = 1; k <= kStages && (uint64_t)k <= n + 1; ++k) { back.back(); bad += !at(back, n + 1 - k); }
            }
        }
    }
    printf("%d\n", bad);
    return bad != 0;
}
"""


def test_ring_positions_across_two_to_the_32(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not found")
    src = tmp_path / "ring.cpp"
    src.write_text(SOURCE)
    exe = str(tmp_path / "ring")
    subprocess.run([cxx, "-std=c++17", "-O1", "-Wall", "-I", os.path.join(ROOT, "quake-dfn_gb300", "csrc"), "-o", exe,
                    str(src)], check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
