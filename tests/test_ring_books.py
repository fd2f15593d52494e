"""A kernel that ends lets every bulk copy it issued land first.  The books a producer keeps for that
(rg_ring.cuh) are run on the host against a model of the FP32 band iteration: stages with a band copy and, for
interior tiles, windows, the next iteration's first band blocks issued ahead, and a wait that gives up
at every possible point.  Afterwards each stage's barrier has got exactly the bytes it was armed for, and
every armed tile was waited for."""
import shutil
import subprocess

import pytest

from conftest import PKG_DIR

MODEL = r"""
#include <cstdio>
#include <cstdlib>
#include <set>
#include <vector>
#include "rg_ring.cuh"
// tiles 1 and 2 from either end have no windows; my tiles are grid b, b + G, ... forwards or backwards
static int run(int ntiles, int grid, int block, int stages, int iters, int fail_at, bool odd_start)
{
    const int my = block < ntiles ? (ntiles - 1 - block) / grid + 1 : 0;
    auto tile_of = [&](int k, bool back) { const int b = back ? ntiles - 1 - block : block; return back ? b - k * grid : b + k * grid; };
    auto interior = [&](int t) { return t >= 2 && t < ntiles - 2; };
    rg::RingBooks ring;
    std::vector<int> armed(stages, 0), got(stages, 0);
    std::vector<long long> latest(stages, -1);
    int step = 0;
    bool failed = false, odd = odd_start;
    auto band = [&](long long c, int k, bool back) {
        if (step++ == fail_at) return false;  // the wait for an empty stage gave up
        const int st = (int)(c % stages);
        if (armed[st] != got[st]) exit(3);    // a stage is refilled only when its phase is complete
        armed[st] += 1 + (interior(tile_of(k, back)) ? 10 : 0);
        got[st] += 1;
        latest[st] = c;
        ring.issued = c + 1;
        return true;
    };
    auto windows = [&](long long c, int k, bool back) {
        if (interior(tile_of(k, back))) got[c % stages] += 10;
        ring.windowed = c + 1;
    };
    long long base = 0;
    for (int it = 0; it < iters && !failed; ++it) {
        for (int k = 0; k < my && !failed; ++k) {
            if (ring.issued <= base + k && !band(base + k, k, odd)) { failed = true; break; }
            windows(base + k, k, odd);
        }
        if (it + 1 < iters && !failed) {
            ring.ahead(base + my, !odd);
            for (int k = 0; k < stages && k < my && !failed; ++k) failed = !band(base + my + k, k, !odd);
        }
        base += my;
        if (step > fail_at + 1000) return 9;
        if (rand() % 3 == 0 && it + 1 < iters) break;  // stopped by the exchange: converged, or another CTA gave up
        odd = !odd;
    }
    std::set<long long> waited;
    ring.drain(stages, windows, [&](long long c) { waited.insert(c); });
    for (int st = 0; st < stages; ++st) {
        if (armed[st] != got[st]) return 1;
        if (latest[st] >= 0 && !waited.count(latest[st])) return 2;
    }
    return 0;
}
int main()
{
    int n = 0;
    for (int ntiles = 1; ntiles < 24; ++ntiles)
        for (int grid = 1; grid < 6; ++grid)
            for (int block = 0; block < grid; ++block)
                for (int stages = 2; stages <= 3; ++stages)
                    for (int fail = 0; fail < 40; ++fail, ++n) {
                        const int r = run(ntiles, grid, block, stages, 5, fail, fail & 1);
                        if (r) { printf("ntiles %d grid %d block %d stages %d fail %d: %d\n", ntiles, grid, block, stages, fail, r); return 1; }
                    }
    printf("ok %d\n", n);
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no C++ compiler")
def test_every_armed_copy_is_completed_and_waited_for(tmp_path):
    (tmp_path / "model.cpp").write_text(MODEL)
    exe = tmp_path / "model"
    subprocess.run(["g++", "-std=c++17", "-O1", "-x", "c++", "-I", PKG_DIR + "/csrc", "-o", str(exe), str(tmp_path / "model.cpp")],
                   check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.startswith("ok"), out.stdout
