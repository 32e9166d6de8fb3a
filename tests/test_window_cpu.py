"""The cell windows of a 1D CTA's warps (emu_window.h), replayed on the host
with signed overflow trapped: a warp without particles has no cells and its
deposit no trips whatever the CTA's first cell is; a warp with particles gets
the cells of its stencils, covered by the tiles once each."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HARNESS = r"""
#include "emu_window.h"
#include <climits>
#include <cstdio>

static int bad(const char* what, int a, int b, int c) { std::printf("%s %d %d %d\n", what, a, b, c); return 1; }

int main()
{
    for (int base = -1000; base <= 1000; base++)
        for (int w = 1; w <= 3; w++) {
            const emu::CellRange e = emu::warp_cells(INT_MAX, INT_MIN, base, w);
            if (e.hi >= e.lo || emu::cell_tiles(e.lo, e.hi) != 0) return bad("idle", base, e.lo, e.hi);
            for (int mn = base; mn <= base + 40; mn++)
                for (int mx = mn; mx <= mn + 40; mx += 3) {
                    const emu::CellRange r = emu::warp_cells(mn, mx, base, w);
                    if (r.lo != mn - base || r.hi != mx - base + w - 1) return bad("range", base, mn, mx);
                    const int n = emu::cell_tiles(r.lo, r.hi);
                    if (r.lo + 8 * (n - 1) > r.hi || r.lo + 8 * n <= r.hi) return bad("tiles", base, mn, mx);
                }
        }
    std::printf("ok\n");
    return 0;
}
"""


def test_windows_of_idle_and_busy_warps(tmp_path):
    src, exe = tmp_path / "window.cpp", tmp_path / "window"
    src.write_text(HARNESS)
    subprocess.run(["g++", "-O1", "-std=c++17", "-fsanitize=undefined", "-fno-sanitize-recover=all", "-I",
                    os.path.join(ROOT, "emu_b200", "csrc"), str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
