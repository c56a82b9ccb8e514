"""make_line / line_at (csrc/geometry.h), the per-line form of the packing the
gather and scatter passes use, against decode() position by position: every
parity of the sizes, both packings, compiled for the host."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "compressedsensingipm.jl_b200", "csrc")

PROGRAM = r"""
#include "geometry.h"
#include <cstdio>
using namespace csipm;
int main() {
    const int S[] = {2, 4, 6, 8, 10, 12, 14, 62};
    long seen = 0;
    for (int dim = 2; dim <= 3; ++dim)
        for (int a : S) for (int b : S) for (int c : S) {
            if (dim == 2 && c != 2) continue;
            const int n[3] = {a, b, dim == 3 ? c : 1};
            const Geom g = make_geom(dim, n, a / 2 + 1);
            for (int sol = 0; sol < 2; ++sol)
                for (int i = 0; i <= g.m1; ++i)
                    for (int k = 0; k < g.n3; ++k) {
                        if (sol && i != 0 && i != g.m1) continue;   // interior lines are pairs
                        const LineMap l = make_line(g, i, k, sol);
                        for (int j = 0; j < g.n2; ++j, ++seen) {
                            const MapEntry e = decode(g, i, j, k), f = line_at(l, j);
                            const bool vert = e.kind == KIND_VERT;
                            const int re = sol ? (int)sol_tail(g, e.re) : e.re;
                            const int im = vert ? -1 : (sol ? (int)sol_tail(g, e.im) : e.im);
                            if (re != f.re || im != f.im || e.kind != f.kind || e.src != f.src) {
                                std::printf("dim %d (%d, %d, %d) sol %d at (%d, %d, %d): re %d im %d kind %d src %d, "
                                            "line gives %d %d %d %d\n", dim, a, b, c, sol, i, j, k, re, im, e.kind,
                                            e.src, f.re, f.im, f.kind, f.src);
                                return 1;
                            }
                        }
                    }
        }
    std::printf("%ld positions\n", seen);
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_line_map_equals_decode(tmp_path):
    src = tmp_path / "line.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "line"
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", CSRC, "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
