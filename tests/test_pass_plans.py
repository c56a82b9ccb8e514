"""Plans and tiles of the run-time-plan passes (csrc/plan.cu, lay_pass in
csrc/passes.cuh): every plan they are given fits the stage tables of a pass's
arguments, and a longer one (the plans of rows transformed in place) is refused
before anything is written.  Host code, compiled by nvcc and run without a GPU."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "compressedsensingipm.jl_b200", "csrc")

PROGRAM = r"""
#include "passes.cuh"
#include <cstdio>
#include <cstring>
using namespace csipm;
struct Box {
    PassCfg c;
    unsigned char guard[256];   // 6 more stages of each direction would fit
};
// an in-place plan, or one of the passes' own, through lay_pass
int lay(const FftPlanDev& p, size_t csize, bool* taken) {
    Box* b = new Box;
    std::memset(b->guard, 0xa5, sizeof(b->guard));
    lay_pass(p, 2 * p.L, 1, 4, PASS_ROWS, 256, csize, &b->c);
    *taken = b->c.smem <= PASS_SMEM;
    int touched = b->c.tb != 1 || (*taken && b->c.tiles != 4);
    for (unsigned char g : b->guard) touched |= g != 0xa5;
    delete b;
    return touched;
}
int main() {
    int bad = 0, refused = 0, most = 0;
    for (int L = 1; L <= 25600; ++L) {
        FftPlanDev p;
        std::string err;
        bool taken = false;
        for (int row = 0; row < 2; ++row) {
            if (!(row ? make_row_plan(L, &p, &err) : make_fft_plan(L, &p, &err))) continue;
            most = std::max(most, p.nst);
            for (size_t csize : {(size_t)8, (size_t)16}) bad += lay(p, csize, &taken);
        }
        if (!make_fft_plan_ip(L, &p, &err)) continue;
        for (size_t csize : {(size_t)8, (size_t)16}) {
            bad += lay(p, csize, &taken);
            if (p.nst > PASS_STAGES) { bad += taken; ++refused; }
        }
    }
    std::printf("most stages %d, refused %d, bad %d\n", most, refused, bad);
    return bad == 0 && most == PASS_STAGES && refused > 0 ? 0 : 1;
}
"""


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="no nvcc")
def test_plans_fit_the_stage_tables(tmp_path):
    src = tmp_path / "plans.cu"
    src.write_text(PROGRAM)
    exe = tmp_path / "plans"
    subprocess.run(["nvcc", "-std=c++17", "--expt-relaxed-constexpr", "-gencode", "arch=compute_100a,code=sm_100a", "-I", CSRC,
                    "-o", str(exe), str(src), os.path.join(CSRC, "plan.cu")], check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
