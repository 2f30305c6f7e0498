"""The order of the asynchronous copies of the nonlocal expansion
(csrc/apply_schedule.h, nl_apply_ring_kernel), replayed on the host: a wait sees
only copies that were put in a committed group, so every coefficient slice and
every group of columns must be in a committed group that has been waited for
before it is read, and no buffer may be refilled while it is still read."""
import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "qumasun-workshop-template_b200", "csrc")

PROGRAM = r"""
#include "apply_schedule.h"
#include <cstdio>
#include <vector>
// the kernel's copies for ncol columns: S ring stages of SG columns, slices of CW columns
template <int S, int SG, int CW>
int replay(int ncol) {
    using O = qsb::ApplySchedule<S, CW / SG>;
    const int groups = (ncol + SG - 1) / SG, slices = (ncol + CW - 1) / CW;
    std::vector<int> group_in(groups + S + 2, -1), slice_in(slices + 2, -1);   // commit that holds it; -1: none yet
    int committed = 0, open_slice = -1, bad = 0;
    auto commit = [&](int n) {
        if (n < groups) group_in[n] = committed;
        if (open_slice >= 0) { slice_in[open_slice] = committed; open_slice = -1; }
        ++committed;
    };
    open_slice = 0;
    for (int n = 0; n < O::PROLOGUE; ++n) commit(n);
    for (int n = 0; n < groups; ++n) {
        const int landed = committed - O::PENDING;      // commits 0 .. landed - 1 are complete
        const int sl = n / (CW / SG);
        auto have = [&](int c) { return c >= 0 && c < landed; };
        if (!have(slice_in[sl])) ++bad;                 // coefficients read in this pass
        if (S > 1 && !have(group_in[n])) ++bad;         // columns read in this pass
        if (n % (CW / SG) == 0 && (sl + 1) * CW < ncol) open_slice = sl + 1;   // into the buffer of slice sl - 1
        if (S > 1 && n + O::PROLOGUE - n >= S) ++bad;   // group n + PROLOGUE must not take group n's stage
        commit(n + O::PROLOGUE);
    }
    return bad;
}
int main() {
    int bad = 0;
    for (int ncol = 1; ncol <= 400; ++ncol) bad += REPLAYS;
    std::printf("%d\n", bad);
    return bad != 0;
}
"""


def test_every_slice_is_committed_and_waited_for(tmp_path):
    text = open(os.path.join(CSRC, "nonlocal.cu")).read()
    cw = int(re.search(r"constexpr int APPLY_CW = (\d+);", text).group(1))
    # ApplyCfg's three forms: direct (real FP64), ring of 3 (complex FP64), ring of 5 (FP32)
    assert re.search(r"static constexpr int SG = DIRECT \? 16 : 8;", text)
    assert re.search(r"static constexpr int S = DIRECT \? 0 : \(sizeof\(T\) == 8 \? 3 : 5\);", text)
    calls = " + ".join(f"replay<{s}, {sg}, {cw}>(ncol)" for s, sg in ((0, 16), (3, 8), (5, 8)))
    src = tmp_path / "replay.cpp"
    src.write_text(PROGRAM.replace("REPLAYS", calls))
    exe = tmp_path / "replay"
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)], check=True, capture_output=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
