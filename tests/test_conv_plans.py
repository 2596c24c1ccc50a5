"""The tilings of the 3x3 convolutions that a thread keeps (csrc/conv_plan.h,
plain C++): a network's layers are searched once, whatever the order of its
shapes and batch sizes, and what is kept is bounded."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INCLUDE = "/usr/local/cuda/include"

PROGRAM = r"""
#include "conv_plan.h"
#include <cstdio>
#include <cstdlib>
using namespace crt;
// the learned denoiser's layers: channels, level; forward and data gradients
static const int kL[11][3] = {{16, 32, 0}, {32, 32, 0}, {32, 64, 1}, {64, 64, 1}, {64, 96, 2}, {96, 96, 2},
                              {160, 64, 1}, {64, 64, 1}, {96, 32, 0}, {32, 32, 0}, {32, 32, 0}};
static int pass(ConvPlans &p, int n, int h, int w, bool train) {
    const long before = p.searches;
    for (int i = 0; i < 11; ++i)
        p.get(n, h >> kL[i][2], w >> kL[i][2], kL[i][0], kL[i][1], !train && i == 10, 148);
    for (int i = 10; train && i > 0; --i) p.get(n, h >> kL[i][2], w >> kL[i][2], kL[i][1], kL[i][0], false, 148);
    return (int)(p.searches - before);
}
int main() {
    ConvPlans p;
    const int sizes[5][3] = {{8, 128, 128}, {32, 256, 256}, {1, 1080, 1920}, {8, 64, 64}, {4, 96, 96}};
    for (int r = 0; r < 3; ++r)
        for (const auto &s : sizes)
            for (int train = 0; train < 2; ++train) printf("%d ", pass(p, s[0], s[1], s[2], train));
    ConvPlans q;  // a batch size of its own for every pass, then all again
    for (int r = 0; r < 2; ++r) {
        int searched = 0;
        for (int n = 1; n <= 32; ++n) searched += pass(q, n, 128, 128, true);
        printf("%d ", searched);
    }
    size_t most = 0;
    ConvPlans b;
    for (int w = 1; w <= 5000; ++w) {
        b.get(1, 8, w, 32, 32, false, 148);
        if (b.size() > most) most = b.size();
    }
    // what is given back is the search's own answer
    const auto a = b.get(1, 8, 77, 32, 32, false, 148).second, c = conv_plan(conv_order(32, 32, 77), 1, 8, 77, 32, 32, 148, false);
    printf("%zu %d\n", most, a.R == c.R && a.Ws == c.Ws && a.grid == c.grid && a.S == c.S && a.KCs == c.KCs);
}
"""


@pytest.mark.skipif(shutil.which("g++") is None or not os.path.isdir(CUDA_INCLUDE), reason="no compiler")
def test_layers_are_searched_once(tmp_path):
    src, exe = tmp_path / "plans.cpp", tmp_path / "plans"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", os.path.join(ROOT, "cudaraytracer_b200", "csrc"), "-I",
                    CUDA_INCLUDE, str(src), "-o", str(exe)], check=True)
    got = [int(v) for v in subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()]
    first, again = got[:10], got[10:30]
    assert all(0 < s <= 21 for s in first) and not any(again)
    assert 0 < got[30] <= 32 * 21 and got[31] == 0
    assert 0 < got[32] <= 1024 and got[33] == 1
