"""What building the shared-memory programs costs a grid's creation, on the CPU, against the grid's own analysis (the best of
five of each): a block's program at most a quarter of it, and next to nothing for grids past a cluster's memory, which get
none. (Built beside the uploads, which take about as long.)"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from gridsim_b200 import synthetic

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "gridsim_b200", "csrc")

HARNESS = r'''
#include <algorithm>
#include <chrono>
#include "gs_host.h"
using namespace gs;
static double Ms() {
    return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now().time_since_epoch()).count();
}
// ms[0]: the analysis, ms[1]: the programs (the best of five); the blocks of the grid's program, 0 = none
extern "C" int build(const gs_grid_desc* d, int qlim, double* ms) {
    HostGrid h;
    if (!CopyGrid(d, h).empty()) return -1;
    int blocks = 0;
    ms[0] = ms[1] = 1e30;
    for (int r = 0; r < 5; r++) {
        Symbolic s;
        const double t0 = Ms();
        if (!Analyze(h, s, qlim != 0).empty()) return -2;
        const double t1 = Ms();
        const SoloProgram P = BuildSolo(s);
        SharedProgram Q;
        if (!P.on) Q = BuildShared(s);
        ms[0] = std::min(ms[0], t1 - t0);
        ms[1] = std::min(ms[1], Ms() - t1);
        blocks = P.on ? 1 : Q.ctas;
    }
    return blocks;
}
'''


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("build")
    src, so = d / "build.cpp", d / "build.so"
    src.write_text(HARNESS)
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-pthread", "-I", CSRC, "-o", str(so), str(src)]
                          + [os.path.join(CSRC, f) for f in ("gs_symbolic.cpp", "gs_solo.cpp", "gs_host.cpp",
                                                             "gs_topology.cpp", "gs_dc.cpp")])
    return ctypes.CDLL(str(so))


@pytest.mark.parametrize("n_bus,qlim,blocks,share", [(300, 0, 1, 0.25), (700, 0, 1, 0.25), (10000, 1, 0, 0.01),
                                                     (12000, 0, 0, 0.01)])
def test_programs_cost_little_beside_the_analysis(lib, n_bus, qlim, blocks, share):
    m = synthetic.make_grid(n_bus, int(round(1.37 * n_bus)), int(round(0.12 * n_bus)), seed=3, operating_point=False)
    d = m.desc()
    ms = np.zeros(2)
    assert lib.build(ctypes.byref(d), qlim, ms.ctypes.data_as(ctypes.c_void_p)) == blocks
    assert ms[1] <= share * ms[0], ms
