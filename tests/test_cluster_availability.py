"""A cluster's program is used only where the device schedules its own clusters: it is asked with the program's blocks and
memory, not with the walk's (64 KB a block), against a fake of the device's answer."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from gridsim_b200 import synthetic

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "gridsim_b200", "csrc")

HARNESS = r'''
#include "gs_host.h"
using namespace gs;
// 1 where a device with room for clusters of `ctas` blocks of `smem` bytes runs the grid's program; asked[0], asked[1]: the
// blocks and bytes it was asked for.
extern "C" int runs(const gs_grid_desc* d, int ctas, long long smem, long long* asked) {
    HostGrid h;
    Symbolic s;
    if (!CopyGrid(d, h).empty() || !Analyze(h, s, false).empty()) return -1;
    const SharedProgram P = BuildShared(s);
    if (!P.on) return -2;
    asked[0] = asked[1] = 0;
    return SharedRuns(P, [&](int c, size_t b) {
        asked[0] = c;
        asked[1] = (long long)b;
        return c <= ctas && (long long)b <= smem ? 3 : 0;
    });
}
'''


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("avail")
    src, so = d / "avail.cpp", d / "avail.so"
    src.write_text(HARNESS)
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-pthread", "-I", CSRC, "-o", str(so), str(src)]
                          + [os.path.join(CSRC, f) for f in ("gs_symbolic.cpp", "gs_solo.cpp", "gs_host.cpp",
                                                             "gs_topology.cpp", "gs_dc.cpp")])
    return ctypes.CDLL(str(so))


@pytest.mark.parametrize("n_bus,ctas", [(1000, 2), (2000, 4), (4000, 8), (8000, 16)])
def test_the_device_is_asked_for_the_programs_own_clusters(lib, n_bus, ctas):
    m = synthetic.make_grid(n_bus, n_bus + n_bus // 3 + 1, n_bus // 8, seed=5, operating_point=False)  # owns d's arrays
    d = m.desc()
    asked = np.zeros(2, np.int64)
    ask = lambda c, b: lib.runs(ctypes.byref(d), c, ctypes.c_longlong(b), asked.ctypes.data_as(ctypes.c_void_p))
    assert ask(16, 227 * 1024) == 1
    assert asked[0] == ctas and 64 * 1024 < asked[1] <= 226 * 1024
    assert ask(16, 64 * 1024) == 0  # a device where only the walk's clusters fit
    assert ask(ctas // 2, 227 * 1024) == 0
    assert ask(ctas, int(asked[1])) == 1 and ask(ctas, int(asked[1]) - 1) == 0
