"""Work-item sizes up to the largest a caller can ask for.

p9idg_plan_set_chunking takes any int32, and the FP32 mode's tensor-core form multiplies it by up to
32, so the planner's size is 64 bits.  A size past every subgrid's length means "do not split": one
item per subgrid, in a finite list.  The planner is compiled on its own and run with a memory limit
and a time limit.
"""
import os
import resource
import shutil
import subprocess

import pytest

from conftest import ROOT, entry

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "p9idg_internal.h"
using namespace p9idg;
int main(int argc, char **argv) {
    std::vector<p9idg_subgrid> subs(3);
    const int32_t counts[3] = {1024, 0, 7};
    for (int i = 0; i < 3; i++) {
        subs[i] = p9idg_subgrid{};
        subs[i].time_sample_start = 10 * i;
        subs[i].time_sample_count = counts[i];
    }
    std::vector<DevSubgrid> dsub;
    std::vector<WorkItem> items;
    build_work_items(subs, std::atoi(argv[1]), std::atoll(argv[2]), dsub, items);
    for (const auto &w : items) std::printf("%d %d %d\n", w.subgrid, w.t0, w.nt);
    return argc == 3 ? 0 : 1;
}
"""


@pytest.fixture(scope="module")
def planner(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("work_items")
    (d / "main.cpp").write_text(PROGRAM)
    csrc = os.path.join(entry.PKG_DIR, "csrc")
    subprocess.run([gxx, "-std=c++17", "-O1", "-pthread", "-I", os.path.join(ROOT, "include"), "-I", csrc,
                    str(d / "main.cpp"), os.path.join(csrc, "planner.cpp"), "-o", str(d / "planner")], check=True,
                   capture_output=True, text=True)
    return str(d / "planner")


@pytest.mark.parametrize("nch", [1, 3, 4, 8, 16])
@pytest.mark.parametrize("size", [1 << 14, 1 << 27, 1 << 30, (1 << 31) - 1])
@pytest.mark.parametrize("factor", [1, 4, 32])
def test_large_sizes_do_not_split(planner, nch, size, factor):
    limit = 1 << 30
    r = subprocess.run([planner, str(nch), str(size * factor)], capture_output=True, text=True, timeout=60,
                       preexec_fn=lambda: resource.setrlimit(resource.RLIMIT_AS, (limit, limit)))
    assert r.returncode == 0, r.stderr[-300:]
    assert r.stdout.split("\n")[:-1] == ["0 0 1024", "2 20 7"]
