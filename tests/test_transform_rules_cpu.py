"""Host rules of the transform passes, compiled from the library's own header: no GPU call made."""
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "matilda.ft_b200", "csrc")
CUDA = os.environ.get("CUDA", "/usr/local/cuda")

PROGRAM = r"""
#include "tild_device.h"
#include <cstdio>
using namespace tild;
int main()
{
    int nx, nz;
    while (std::scanf("%d %d", &nx, &nz) == 2) {
        Geom g{};
        FftLine ly{};
        g.nx = nx;
        g.nz = nz;
        g.nxh = nx / 2 + 1;
        g.hp = (g.nxh + 3) & ~3;
        g.dhp = make_fastdiv((unsigned)g.hp);
        ly.r1 = 1;
        std::printf("%d %u\n", fft2_columns(g, ly) ? 1 : 0, g.dhp.m);
    }
}
"""


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    (d / "r.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I" + CSRC, "-I" + os.path.join(ROOT, "include"), "-I" + CUDA + "/include",
                    str(d / "r.cpp"), "-o", str(d / "r")], check=True)

    def ask(grids):
        out = subprocess.run([str(d / "r")], input="\n".join("%d %d" % g for g in grids), text=True, check=True,
                             stdout=subprocess.PIPE).stdout.split()
        return [(int(a), int(m)) for a, m in zip(out[::2], out[1::2])]
    return ask


def test_column_division_is_exact_wherever_the_y_pass_is_taken(rule):
    """Every column index of the two-stage y pass, divided as the kernel divides it: exact on
    every grid that the rule accepts (the shared memory of the other passes ends at nx = 8533,
    nz = 1505); 3438 x 1500 and 3910 x 1200, where the division fails, are refused, and every
    box of three two-stage axes is accepted."""
    rng = np.random.default_rng(1)
    grids = [(3438, 1500), (3910, 1200), (256, 256), (256, 1), (8, 8), (2900, 1505), (8533, 235), (8533, 200), (3300, 1505),
             (3373, 1505), (4057, 1040)]
    grids += [(int(rng.integers(6, 8534)), int(rng.integers(1, 1506))) for _ in range(60)]
    wrong = 0
    for (nx, nz), (ok, m) in zip(grids, rule(grids)):
        hp = (nx // 2 + 4) & ~3
        j = np.arange(nz * hp, dtype=np.uint64)
        exact = bool(np.array_equal((j * np.uint64(m)) >> np.uint64(32), j // np.uint64(hp)))
        assert exact or not ok, (nx, nz)
        wrong += not exact
        if nx <= 256 and nz <= 256:
            assert ok
    assert wrong >= 2 and [ok for ok, _ in rule(grids[:2])] == [0, 0]
