"""CPU tests of the launch shapes: grids of the kernels over tiles of sites and groups of systems stay within the
device's limits (2^31 - 1 blocks in x, 65,535 in y and z) on every lattice a context accepts, and cover every site of
every group.  The header that holds the rule is compiled with the host compiler."""
import os
import re
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "kuqcd_b200" / "csrc"
CUDA = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda"))

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "kq_internal.h"
int main(int argc, char **argv)
{
    for (int a = 1; a + 2 < argc; a += 3) {
        const dim3 g = kq::tile_group_grid(atoi(argv[a]), atoi(argv[a + 1]), atoi(argv[a + 2]));
        printf("%u %u %u\n", g.x, g.y, g.z);
    }
}
"""

# sites per parity: 16^4, 64^4, 48^3 x 192, 64^3 x 96, 64^3 x 128, an odd remainder, the most a context accepts
SITES = [32768, 8388608, 10616832, 12582912, 16777216, 8388608 + 1, 1, 2000000000]


@pytest.fixture(scope="module")
def grids(tmp_path_factory):
    d = tmp_path_factory.mktemp("shapes")
    (d / "shapes.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", str(ROOT / "include"), "-I", str(CSRC), "-I", str(CUDA / "include"),
                    str(d / "shapes.cpp"), "-o", str(d / "shapes")], check=True)
    want = [(n, block, ng) for n in SITES for block in (128, 256) for ng in (1, 3, 16)]
    out = subprocess.run([str(d / "shapes"), *(str(v) for w in want for v in w)], check=True, capture_output=True,
                         text=True).stdout.split()
    it = iter(int(v) for v in out)
    return {w: (next(it), next(it), next(it)) for w in want}


def test_tile_group_grids_fit_and_cover(grids):
    for (n, block, ng), (x, y, z) in grids.items():
        assert x <= 2 ** 31 - 1 and (y, z) == (1, 1), (n, block, ng)
        assert x % ng == 0 and x // ng * block >= n > (x // ng - 1) * block, (n, block, ng)


def test_no_kernel_keeps_sites_on_y():
    """A grid ends at 65,535 blocks in y: 128-site tiles of 64^4 reach 65,536 there."""
    for f in sorted(CSRC.glob("*.cu*")):
        assert not re.search(r"blockIdx\.y|gridDim\.y", f.read_text()), f.name
