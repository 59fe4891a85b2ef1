"""KUQCD_HALF_DSLASH names the HALF kernel for every lattice size.  A periodic copy of a small lattice on a larger one has
the same sum at every site; where both run the same kernel the terms are added in the same order and the results are equal
bit for bit.  Without a name the small lattice runs several threads per site, whose sums are in another order."""
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

import kuqcd_b200 as K
from oracle import oracle as O
from tests.conftest import dev_buffer

ROOT = Path(__file__).resolve().parents[1]
SMALL, LARGE = (8, 8, 8, 8), (24, 24, 24, 24)  # 165,888 sites per parity: two sites per thread by default


def copy_map(parity):
    """Small-lattice site of every site of one parity of the large lattice (checkerboard order)."""
    nx, ny, nz, nt = LARGE
    t, z, y, h = np.meshgrid(*(np.arange(n) for n in (nt, nz, ny, nx // 2)), indexing="ij")
    x = 2 * h + ((y + z + t + parity) & 1)
    a, b, c, d = SMALL
    return ((x % a) // 2 + a // 2 * (y % b + b * (z % c + c * (t % d)))).ravel()


def operators():
    """(dslash, sigma - D D) of the small lattice, and whether the large one's are its copies bit for bit."""
    vs = int(np.prod(SMALL)) // 2
    rec = [r.reshape(2, vs, 72) for r in O.make_links(SMALL, 0.3, 5)]
    maps = [copy_map(0), copy_map(1)]
    src = O.make_source(SMALL, 0, 3).reshape(vs, 6)
    out = []
    for dims, links, s in ((SMALL, rec, src), (LARGE, [np.stack([r[p][maps[p]] for p in (0, 1)]) for r in rec],
                                               src[maps[0]])):
        ctx = K.Context(dims)
        ctx.load_links(K.KUQCD_FAT_LINK, np.ascontiguousarray(links[0]).ravel())
        ctx.load_links(K.KUQCD_LONG_LINK, np.ascontiguousarray(links[1]).ravel())
        nb = ctx.spinor_bytes(K.KUQCD_HALF)
        a, b, t = dev_buffer(nb), dev_buffer(nb), dev_buffer(nb)
        ctx.upload(K.KUQCD_HALF, np.ascontiguousarray(s).ravel(), a)
        ctx.dslash(K.KUQCD_HALF, a, b, 1)
        d = ctx.download(K.KUQCD_HALF, b).reshape(-1, 6)
        ctx.mdagm(K.KUQCD_HALF, 0.37, a, b, t, 0)
        out.append((d, ctx.download(K.KUQCD_HALF, b).reshape(-1, 6)))
        ctx.close()
    (ds, ms), (dl, ml) = out
    return bool(np.array_equal(ds[maps[1]], dl) and np.array_equal(ms[maps[0]], ml))


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["site", "pair4", "pair5", "pair6", "pair7"])
def test_a_named_kernel_runs_on_small_lattices_too(cuda, name):
    r = subprocess.run([sys.executable, "-c", "from tests.test_gpu_half_kernel import operators; print(operators())"],
                       cwd=ROOT, env=dict(os.environ, KUQCD_HALF_DSLASH=name), capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    assert r.stdout.split()[-1] == "True"
