"""The workspace a context keeps: what calls take for speed alone is bounded, goes back to the device, and a size that
could not be allocated is not asked for again until there is more room (csrc/kq_work.h, compiled with the host
compiler); on the GPU, the memory that the FP64 multishift CG and the residual check leave behind."""
import subprocess
from pathlib import Path

import numpy as np
import pytest
import torch

import kuqcd_b200 as K
from tests.conftest import dev_buffer

ROOT = Path(__file__).resolve().parents[1]
MIB = 1 << 20
KEEP = 512 * MIB

PROGRAM = r"""
#include <cstdio>
#include "kq_work.h"
using kq::WorkPolicy;
int main()
{
    const size_t M = size_t(1) << 20;
    WorkPolicy p;
    // a quarter of the free memory beyond the workspace there is, all of it for share 1
    printf("%d %d %d %d\n", p.may_grow(300 * M, 100 * M, 800 * M, 4), p.may_grow(301 * M, 100 * M, 800 * M, 4),
           p.may_grow(301 * M, 100 * M, 800 * M, 1), p.may_grow(100 * M, 100 * M, 0, 4));
    // a failure at 200 MiB with room for 900: no second try at that size or above until there is more room
    p.note_failure(200 * M, 900 * M);
    printf("%d %d %d %d\n", p.may_grow(199 * M, 0, 900 * M, 4), p.may_grow(200 * M, 0, 900 * M, 4),
           p.may_grow(220 * M, 50 * M, 850 * M, 4), p.may_grow(200 * M, 0, 901 * M, 4));
    // the free memory is looked at for more than 64 MiB, and for anything after a failure
    printf("%d %d %d %d\n", WorkPolicy().asks(164 * M, 100 * M), WorkPolicy().asks(164 * M + 1, 100 * M),
           WorkPolicy().asks(M, 100 * M), p.asks(M, 0));
    // what stays with the context: up to 512 MiB above what the call needs or found
    printf("%d %d %d\n", p.keeps(612 * M, 0, 100 * M), p.keeps(612 * M + 1, 0, 100 * M),
           p.keeps(612 * M + 1, 612 * M + 1, 100 * M));
    printf("%d %d\n", (int)(p.budget(0) / M), (int)(p.budget(700 * M) / M));
    // a limit of the caller's takes the place of the 512 MiB
    WorkPolicy q;
    q.limit = 64 * M;
    printf("%d %d %d %d %d\n", q.may_grow(64 * M, 0, 800 * M, 4), q.may_grow(65 * M, 0, 800 * M, 4),
           q.keeps(612 * M + 1, 0, 0), (int)(q.budget(0) / M), (int)(q.budget(700 * M) / M));
}
"""


def test_policy(tmp_path):
    (tmp_path / "w.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", str(ROOT / "kuqcd_b200" / "csrc"), str(tmp_path / "w.cpp"), "-o",
                    str(tmp_path / "w")], check=True)
    out = subprocess.run([str(tmp_path / "w")], check=True, capture_output=True, text=True).stdout.splitlines()
    assert out == ["1 0 1 1", "1 0 0 1", "0 1 0 1", "1 0 1", "512 700", "1 0 1 64 700"]


def held(before):
    torch.cuda.synchronize()
    return before - torch.cuda.mem_get_info()[0]


@pytest.mark.gpu
def test_memory_left_behind_by_solves_and_checks(cuda):
    """At 48 x 48 x 32 x 32 an FP64 field is 54 MiB: the windowed FP64 solve of 12 shifts works in 30 of them where the
    reference's kernel order needs 15, and the residual check would take 12.  What later allocations of the process cannot
    have is at most 512 MiB above what the calls cannot do without (64 MiB of slack for the kernels' code and the partial
    sums): one allocation of all the rest succeeds, and the next solve works."""
    dims, ns, slack = (48, 48, 32, 32), 12, 64 * MIB
    v = int(np.prod(dims))
    ctx = K.Context(dims)
    rng = np.random.default_rng(1)
    rec = 0.1 * rng.standard_normal(v * 72)
    ctx.load_links(K.KUQCD_FAT_LINK, rec)
    ctx.load_links(K.KUQCD_LONG_LINK, rec)
    del rec
    vb = ctx.spinor_bytes(K.KUQCD_DOUBLE)
    assert 15 * vb > KEEP + slack
    d_b, d_x = dev_buffer(vb), dev_buffer(ns * vb)
    ctx.upload(K.KUQCD_DOUBLE, rng.standard_normal(v // 2 * 6), d_b)
    sig = list(0.01 + np.logspace(-2, 0, ns))
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    first = ctx.true_residuals(0, sig, d_b, d_x)
    assert held(free) <= KEEP + slack
    assert np.allclose(first, 1.0, rtol=1e-12, atol=0)  # x = 0
    solutions = []
    for cap in (64, 64, 3):  # windowed, windowed with what the first left, in the reference's order
        info = ctx.solve_device(d_b, d_x, sig, solver=K.KQ_SOLVER_CGM, tol=0.0, max_iter=cap)
        assert info.kernel_launches == (1 + 32 if cap == 3 else 1 + 8 * 26)
        solutions.append(d_x.cpu())
        rest = torch.empty(free - (ns + 3) * vb - KEEP - slack, dtype=torch.uint8, device="cuda")
        del rest
        torch.cuda.empty_cache()
    assert torch.equal(solutions[0], solutions[1])
    # the explicit windowed solver needs its ring and keeps it; the others then use what is there
    ctx.solve_device(d_b, d_x, sig, solver=K.KQ_SOLVER_CGM_WINDOWED, tol=0.0, max_iter=64)
    assert torch.equal(solutions[0], d_x.cpu())
    ctx.set_workspace_limit(0)
    ring = held(free)
    assert ring >= (ns + 18) * vb
    ctx.true_residuals(0, sig, d_b, d_x)
    ctx.solve_device(d_b, d_x, sig, solver=K.KQ_SOLVER_CGM, tol=0.0, max_iter=64)
    assert abs(held(free) - ring) <= slack
    ctx.close()
