"""Block-ILU(0) applies where device memory is short. The packed copies of the
factors that the strip apply reads are extra: a solve that fits without them
runs (by the data-flow apply, the same results bit for bit), and a copy that is
held is given back when the context needs memory for something else."""
import contextlib

import numpy as np
import pytest
import torch

from specs import NS, Spec
from test_gpu_ilu_tiles import _jacobian

pytestmark = pytest.mark.gpu

MARGIN = 16 << 20  # left beside what is counted: 2 MiB units of the allocations
NX = NY = 240      # exchange rows of 33 MB; packed copies, one row per strip, of 3.0 GB (FP64) and 1.5 GB (FP32)
EXCHANGE, PACKED = 2 * NX * NY * 36 * 8, 5 * NX * NY * 36 * 36 * 8


@contextlib.contextmanager
def left(leave):
    """so many bytes of the device are free, the rest is held by one block"""
    torch.cuda.empty_cache()
    hold = torch.empty(torch.cuda.mem_get_info()[0] - leave, dtype=torch.uint8, device="cuda")
    try:
        yield
        torch.cuda.synchronize()
    finally:
        del hold
        torch.cuda.empty_cache()


@pytest.fixture(scope="module")
def problem():
    spec = Spec(pde=NS, nx=NX, ny=NY, p=2, g=1, ip=True)
    ctx = spec.context()
    vals, _, _, _ = _jacobian(ctx, spec)
    x = torch.from_numpy(np.random.default_rng(1).standard_normal(ctx.layout.n_dof)).cuda()
    ys = [torch.empty_like(x) for _ in range(2)]
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    ctx.pc_factor(vals, 0)
    ctx.pc_apply(x, ys[0], 0)
    torch.cuda.synchronize()
    used = free - torch.cuda.mem_get_info()[0]
    ctx.tile = {"ilu_sched": [1, 1]}  # the data-flow kernels are loaded
    ctx.pc_apply(x, ys[0], 0)
    ctx.tile = {"ilu_sched": [2, 2], "ilu_ctas": [1, 1]}
    ctx.pc_apply(x, ys[0], 0)
    ctx.pc_factor(vals, 1)
    ctx.pc_apply(x, ys[1], 1)
    torch.cuda.synchronize()
    ctx.close()
    return spec, vals, x, ys, used


def same(a, b):
    return torch.equal(a.view(torch.int64), b.view(torch.int64))


def test_factors_fit_without_the_copies(problem):
    spec, vals, x, ys, used = problem
    ctx = spec.context()
    y = torch.empty_like(x)
    with left(used - PACKED - EXCHANGE + MARGIN):
        ctx.pc_factor(vals, 0)
        ctx.pc_apply(x, y, 0)
    assert same(y, ys[0])
    ctx.close()


def test_copy_is_given_back(problem):
    spec, vals, x, ys, used = problem
    ctx = spec.context()
    y = torch.empty_like(x)
    ctx.pc_factor(vals, 0)
    ctx.pc_apply(x, y, 0)
    torch.cuda.synchronize()
    assert same(y, ys[0])
    # Jacobian, factors and inverses in FP32, a Krylov basis of 31 vectors, one FP64 vector
    fp32 = 4 * (2 * ctx.layout.nnz_blocks + NX * NY) * 36 * 36 + (4 * 31 + 8) * ctx.layout.n_dof
    with left(fp32 - PACKED + 3 * MARGIN):
        ctx.pc_factor(vals, 1)
        ctx.pc_apply(x, y, 1)
    assert same(y, ys[1])
    ctx.pc_factor(vals, 0)
    ctx.pc_apply(x, y, 0)
    torch.cuda.synchronize()
    assert same(y, ys[0])
    ctx.close()
