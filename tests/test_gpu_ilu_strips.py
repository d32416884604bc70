"""The block-ILU(0) apply by strips of grid rows (the default on whole grids for
blocks up to 36 x 36) against the data-flow apply on completion counters: the
same sums in the same order, so the results are equal bit for bit. Sizes: one
row, one column, fewer rows than a strip, ragged last strips, wide rows, more strips than
a cluster and more than are resident at once; batches of grids; both
precisions; repeated applies (the exchange rows are left ready for the next)."""
import numpy as np
import pytest
import torch

import iceicle_b200 as icx
from iceicle_b200.workloads import advection_diffusion_problem
from specs import BURGERS, NS, Spec

pytestmark = pytest.mark.gpu

CASES = [dict(pde=BURGERS, p=p, g=1, nx=nx, ny=ny) for p in (1, 2, 3, 4)
         for nx, ny in ((1, 1), (1, 19), (23, 1), (7, 5), (12, 33), (3, 90))]
CASES += [dict(pde=NS, p=1, g=1, nx=9, ny=14), dict(pde=NS, p=2, g=1, nx=5, ny=20),
          dict(pde=NS, p=2, g=1, nx=2, ny=300),
          dict(pde=NS, p=2, g=1, nx=400, ny=3)]  # rows too wide for an inbox


def check(ctx, n, precision):
    bs, nnz = ctx.layout.block_size, ctx.layout.nnz_blocks
    rng = np.random.default_rng(nnz)
    rp = None
    vals = torch.from_numpy(rng.standard_normal((nnz, bs, bs)) * (0.3 / bs ** 0.5)).cuda()
    rp, ci = ctx.jacobian_pattern()
    rows = np.repeat(np.arange(len(rp) - 1), np.diff(rp))
    vals[torch.from_numpy(rows == ci).cuda()] += 2.0 * torch.eye(bs, dtype=torch.float64, device="cuda")
    x = torch.from_numpy(rng.standard_normal(n)).cuda()
    ys = [torch.empty_like(x) for _ in range(4)]
    ctx.pc_factor(vals, precision)
    for y in ys[:3]:
        ctx.pc_apply(x, y, precision)
    ctx.tile = {"ilu_sched": [1, 1]}
    ctx.pc_apply(x, ys[3], precision)
    torch.cuda.synchronize()
    for y in ys[:3]:
        assert torch.equal(y.view(torch.int64), ys[3].view(torch.int64))


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("kw", CASES, ids=[str(c) for c in CASES])
def test_strip_apply_bitwise(kw, precision):
    ctx = Spec(**kw).context()
    check(ctx, ctx.layout.n_dof, precision)
    ctx.close()


@pytest.mark.parametrize("p", [2, 4])
def test_strip_apply_batch(p):
    parts = [advection_diffusion_problem(dict(n=n, p=p, mu=0.01, theta=0.3, kx=1, ky=1, phx=0.0, phy=0.0))[0]
             for n in (3, 17, 1, 30)]
    b = icx.batch(parts)
    check(b, b.layout.n_dof, 0)
    b.close()
