"""Strip applies in which a CTA runs several strips one after the other, carrying
its ring of staged factors and the phases of its barriers on: rows too wide for
an inbox, and more strips than CTAs that are resident. Equal bit for bit to the
data-flow apply on completion counters, three applies in a row."""
import numpy as np
import pytest
import torch

from specs import NS, Spec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,precision", [(365, 160, 0), (580, 152, 1)])
def test_several_strips_per_cta(nx, ny, precision):
    ctx = Spec(pde=NS, p=2, g=1, nx=nx, ny=ny, perturb=0.0).context()
    bs, nnz = ctx.layout.block_size, ctx.layout.nnz_blocks
    g = torch.Generator(device="cuda").manual_seed(nx)
    vals = torch.randn(nnz, bs, bs, dtype=torch.float64, device="cuda", generator=g) * (0.3 / bs ** 0.5)
    rp, ci = ctx.jacobian_pattern()
    diag = np.flatnonzero(np.repeat(np.arange(len(rp) - 1), np.diff(rp)) == ci)
    vals[torch.from_numpy(diag).cuda()] += 2.0 * torch.eye(bs, dtype=torch.float64, device="cuda")
    x = torch.randn(ctx.layout.n_dof, dtype=torch.float64, device="cuda", generator=g)
    ys = [torch.full_like(x, float("nan")) for _ in range(4)]
    ctx.pc_factor(vals, precision)
    for y in ys[:3]:
        ctx.pc_apply(x, y, precision)
    ctx.tile = {"ilu_sched": [1, 1]}
    ctx.pc_apply(x, ys[3], precision)
    torch.cuda.synchronize()
    assert torch.isfinite(ys[3]).all()
    for y in ys[:3]:
        assert torch.equal(y.view(torch.int64), ys[3].view(torch.int64))
    ctx.close()
    del vals
    torch.cuda.empty_cache()
