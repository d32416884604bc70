"""Which form applies tiled factors on either side of the lines of the rule: few
elements per tile in few and in many rounds over the SMs, and 16 x 16 blocks on
wide levels. FP64 equals the data-flow apply bit for bit on both sides; FP32 is
within 1e-5 and BF16 within 5e-2 of it, and repeated applies agree bit for
bit."""
import numpy as np
import pytest
import torch

from specs import BURGERS, NS, Spec
from test_gpu_ilu_tiles import _jacobian

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw,tile", [
    (dict(pde=BURGERS, p=1, nx=7, ny=3), 1), (dict(pde=BURGERS, p=1, nx=90, ny=85), 4),
    (dict(pde=BURGERS, p=1, nx=90, ny=85), 5), (dict(pde=BURGERS, p=3, nx=50, ny=49), 2),
    (dict(pde=BURGERS, p=3, nx=20, ny=21), 1), (dict(pde=BURGERS, p=3, nx=16, ny=17), 16),
    (dict(pde=BURGERS, p=3, nx=35, ny=17), 17), (dict(pde=BURGERS, p=3, nx=41, ny=40), 40),
    (dict(pde=NS, p=2, nx=5, ny=4), 1), (dict(pde=NS, p=2, nx=7, ny=1), 8), (dict(pde=NS, p=2, nx=8, ny=1), 8),
    (dict(pde=NS, p=2, nx=41, ny=39), 2), (dict(pde=NS, p=3, nx=11, ny=1), 12), (dict(pde=NS, p=3, nx=12, ny=2), 12),
], ids=str)
def test_both_sides(kw, tile):
    spec = Spec(ip=kw["pde"] == NS, **kw)
    ctx = spec.context()
    vals, _, _, _ = _jacobian(ctx, spec)
    ctx.ilu_tile = tile
    x = torch.from_numpy(np.random.default_rng(3).standard_normal(ctx.layout.n_dof)).cuda()
    ref = torch.full_like(x, float("nan"))
    ctx.tile = {"ilu_sched": [2, 2]}
    ctx.ilu_apply(vals, x, ref, 0, 1)
    ctx.tile = {}
    for precision, tol in ((0, 0.0), (1, 1e-5), (2, 5e-2)):
        ys = [torch.full_like(x, float("nan")) for _ in range(2)]
        for y in ys:
            ctx.ilu_apply(vals, x, y, precision, 1, repeat=3)
        assert torch.equal(ys[0].view(torch.int64), ys[1].view(torch.int64)), precision
        assert float((ys[0] - ref).abs().max()) <= tol * float(ref.abs().max()), precision
    ctx.close()
