"""Tiled applies whose dynamic shared memory is just what a launch may have
without raising the kernel's limit, the static memory beside it not counted:
16 x 16 blocks on 16 x 16 tiles (48 KB) and their neighbours. FP32 within 1e-5
and BF16 factors within 5e-2 of the FP64 apply's largest entry, as for the
other tile sizes; the one-lane-per-row form in FP64 within 1e-13."""
import numpy as np
import pytest
import torch

from specs import BURGERS, NS, Spec
from test_gpu_ilu_tiles import _jacobian

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [dict(pde=NS, p=1, nx=16, ny=16, ip=True), dict(pde=BURGERS, p=3, nx=16, ny=16),
                                dict(pde=NS, p=1, nx=17, ny=15, ip=True)])
@pytest.mark.parametrize("tile", [15, 16])
def test_limit(kw, tile):
    spec = Spec(**kw)
    ctx = spec.context()
    vals, _, _, _ = _jacobian(ctx, spec)
    ctx.ilu_tile = tile
    x = torch.from_numpy(np.random.default_rng(3).standard_normal(ctx.layout.n_dof)).cuda()
    y0 = torch.empty_like(x)
    ctx.ilu_apply(vals, x, y0, 0, 1)
    for precision, sched, tol in ((1, 0, 1e-5), (1, 4, 1e-5), (2, 0, 5e-2), (0, 5, 1e-13)):
        ctx.tile = {"ilu_sched": [sched, sched]}
        y = torch.full_like(x, float("nan"))
        ctx.ilu_apply(vals, x, y, precision, 1)
        assert float((y - y0).abs().max()) <= tol * float(y0.abs().max()), (precision, sched)
    ctx.close()
