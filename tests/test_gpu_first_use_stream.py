"""The first solve of a context on a caller's own non-blocking stream: what the
solver sets up on first use (plans, counters) is ready for that stream. The
solution equals, bit for bit, that of a solve on the default stream by another
context."""
import numpy as np
import pytest
import torch

import iceicle_b200 as ib
from specs import BURGERS, NS, Spec
from test_gpu_ilu_tiles import _jacobian

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw,tile", [(dict(pde=NS, nx=5, ny=4, p=3, ip=True), 0), (dict(pde=NS, nx=5, ny=4, p=3, ip=True), 2),
                                     (dict(pde=BURGERS, nx=40, ny=33, p=2), 4), (dict(pde=BURGERS, nx=40, ny=33, p=2), 0)])
def test_first_solve_on_a_stream(kw, tile):
    spec = Spec(**kw)
    x = []
    for stream in (None, torch.cuda.Stream()):
        ctx = spec.context()
        vals, _, _, _ = _jacobian(ctx, spec)
        ctx.ilu_tile = tile
        b = torch.from_numpy(np.random.default_rng(2).standard_normal(ctx.layout.n_dof)).cuda()
        x.append(torch.zeros_like(b))
        torch.cuda.synchronize()
        ctx.gmres_solve(vals, b, x[-1], restart=20, maxit=200, rtol=1e-8, stream=stream)
        torch.cuda.synchronize()
        ctx.close()
    assert torch.isfinite(x[0]).all() and float(x[0].abs().max()) > 0
    assert torch.equal(x[0].view(torch.int64), x[1].view(torch.int64))
