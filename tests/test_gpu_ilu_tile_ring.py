"""Tiled block-ILU(0) apply with the factors streamed through shared memory, at the sizes where its
ring, its chunks and its launch rule change: more tiles than SMs (several CTAs on one, rings of few
slots), levels wider than the ring, ragged tiles, tiles of one row, every block size it runs.

FP64 and FP32 results are the data-flow apply's, bit for bit (the sums are folded in the same
order).  BF16 factors differ from FP64 ones by 2^-9 relative per value: within 5e-2 of the result's
largest entry, as for the other forms.  Repeated applies of one factorisation agree bit for bit.
"""
import numpy as np
import pytest
import torch

from specs import BURGERS, NS, Spec
from test_gpu_ilu_tiles import _jacobian

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw,tile", [
    (dict(pde=NS, nx=100, ny=97, p=2, ip=True), 8),    # 169 tiles
    (dict(pde=NS, nx=33, ny=18, p=2, ip=True), 16),    # levels of 16 elements
    (dict(pde=NS, nx=9, ny=1, p=2, ip=True), 8),
    (dict(pde=NS, nx=17, ny=9, p=3, ip=True), 8),      # 64 x 64 blocks
    (dict(pde=NS, nx=61, ny=40, p=1, ip=True), 3),
    (dict(pde=BURGERS, nx=70, ny=65, p=1), 4),         # 4 x 4 blocks
    (dict(pde=NS, nx=5, ny=4, p=4, ip=True), 4),       # 100 x 100: the other forms
])
def test_streamed_tiles_match_data_flow(kw, tile):
    spec = Spec(**kw)
    ctx = spec.context()
    vals, _, _, _ = _jacobian(ctx, spec)
    ctx.ilu_tile = tile
    x = torch.from_numpy(np.random.default_rng(3).standard_normal(ctx.layout.n_dof)).cuda()
    y64 = None
    for precision in (0, 1):
        ctx.tile = {"ilu_sched": [2, 2]}
        ref = torch.full_like(x, float("nan"))
        ctx.ilu_apply(vals, x, ref, precision, 1)
        ctx.tile = {}
        y = torch.full_like(x, float("nan"))
        ctx.ilu_apply(vals, x, y, precision, 1, repeat=5)
        assert torch.isfinite(ref).all()
        if precision == 0 or ctx.layout.block_size in (16, 36, 64):
            assert torch.equal(ref.view(torch.int64), y.view(torch.int64)), precision
        else:
            assert float((ref - y).abs().max()) <= 1e-5 * float(ref.abs().max())
        y64 = y if precision == 0 else y64
    y16 = [torch.full_like(x, float("nan")) for _ in range(2)]
    for y in y16:
        ctx.ilu_apply(vals, x, y, 2, 1, repeat=5)
    assert torch.equal(y16[0].view(torch.int64), y16[1].view(torch.int64))
    assert float((y16[0] - y64).abs().max()) <= 5e-2 * float(y64.abs().max())
    ctx.close()
