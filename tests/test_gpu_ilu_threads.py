"""Block-ILU(0) applies of several contexts at once, a thread and a stream each:
the contexts need different amounts of shared memory of the same kernel, and
none may see the other's. Every result equals the context's own, alone, bit for
bit."""
import threading

import numpy as np
import pytest
import torch

from specs import BURGERS, NS, Spec
from test_gpu_ilu_tiles import _jacobian

pytestmark = pytest.mark.gpu


def applies(ctx, x, want, n, stream, bad):
    try:
        y = torch.empty_like(x)
        for k in range(n):
            ctx.pc_apply(x, y, 0, stream)
            if k % 200 == 199:
                stream.synchronize()
                if not torch.equal(y.view(torch.int64), want.view(torch.int64)):
                    raise AssertionError("another result than alone")
    except Exception as e:
        bad.append(e)


@pytest.mark.parametrize("kws,tile", [
    ([dict(pde=BURGERS, p=2, g=1, nx=300, ny=3), dict(pde=BURGERS, p=2, g=1, nx=2, ny=3)], 0),  # by strips
    ([dict(pde=NS, p=2, g=1, nx=24, ny=1), dict(pde=NS, p=2, g=1, nx=3, ny=2)], 24),  # factors streamed
    ([dict(pde=NS, p=4, g=1, nx=12, ny=1), dict(pde=NS, p=4, g=1, nx=2, ny=1)], 12),  # staged rows
])
def test_applies_side_by_side(kws, tile):
    runs, bad = [], []
    for kw in kws:
        spec = Spec(**kw)
        ctx = spec.context()
        vals, _, _, _ = _jacobian(ctx, spec)
        ctx.ilu_tile = tile
        ctx.pc_factor(vals, 0)
        x = torch.from_numpy(np.random.default_rng(1).standard_normal(ctx.layout.n_dof)).cuda()
        y = torch.empty_like(x)
        ctx.pc_apply(x, y, 0)
        torch.cuda.synchronize()
        runs.append((ctx, x, y, 6000, torch.cuda.Stream(), bad))
    threads = [threading.Thread(target=applies, args=r) for r in runs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad
    for r in runs:
        r[0].close()
