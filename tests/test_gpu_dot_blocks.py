"""Dot products of the Krylov solver on both sides of the size where the last block adds the blocks'
partial sums itself (a block of 256 rows per SM: 37888 unknowns), and on a single block.  The solution
is checked against a BSR product in numpy: the residual is what the solver reports, to the rounding of
the two products (1e-12 of |b|, rtol 1e-8), and a repeated solve agrees bit for bit."""
import numpy as np
import pytest
import torch

from specs import BURGERS, Spec
from test_gpu_ilu_tiles import _jacobian

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(1, 1), (65, 64), (66, 64)])
def test_solution_on_both_sides_of_the_fused_sum(nx, ny):
    spec = Spec(pde=BURGERS, nx=nx, ny=ny, p=2)
    ctx = spec.context()
    vals, rowptr, colidx, bs = _jacobian(ctx, spec)
    n = ctx.layout.n_dof
    b = torch.from_numpy(np.random.default_rng(8).standard_normal(n)).cuda()
    xs = [torch.zeros_like(b) for _ in range(2)]
    for x in xs:
        _, reported, _ = ctx.gmres_solve(vals, b, x, restart=30, maxit=900, rtol=1e-8, preconditioner=2)
    assert torch.equal(xs[0].view(torch.int64), xs[1].view(torch.int64))
    A, xh, bh = vals.cpu().numpy().reshape(-1, bs, bs), xs[0].cpu().numpy().reshape(-1, bs), b.cpu().numpy()
    Ax = np.zeros_like(xh)
    np.add.at(Ax, np.repeat(np.arange(len(rowptr) - 1), np.diff(rowptr)), np.einsum("bij,bj->bi", A, xh[colidx]))
    true = np.linalg.norm(bh - Ax.reshape(-1)) / np.linalg.norm(bh)
    assert true <= 1e-8 + 1e-12
    assert abs(true - reported) <= 1e-12
    ctx.close()
