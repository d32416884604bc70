"""The block-ILU(0) factorisation at every compiled block size (matrix-instruction
and odd sizes, the one with two operand buffers), with blocks that need row
exchanges, against NumPy: the apply of the factors is (L U)^-1 x of the ILU(0)
computed block by block with numpy.linalg.inv. Tolerance: the elements' chains
are at most 7 long and the blocks' condition numbers below 100, so 64-bit sums
of at most 100 terms leave the two results within 1e-11 of each other
(100 terms x 100 x 7 x 1.1e-16). A singular diagonal block is refused."""
import numpy as np
import pytest
import torch

import iceicle_b200 as icx
from specs import BURGERS, NS, Spec

pytestmark = pytest.mark.gpu

SIZES = [(pde, p) for pde in (BURGERS, NS) for p in (1, 2, 3, 4)]


def problem(pde, p, nx=4, ny=4):
    ctx = Spec(pde=pde, p=p, g=1, nx=nx, ny=ny).context()
    bs = ctx.layout.block_size
    rp, ci = ctx.jacobian_pattern()
    rng = np.random.default_rng(bs)
    A = rng.standard_normal((len(ci), bs, bs)) * (0.2 / bs ** 0.5)
    for e in range(len(rp) - 1):
        for k in range(rp[e], rp[e + 1]):
            if ci[k] == e:  # a scaled permutation: every pivot needs an exchange
                A[k] += 2.0 * np.eye(bs)[rng.permutation(bs)]
    return ctx, bs, rp, ci, A, rng.standard_normal(ctx.layout.n_dof)


@pytest.mark.parametrize("pde,p", SIZES)
def test_factor_and_apply(pde, p):
    ctx, bs, rp, ci, A, x = problem(pde, p)
    E = len(rp) - 1
    at = {(e, ci[k]): A[k].copy() for e in range(E) for k in range(rp[e], rp[e + 1])}
    inv = {}
    for e in range(E):
        for k in [c for c in ci[rp[e]:rp[e + 1]] if c < e]:
            at[e, k] = at[e, k] @ inv[k]
            at[e, e] = at[e, e] - at[e, k] @ at[k, e]
        inv[e] = np.linalg.inv(at[e, e])
    f, y = x.reshape(E, bs).copy(), np.zeros((E, bs))
    for e in range(E):
        for k in [c for c in ci[rp[e]:rp[e + 1]] if c < e]:
            f[e] -= at[e, k] @ f[k]
    for e in reversed(range(E)):
        s = f[e].copy()
        for k in [c for c in ci[rp[e]:rp[e + 1]] if c > e]:
            s -= at[e, k] @ y[k]
        y[e] = inv[e] @ s
    ctx.pc_factor(torch.from_numpy(A.reshape(-1)).cuda(), 0)
    z = torch.empty(x.size, dtype=torch.float64, device="cuda")
    ctx.pc_apply(torch.from_numpy(x).cuda(), z, 0)
    torch.cuda.synchronize()
    err = np.linalg.norm(z.cpu().numpy() - y.reshape(-1)) / np.linalg.norm(y)
    assert err <= 1e-11, err
    ctx.close()


@pytest.mark.parametrize("pde,p", [(BURGERS, 2), (NS, 2), (NS, 4)])
def test_singular_block_is_refused(pde, p):
    ctx, bs, rp, ci, A, x = problem(pde, p, 1, 1)
    A[0][:, 1] = 0.0
    with pytest.raises(icx.IcxError):
        ctx.pc_factor(torch.from_numpy(A.reshape(-1)).cuda(), 0)
    ctx.close()
