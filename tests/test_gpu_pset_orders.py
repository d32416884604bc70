"""Sets whose groups apply their preconditioner in different ways at the same
time: Navier-Stokes problems of orders 2 (strips), 3 and 4 (64 x 64 and
100 x 100 blocks: whole-GPU data-flow applies, in turn), and a set on element
tiles. Each part reaches the state of its own solve within 1e-10 (L2,
relative) in as many Newton steps, in FP64 with its GMRES iterations within 2
of it (the dot products of a set are summed in another order; in mixed
precision the single solve keeps its Krylov basis in FP32, the set in FP64),
and replayed steps give the eager ones' states bit for bit."""
import numpy as np
import pytest
import torch

import iceicle_b200 as ib
from specs import NS, Spec

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def parts():
    out = []
    for p, nx, ny in ((2, 6, 5), (3, 4, 3), (4, 3, 3), (3, 5, 2), (4, 2, 4)):
        spec = Spec(pde=NS, nx=nx, ny=ny, p=p, g=2, ip=True, source=True, perturb=0.05)
        out.append((spec.context(), spec.mms_state(spec.coords(), noise=1e-2)))
    return out


@pytest.mark.parametrize("tile", [0, 2])
@pytest.mark.parametrize("precision", [0, 1])
def test_set_equals_parts_alone(parts, precision, tile):
    s = ib.ProblemSet([c for c, _ in parts])
    o = ib.default_newton_options()
    o.tau_abs, o.kmax, o.gmres_rtol, o.gmres_max_it = 1e-10, 20, 1e-8, 5000
    o.precision, o.ilu_tile = precision, tile
    states = []
    for graphs in (1, 0):
        o.cuda_graphs = graphs
        u = torch.from_numpy(s.gather([u0 for _, u0 in parts])).cuda()
        reps, stats = s.newton_solve(u, o)
        assert stats.orders == 3 and (stats.graph_launches > 0) == bool(graphs)
        states.append(u)
    assert torch.equal(states[0].view(torch.int64), states[1].view(torch.int64))
    u = states[0].cpu().numpy()
    for k, (c, u0) in enumerate(parts):
        uk = torch.from_numpy(u0.copy()).cuda()
        rk = c.newton_solve(uk, o)
        assert rk.converged and reps[k].converged, k
        assert reps[k].iterations == rk.iterations, (k, reps[k].iterations, rk.iterations)
        if precision == 0:
            assert abs(reps[k].linear_iterations_total - rk.linear_iterations_total) <= 2, k
        ref = uk.cpu().numpy()
        assert np.linalg.norm(s.part(u, k) - ref) <= 1e-10 * np.linalg.norm(ref), k
    s.close()
