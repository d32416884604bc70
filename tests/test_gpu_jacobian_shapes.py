"""The FD Jacobian at every compiled (equations, order, geometry order), on the
nodal basis (convective fluxes of the functions off a face taken from the base
flux) and the modal one (all evaluated), with and without second derivatives,
against the oracle's FD Jacobian.

Tolerance: 1e-6 of the largest entry, as for the other Jacobian cases: one-sided
differences with eps = sqrt(machine eps) carry the last bits of the fluxes
amplified by 1 / eps (1e-8 of the fluxes, which for Navier-Stokes exceed the
entries by an order of magnitude)."""
import numpy as np
import pytest
import torch

import oracle_bindings as ob
from specs import BURGERS, NS, Spec

pytestmark = pytest.mark.gpu

CASES = [dict(pde=pde, p=p, g=g, ip=ip, nx=3, ny=2)
         for pde in (BURGERS, NS) for p in (1, 2, 3, 4) for g in (1, 2) for ip in (False, True)]
CASES += [dict(pde=BURGERS, p=4, basis=1, nx=2, ny=2), dict(pde=NS, p=3, basis=1, nx=2, ny=2),
          dict(pde=BURGERS, p=3, sigma_ic=0.5, bct=(3, 2, 4, 3), nx=3, ny=2),
          dict(pde=NS, p=4, ns_flux=2, nx=2, ny=1)]


@pytest.mark.parametrize("kw", CASES, ids=[str(c) for c in CASES])
def test_jacobian_shapes(kw):
    spec = Spec(**kw)
    ctx = spec.context()
    u0 = spec.state(np.random.default_rng(3))
    _, _, _, v_or = ob.jacobian_bsr(spec.oracle_problem(), spec.coords(), u0)
    u = torch.from_numpy(u0).cuda()
    v = torch.full((v_or.size,), float("nan"), dtype=torch.float64, device="cuda")
    ctx.form_jacobian_fd(u, torch.empty_like(u), v)
    err = np.abs(v.cpu().numpy().reshape(v_or.shape) - v_or).max()
    assert err <= 1e-6 * np.abs(v_or).max(), err / np.abs(v_or).max()
    ctx.close()
