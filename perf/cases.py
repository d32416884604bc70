"""The performance cases of the framework: its main calls over the sizes that users run.

A case names a kind of call and its sizes:

  residual   R(u) into device memory: what every solver here evaluates most often
  jacobian   the finite-difference Jacobian in BSR (FP64, or with FP32 flux quadrature)
  spmv       the BSR product of an assembled Jacobian (the operator of an assembled Krylov solve)
  factor     block-ILU(0): factors of a Jacobian and one apply of them (the set-up of each Newton step)
  apply      the apply of factors in hand (once per Krylov step), on element tiles
  newton     a whole Newton solve, from the initial state to |R| <= 1e-10
  pset       a Newton solve of a set of independent problems of uneven size and order
  mdg        MDG-ICE: the residual and Jacobian of [u; x] that each Levenberg-Marquardt step forms

prepare() makes what such a program holds before the call (the set-up Context, states, a
Jacobian), run() is the call, exact() the same result in 64 bits in plain torch.
"""
import ctypes as C
import math

import numpy as np
import torch

import iceicle_b200 as ib

GAMMA, PR, MU, MACH, AMP, U0, V0 = 1.4, 0.72, 0.01, 0.3, 0.1, 1.0, 0.5
PINF = (U0 * U0 + V0 * V0) / (GAMMA * MACH * MACH)
BURGERS_MU, BURGERS_B, BURGERS_IN, BURGERS_SRC = 1e-2, (1.0, 0.5), 0.25, 0.2  # boundary value, source amplitude
DEV = "cuda"


# ------------------------------------------------------------------- cases
def listed():
    return [
        # the smallest mesh of the benchmark: launches and latency
        dict(name="residual_burgers_32x32_p2", kind="residual", pde="burgers", nx=32, ny=32, p=2, g=2, flux="upwind",
             ip=False),
        # the headline workload: the manufactured Navier-Stokes solution at 2^20 unknowns
        dict(name="residual_ns_128x128_p3", kind="residual", pde="ns", nx=128, ny=128, p=3, g=2, flux="vanleer",
             ip=True),
        # a ragged large mesh of the highest order, with the DDG flux (second derivatives) and Roe's solver
        dict(name="residual_ns_ddg_193x167_p4", kind="residual", pde="ns", nx=193, ny=167, p=4, g=2, flux="roe",
             ip=False),
        # a linearisation of the headline order
        dict(name="jacobian_ns_64x64_p3", kind="jacobian", pde="ns", nx=64, ny=64, p=3, g=2, flux="vanleer", ip=True,
             f32=False),
        # FP32 flux quadrature on a ragged mesh of the preconditioned solves' order
        dict(name="jacobian_ns_f32_131x77_p2", kind="jacobian", pde="ns", nx=131, ny=77, p=2, g=2, flux="vanleer",
             ip=True, f32=True),
        # the operator of the assembled solve on the largest mesh of the benchmark
        dict(name="spmv_ns_256x256_p2", kind="spmv", pde="ns", nx=256, ny=256, p=2, g=2, flux="vanleer", ip=True),
        # the set-up of a Newton step with the default preconditioner (ILU(0) of the whole grid, FP64)
        dict(name="factor_ns_96x96_p3", kind="factor", pde="ns", nx=96, ny=96, p=3, g=2, flux="vanleer", ip=True,
             tile=0),
        # the preconditioner of the solves on element tiles, on the largest mesh
        dict(name="apply_tiled_ns_256x256_p2", kind="apply", pde="ns", nx=256, ny=256, p=2, g=2, flux="vanleer",
             ip=True, tile=8),
        # a small whole solve with the default options
        dict(name="newton_burgers_32x32_p2", kind="newton", pde="burgers", nx=32, ny=32, p=2, g=2, flux="upwind",
             ip=False, precision=0, tile=0, matrix_free=False),
        # the fastest options of a large solve: BF16 factors on tiles, matrix-free operator
        dict(name="newton_ns_128x128_p2_tiled", kind="newton", pde="ns", nx=128, ny=128, p=2, g=2, flux="vanleer",
             ip=True, precision=3, tile=8, matrix_free=True),
        # independent advection-diffusion problems of orders 1 to 4 and 8 to 96 elements a side, as one set
        dict(name="pset_16", kind="pset", parts=16, n_lo=8, n_hi=96),
        # a shock-aligning solve's linearisation, all interior traces selected
        dict(name="mdg_64x64_p1", kind="mdg", nx=64, ny=64, p=1),
    ]


def draw(rng):
    """one more case of the same kinds, sizes between the listed extremes"""

    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["residual", "residual", "residual", "jacobian", "jacobian", "spmv", "factor", "apply",
                       "newton", "newton", "pset", "mdg"])
    if kind == "pset":
        lo = rng.randint(8, 16)
        return dict(kind=kind, parts=rng.randint(6, 16), n_lo=lo, n_hi=rng.randint(lo + 8, 80))
    if kind == "mdg":
        return dict(kind=kind, nx=size(12, 64), ny=size(12, 64), p=1)
    pde = rng.choice(["burgers", "ns", "ns"])
    p, g = rng.choice([1, 2, 3, 4]), rng.choice([1, 2, 2])
    flux = "upwind" if pde == "burgers" else rng.choice(["vanleer", "vanleer", "roe"])
    c = dict(kind=kind, pde=pde, nx=0, ny=0, p=p, g=g, flux=flux, ip=rng.random() < 0.6)
    if kind == "residual":
        top = 180 if p == 4 else 256
        c.update(nx=size(16, top), ny=size(16, top))
    elif kind == "jacobian":
        top = {1: 160, 2: 110, 3: 64, 4: 40}[p]
        c.update(nx=size(12, top), ny=size(12, top), f32=rng.random() < 0.35)
    elif kind in ("spmv", "apply"):
        top = {1: 256, 2: 220, 3: 128, 4: 80}[p]
        c.update(nx=size(32, top), ny=size(32, top))
        if kind == "apply":
            c.update(tile=rng.choice([8, 8, 16]))
    elif kind == "factor":
        top = {1: 160, 2: 128, 3: 90, 4: 56}[p]
        c.update(nx=size(16, top), ny=size(16, top), tile=rng.choice([0, 0, 8]))
    else:
        fast = rng.random() < 0.5
        # the manufactured solution and the smooth Burgers state: orders 1 to 3, meshes that converge in a few steps
        p = min(p, 3)
        top = {1: 96, 2: 72, 3: 48}[p]
        c.update(p=p, nx=size(16, top), ny=size(16, top), precision=rng.choice([1, 3]) if fast else 0,
                 tile=8 if fast else 0, matrix_free=fast and rng.random() < 0.5)
        if pde == "ns":
            c.update(flux="vanleer", ip=True)
    return c


# -------------------------------------------------- problems: plain numpy
def gauss(n):
    return np.polynomial.legendre.leggauss(n)


def lagrange(order, x, deriv=0):
    """[len(x), order + 1]: the equispaced Lagrange polynomials of [-1, 1], or their deriv-th derivatives"""
    nodes = np.linspace(-1.0, 1.0, order + 1)
    out = np.zeros((len(x), order + 1))
    for k in range(order + 1):
        poly = np.poly1d([1.0])
        for j in range(order + 1):
            if j != k:
                poly = poly * np.poly1d([1.0, -nodes[j]]) / (nodes[k] - nodes[j])
        out[:, k] = np.polyval(np.polyder(poly, deriv) if deriv else poly, x)
    return out


def lattice(nx, ny, g):
    """node coordinates of the unit square, x fastest"""
    x, y = np.meshgrid(np.linspace(0.0, 1.0, nx * g + 1), np.linspace(0.0, 1.0, ny * g + 1))
    return np.stack([x.ravel(), y.ravel()], axis=1)


def smooth_move(xy, nx, ny, amp, rng):
    """a smooth displacement of the nodes by amp element widths, zero on the boundary"""
    bump = np.sin(np.pi * xy[:, 0]) * np.sin(np.pi * xy[:, 1])
    k, ph = rng.integers(1, 4, size=(2, 2)), rng.uniform(0, 2 * np.pi, size=2)
    out = xy.copy()
    for d, h in enumerate((1.0 / nx, 1.0 / ny)):
        out[:, d] += amp * h * bump * np.sin(2 * np.pi * (k[d, 0] * xy[:, 0] + k[d, 1] * xy[:, 1]) + ph[d])
    return np.ascontiguousarray(out)


def element_nodes(xy, nx, ny, g):
    """[ny * nx, g + 1 (dim 0), g + 1 (dim 1), 2]: each element's nodes"""
    grid = xy.reshape(ny * g + 1, nx * g + 1, 2)
    j, i = np.divmod(np.arange(nx * ny), nx)
    a = np.arange(g + 1)
    return grid[(j * g)[:, None, None] + a[None, None, :], (i * g)[:, None, None] + a[None, :, None]]


def mms_state(x, y, m):
    """the manufactured state (conservative variables) with the functions of m (numpy or torch)"""
    t = 2 * math.pi
    rho = 1 + AMP * m.sin(t * x) * m.sin(t * y)
    u = U0 * (1 + AMP * m.cos(t * x) * m.sin(t * y))
    v = V0 * (1 + AMP * m.sin(t * x) * m.cos(t * y))
    pr = PINF * (1 + AMP * m.cos(t * x) * m.cos(t * y))
    return m.stack([rho, rho * u, rho * v, pr / (GAMMA - 1) + 0.5 * rho * (u * u + v * v)], -1)


def grid_problem(c, seed):
    """(node coordinates, initial state [E, nb, neq]) of a Burgers or Navier-Stokes case"""
    rng = np.random.default_rng(seed)
    nx, ny, p, g = c["nx"], c["ny"], c["p"], c["g"]
    xy = smooth_move(lattice(nx, ny, g), nx, ny, 0.05, rng)
    b = lagrange(g, np.linspace(-1.0, 1.0, p + 1))
    pt = np.einsum("ia,jb,eabd->eijd", b, b, element_nodes(xy, nx, ny, g)).reshape(nx * ny, -1, 2)
    if c["pde"] == "ns":
        u = mms_state(pt[..., 0], pt[..., 1], np) * (1.0 + 1e-3 * rng.standard_normal(pt.shape[:2] + (4,)))
    else:
        u = BURGERS_IN + 0.5 * np.sin(2 * np.pi * pt[..., :1]) * np.sin(2 * np.pi * pt[..., 1:])
        u = u + 1e-3 * rng.standard_normal(u.shape)
    return xy, np.ascontiguousarray(u)


def stencil(nx, ny):
    """[5, E]: the element below, left, itself, right and above (-1: none), the ascending columns of a block row"""
    E = np.arange(nx * ny).reshape(ny, nx)
    out = np.full((5, ny, nx), -1)
    out[0, 1:], out[1, :, 1:], out[2], out[3, :, :-1], out[4, :-1] = E[:-1], E[:, :-1], E, E[:, 1:], E[1:]
    return out.reshape(5, -1)


def matrix(c, seed):
    """(blocks [nnz, bs, bs] in BSR order, vector) with the dominance of a DG Jacobian's diagonal blocks"""
    nbr = stencil(c["nx"], c["ny"]).T
    bs = (c["p"] + 1) ** 2 * (4 if c["pde"] == "ns" else 1)
    gen = torch.Generator(device=DEV).manual_seed(seed)
    A = torch.randn(int((nbr >= 0).sum()), bs, bs, dtype=torch.float64, device=DEV, generator=gen).mul_(0.3 / bs ** 0.5)
    A[torch.as_tensor(np.nonzero(nbr >= 0)[1] == 2, device=DEV)] += 2.0 * torch.eye(bs, dtype=torch.float64, device=DEV)
    return A, torch.randn(len(nbr) * bs, dtype=torch.float64, device=DEV, generator=gen)


def mdg_problem(c, seed):
    """(jittered nodes, initial state) of the steady oblique shock of (u^2 / 2)_x + u_y = 0"""
    rng = np.random.default_rng(seed)
    nx, ny, p = c["nx"], c["ny"], c["p"]
    xy = lattice(nx, ny, 1).reshape(ny + 1, nx + 1, 2)
    xy[1:-1, 1:-1] += rng.uniform(-0.2, 0.2, (ny - 1, nx - 1, 2)) / np.array([nx, ny])
    xy = np.ascontiguousarray(xy.reshape(-1, 2))
    b = lagrange(1, np.linspace(-1.0, 1.0, p + 1))
    pt = np.einsum("ia,jb,eabd->eijd", b, b, element_nodes(xy, nx, ny, 1)).reshape(nx * ny, -1, 2)
    u = np.where(pt[..., :1] < 0.4 + 0.2 * pt[..., 1:], 1.0, -0.5) + 1e-2 * rng.standard_normal(pt[..., :1].shape)
    return xy, np.ascontiguousarray(u)


# ----------------------------------------------------------------- prepare
def make_context(c, xy):
    nx, ny = c["nx"], c["ny"]
    ctx = ib.Context(0)
    ctx.mesh_uniform((nx, ny), (0.0, 0.0), (1.0, 1.0), c["g"], (ib.DIRICHLET,) * 4, (0,) * 4)
    ctx.set_coords(xy)
    ctx.fespace(c["p"])
    if c["pde"] == "ns":
        ctx.disc_navier_stokes(GAMMA, PR, MU, ib.FLUX_ROE if c["flux"] == "roe" else ib.FLUX_VANLEER)
        prm = (C.c_double * 7)(GAMMA, PR, MU, PINF, AMP, U0, V0)
        ctx.dirichlet(0, ib.workload_fn("ns_mms_state"), C.cast(prm, C.c_void_p))
        ctx.source(ib.workload_fn("ns_mms_source"), C.cast(prm, C.c_void_p))
    else:
        ctx.disc_burgers(BURGERS_MU, (0.0, 0.0), BURGERS_B)
        prm = (C.c_double * 3)(1.0, BURGERS_IN, BURGERS_SRC)
        ctx.dirichlet(0, ib.workload_fn("constant"), C.cast(prm, C.c_void_p))
        ctx.source(ib.workload_fn("sine_product"), C.c_void_p(C.addressof(prm) + 16))
    ctx.disc_options(c["ip"], 0.0)
    ctx.setup()
    ctx._keep.append(prm)
    return ctx


def newton_options(c):
    o = ib.default_newton_options()
    o.tau_abs, o.kmax, o.gmres_max_it, o.linesearch = 1e-10, 20, 4000, 1
    o.precision, o.ilu_tile, o.matrix_free = c.get("precision", 0), c.get("tile", 0), int(c.get("matrix_free", False))
    o.gmres_cgs_refine = 0
    return o


def pset_specs(c, seed):
    rng = np.random.default_rng(seed)
    # sizes and orders are the case's own; the coefficients and states change with the seed
    shape = np.random.default_rng(c["parts"] * 1000 + c["n_lo"] * 7 + c["n_hi"])
    out = []
    for k in range(c["parts"]):
        out.append(dict(n=int(shape.integers(c["n_lo"], c["n_hi"] + 1)), p=k % 4 + 1,
                        mu=float(10.0 ** rng.uniform(-3.0, -1.0)), theta=float(rng.uniform(0.0, 2 * np.pi)),
                        k=rng.integers(1, 4, 2), ph=rng.uniform(0.0, 2 * np.pi, 2)))
    return out


def prepare(case, seed):
    c = case
    s = {"case": c}
    if c["kind"] == "pset":
        parts, states = [], []
        for sp in pset_specs(c, seed):
            n = sp["n"]
            ctx = ib.Context(0)
            ctx.mesh_uniform((n, n), (0.0, 0.0), (1.0, 1.0), 1, (ib.DIRICHLET,) * 4, (0,) * 4)
            ctx.set_coords(lattice(n, n, 1))
            ctx.fespace(sp["p"])
            ctx.disc_burgers(sp["mu"], (math.cos(sp["theta"]), math.sin(sp["theta"])), (0.0, 0.0))
            ctx.disc_options(False, 0.0)
            step = (C.c_double * 4)(0.5, 0.3, 1.0, 0.0)
            ctx.dirichlet(0, ib.workload_fn("oblique_step"), C.cast(step, C.c_void_p))
            ctx.setup()
            ctx._keep.append(step)
            xy = ctx.basis_node_coords()
            states.append((np.sin(2 * np.pi * sp["k"][0] * xy[..., 0] + sp["ph"][0]) *
                           np.sin(2 * np.pi * sp["k"][1] * xy[..., 1] + sp["ph"][1])).reshape(-1))
            parts.append(ctx)
        s["set"] = ib.ProblemSet(parts)
        s["u0"] = torch.from_numpy(s["set"].gather(states)).to(DEV)
        s["u"] = torch.empty_like(s["u0"])
        s["opt"] = newton_options({})
        return s
    if c["kind"] == "mdg":
        xy, u = mdg_problem(c, seed)
        ctx = ib.Context(0)
        ctx.mesh_uniform((c["nx"], c["ny"]), (0.0, 0.0), (1.0, 1.0), 1,
                         (ib.DIRICHLET, ib.DIRICHLET, ib.DIRICHLET, ib.EXTRAPOLATION), (0,) * 4)
        ctx.set_coords(xy)
        ctx.fespace(c["p"])
        ctx.disc_burgers(0.0, (0.0, 1.0), (1.0, 0.0))
        ctx.disc_options(False, 0.0)
        step = (C.c_double * 4)(0.4, 0.2, 1.0, -0.5)
        ctx.dirichlet(0, ib.workload_fn("oblique_step"), C.cast(step, C.c_void_p))
        ctx.setup()
        ctx._keep.append(step)
        ctx.mdg_select(np.arange(ctx.topology()[2]), True)
        s["x"] = ctx.mdg_get_x()
        nnz = len(ctx.mdg_jacobian_pattern()[3])
        s["ctx"] = ctx
        s["u"] = torch.from_numpy(u.reshape(-1)).to(DEV)
        s["res"] = torch.empty_like(s["u"])
        s["ic"] = torch.empty(ctx.mdg_nsel, dtype=torch.float64, device=DEV)
        s["vals"] = torch.empty(nnz, dtype=torch.float64, device=DEV)
        return s
    xy, u = grid_problem(c, seed)
    ctx = s["ctx"] = make_context(c, xy)
    s["u0"] = torch.from_numpy(u.reshape(-1)).to(DEV)
    if c["kind"] == "residual":
        s["res"] = torch.empty_like(s["u0"])
    elif c["kind"] == "jacobian":
        s["res"] = torch.empty_like(s["u0"])
        nv = ctx.layout.nnz_blocks * ctx.layout.block_size ** 2
        s["vals"] = torch.empty(nv, dtype=torch.float32 if c["f32"] else torch.float64, device=DEV)
    elif c["kind"] in ("spmv", "factor", "apply"):
        s["vals"], s["x"] = matrix(c, seed)
        s["y"] = torch.empty_like(s["x"])
        if c["kind"] != "spmv":
            ctx.ilu_tile = c["tile"]
        if c["kind"] == "apply":
            ctx.pc_factor(s["vals"], 0)
            del s["vals"]
    elif c["kind"] == "newton":
        s["u"] = torch.empty_like(s["u0"])
        s["opt"] = newton_options(c)
    return s


# --------------------------------------------------------------------- run
def run(state):
    s, kind = state, state["case"]["kind"]
    if kind == "residual":
        s["ctx"].form_residual(s["u0"], s["res"])
        return s["res"]
    if kind == "jacobian":
        if s["case"]["f32"]:
            s["ctx"].form_jacobian_fd_f32(s["u0"], s["res"], s["vals"])
        else:
            s["ctx"].form_jacobian_fd(s["u0"], s["res"], s["vals"])
        return {"res": s["res"], "vals": s["vals"]}
    if kind == "spmv":
        s["ctx"].bsr_spmv(s["vals"], s["x"], s["y"])
        return s["y"]
    if kind == "factor":
        s["ctx"].pc_factor(s["vals"], 0)
        s["ctx"].pc_apply(s["x"], s["y"], 0)
        return s["y"]
    if kind == "apply":
        s["ctx"].pc_apply(s["x"], s["y"], 0)
        return s["y"]
    if kind == "newton":
        s["u"].copy_(s["u0"])
        s["ctx"].newton_solve(s["u"], s["opt"])
        return s["u"]
    if kind == "pset":
        s["u"].copy_(s["u0"])
        s["set"].newton_solve(s["u"], s["opt"])
        return s["u"]
    s["ctx"].form_residual_mdg(s["u"], s["x"], s["res"], s["ic"])
    s["ctx"].form_jacobian_mdg_fd(s["u"], s["res"], s["ic"], s["vals"])
    return {"res": s["res"], "ic": s["ic"], "vals": s["vals"]}


# -------------------------------------------------------------------- work
def work(case):
    """each call's inputs read once and its outputs written once; operations of the contractions as a
    tensor-product basis needs them, of the point fluxes, and of the block products"""
    c = case
    if c["kind"] == "pset":
        n = bytes_ = flops = 0
        for sp in pset_specs(c, 0):
            b = (sp["p"] + 1) ** 2
            e = sp["n"] ** 2
            n += e * b
            bytes_ += 8.0 * (2 * e * b + 3 * 5 * e * b * b)  # the state; Jacobian, factors, one product
            flops += e * b * b * (20.0 + 6.0 * b)
        return {"bytes": bytes_, "flops": flops}
    e = c["nx"] * c["ny"]
    if c["kind"] == "mdg":
        b = (c["p"] + 1) ** 2
        nnz = e * b * (5 * b + 8.0) + e * 2 * (9 * 2 + 16 * b)
        return {"bytes": 8.0 * (2 * e * b + 2 * e + nnz), "flops": 60.0 * nnz}
    neq = 4 if c["pde"] == "ns" else 1
    nb, q = (c["p"] + 1) ** 2, c["p"] + c["g"]
    bs = nb * neq
    n, blocks = e * bs, 5 * e - 2 * (c["nx"] + c["ny"])
    n1 = c["p"] + 1
    point = 150.0 if c["pde"] == "ns" else 12.0
    res_flops = e * (neq * (4.0 * n1 * q * (n1 + 1.5 * q) * 2) + point * (q * q + 4.0 * q))
    res_bytes = 8.0 * (2 * n + 2 * e * c["g"] ** 2)
    jac_flops = res_flops + e * (4.0 * q * bs * point + neq * neq * nb * nb * q * (2.0 * q + 6.0)) + blocks * bs * nb * q * 2.0
    if c["kind"] == "residual":
        return {"bytes": res_bytes, "flops": res_flops}
    if c["kind"] == "jacobian":
        return {"bytes": res_bytes + (4.0 if c["f32"] else 8.0) * blocks * bs * bs, "flops": jac_flops}
    if c["kind"] == "spmv":
        return {"bytes": 8.0 * (blocks * bs * bs + 2 * n), "flops": 2.0 * blocks * bs * bs}
    # blocks that the factors keep: those within a tile
    t = c["tile"]
    kept = blocks if not t else blocks - 2 * (((c["nx"] - 1) // t) * c["ny"] + ((c["ny"] - 1) // t) * c["nx"])
    if c["kind"] == "apply":
        return {"bytes": 8.0 * kept * bs * bs + 16.0 * n, "flops": 2.0 * kept * bs * bs}
    factor_flops = 2.0 * bs ** 3 * (e + 1.5 * (kept - e))
    if c["kind"] == "factor":
        return {"bytes": 8.0 * (2 * kept * bs * bs + 2 * n), "flops": factor_flops + 2.0 * kept * bs * bs}
    steps = 3 if c["pde"] == "ns" else 7
    return {"bytes": steps * (res_bytes + 8.0 * (blocks + kept) * bs * bs) + 16.0 * n,
            "flops": steps * (jac_flops + factor_flops)}


# ------------------------------------------------------- exact: plain torch
class Plain:
    """the DG residual of a grid case in plain torch, 64 bits, point by point from the definition"""

    def __init__(self, c, xy, dev):
        self.c, self.nx, self.ny, self.p, self.g = c, c["nx"], c["ny"], c["p"], c["g"]
        self.q = self.p + self.g
        self.dev = dev
        self.neq = 4 if c["pde"] == "ns" else 1
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)  # noqa: E731
        x1, w1 = gauss(self.q)
        self.nodes = t(element_nodes(xy, self.nx, self.ny, self.g))
        self.beta0 = float((self.p + 1) ** 2)
        self.beta1 = 0.0 if c["ip"] else 1.0 / (2 * self.p * (self.p + 1))
        cen = lagrange(self.g, np.zeros(1))[0]
        self.cen = torch.einsum("a,b,eabd->ed", t(cen), t(cen), self.nodes)
        # volume points
        self.vol = self.tables(x1, x1, t)
        X, J, _ = self.geometry(self.vol, slice(None))
        det = J[..., 0, 0] * J[..., 1, 1] - J[..., 0, 1] * J[..., 1, 0]
        self.vJi, self.vx = torch.linalg.inv(J), X
        self.vw = det.clamp(min=0.0) * t(np.outer(w1, w1).reshape(-1))
        self.src = self.source(X)
        # faces by local side: 0 left, 1 bottom, 2 right, 3 top
        self.sides = []
        one = np.ones(1)
        for lf in range(4):
            fixed = -one if lf < 2 else one
            tab = self.tables(fixed, x1, t) if lf % 2 == 0 else self.tables(x1, fixed, t)
            X, J, H = self.geometry(tab, slice(None))
            tang = J[..., :, 1] if lf % 2 == 0 else J[..., :, 0]
            length = tang.norm(dim=-1)
            n = torch.stack([tang[..., 1], -tang[..., 0]], -1) / length[..., None]
            if lf in (0, 3):
                n = -n
            self.sides.append(dict(tab=tab, x=X, Ji=torch.linalg.inv(J), H=H, n=n, w=length * t(w1)))
        E = torch.arange(self.nx * self.ny, device=dev).reshape(self.ny, self.nx)
        self.interior = [(E[:, :-1].reshape(-1), 2, E[:, 1:].reshape(-1), 0),
                         (E[:-1].reshape(-1), 3, E[1:].reshape(-1), 1)]
        self.boundary = [(E[:, 0], 0), (E[0], 1), (E[:, -1], 2), (E[-1], 3)]

    def tables(self, x0, x1, t):
        """values, first and second derivatives of the solution and geometry bases at the points (x0, x1)"""
        out = {}
        for key, order in (("u", self.p), ("g", self.g)):
            b = [[lagrange(order, x, d) for d in range(3)] for x in (x0, x1)]
            f = lambda i, j: t(np.einsum("qi,rj->qrij", b[0][i], b[1][j]).reshape(len(x0) * len(x1), -1))  # noqa: E731
            out[key] = [f(0, 0), f(1, 0), f(0, 1), f(2, 0), f(1, 1), f(0, 2)]
        return out

    def geometry(self, tab, at):
        xn = self.nodes[at].reshape(-1, (self.g + 1) ** 2, 2)
        v = [torch.einsum("qn,end->eqd", m, xn) for m in tab["g"]]
        return v[0], torch.stack([v[1], v[2]], -1), torch.stack([v[3], v[4], v[5]], -1)

    def source(self, X):
        """Navier-Stokes: -div F of the manufactured state, by nested forward derivatives"""
        x, y = X[..., 0].contiguous(), X[..., 1].contiguous()
        if self.c["pde"] != "ns":
            return (BURGERS_SRC * torch.sin(2 * math.pi * x) * torch.sin(2 * math.pi * y))[..., None]
        one, zero = torch.ones_like(x), torch.zeros_like(x)
        jvp = torch.func.jvp
        st = lambda a, b: mms_state(a, b, torch)  # noqa: E731

        def F(a, b):
            u, ux = jvp(st, (a, b), (one, zero))
            _, uy = jvp(st, (a, b), (zero, one))
            return ns_flux(u, torch.stack([ux, uy], -1))

        fx = jvp(F, (x, y), (one, zero))[1][..., 0]
        fy = jvp(F, (x, y), (zero, one))[1][..., 1]
        return -(fx + fy)

    def state(self, u, tab, Ji, H=None):
        """value, physical gradient and Hessian of the coefficients u [e, nb, neq] at the points"""
        n = 6 if H is not None and self.beta1 else 3
        v = [torch.einsum("qi,eik->eqk", m, u) for m in tab["u"][:n]]
        gxi = torch.stack([v[1], v[2]], -1)
        gx = torch.einsum("eqka,eqad->eqkd", gxi, Ji)
        if n == 3:
            return v[0], gx, None
        h = [v[3 + i] - torch.einsum("eqd,eqkd->eqk", H[..., i], gx) for i in range(3)]
        m = torch.stack([torch.stack([h[0], h[1]], -1), torch.stack([h[1], h[2]], -1)], -2)
        return v[0], gx, torch.einsum("eqla,eqklm,eqmb->eqkab", Ji, m, Ji)

    def convective(self, uL, uR, n):
        if self.c["pde"] == "ns":
            return (ns_roe if self.c["flux"] == "roe" else ns_vanleer)(uL, uR, n)
        lam = BURGERS_B[0] * n[..., 0] + BURGERS_B[1] * n[..., 1]
        avg = 0.5 * (uL + uR)[..., 0]
        up = torch.where(0.5 * lam * avg > 0, uL[..., 0], uR[..., 0])
        return (0.5 * lam * up * up)[..., None]

    def viscous(self, u, g, n):
        if self.c["pde"] == "ns":
            return ns_viscous(u, g, n)
        return BURGERS_MU * torch.einsum("eqkd,eqd->eqk", g, n)

    def __call__(self, u):
        """R(u) for u [E, nb, neq]"""
        u = u.reshape(self.nx * self.ny, -1, self.neq)
        v, gx, _ = self.state(u, self.vol, self.vJi)
        if self.c["pde"] == "ns":
            F = ns_flux(v, gx)
        else:
            F = torch.stack([0.5 * BURGERS_B[d] * v * v - BURGERS_MU * gx[..., d] for d in range(2)], -1)
        G = torch.einsum("eqkd,eqad,eq->eqka", F, self.vJi, self.vw)
        r = torch.einsum("qi,eqk->eik", self.vol["u"][1], G[..., 0]) + torch.einsum("qi,eqk->eik", self.vol["u"][2],
                                                                                    G[..., 1])
        r = r - torch.einsum("qi,eqk,eq->eik", self.vol["u"][0], self.src, self.vw)
        for eL, fL, eR, fR in self.interior:
            L, R = self.sides[fL], self.sides[fR]
            n, w = L["n"][eL], L["w"][eL]
            h = torch.einsum("eqd,ed->eq", n, self.cen[eR] - self.cen[eL])
            uL, gL, hL = self.state(u[eL], L["tab"], L["Ji"][eL], L["H"][eL])
            uR, gR, hR = self.state(u[eR], R["tab"], R["Ji"][eR], R["H"][eR])
            gd = self.beta0 * ((uR - uL) / h[..., None])[..., None] * n[:, :, None] + 0.5 * (gL + gR)
            if self.beta1:
                gd = gd + self.beta1 * h[..., None, None] * torch.einsum("eqkab,eqa->eqkb", hR - hL, n)
            f = (self.viscous(0.5 * (uL + uR), gd, n) - self.convective(uL, uR, n)) * w[..., None]
            r.index_add_(0, eL, torch.einsum("qi,eqk->eik", L["tab"]["u"][0], f))
            r.index_add_(0, eR, -torch.einsum("qi,eqk->eik", R["tab"]["u"][0], f))
        for e, lf in self.boundary:
            S = self.sides[lf]
            n, w, X = S["n"][e], S["w"][e], S["x"][e]
            uL, gL, _ = self.state(u[e], S["tab"], S["Ji"][e])
            ud = mms_state(X[..., 0], X[..., 1], torch) if self.c["pde"] == "ns" else torch.full_like(uL, BURGERS_IN)
            h = ((X - self.cen[e][:, None]) * n).abs().sum(-1)
            gd = self.beta0 * ((ud - uL) / h[..., None])[..., None] * n[:, :, None] + gL
            f = (self.viscous(0.5 * (uL + ud), gd, n) - self.convective(uL, ud, n)) * w[..., None]
            r.index_add_(0, e, torch.einsum("qi,eqk->eik", S["tab"]["u"][0], f))
        return r

    def jacobian(self, u):
        """the blocks of dR/du [block][row][column] in BSR order, by central differences over five element
        colours (i + 2 j mod 5: no two elements of a colour share a neighbour)"""
        E, nb, bs = self.nx * self.ny, u.shape[1], u.shape[1] * self.neq
        e = torch.arange(E, device=self.dev)
        colour = ((e % self.nx) + 2 * (e // self.nx)) % 5
        nbr = torch.as_tensor(stencil(self.nx, self.ny), device=self.dev)
        J = torch.zeros(E, 5, bs, bs, dtype=torch.float64, device=self.dev)
        ncol = torch.where(nbr >= 0, colour[nbr.clamp(min=0)], -1)
        for col in range(5):
            own = (colour == col).double()[:, None]
            rows = [torch.nonzero(ncol[k] == col)[:, 0] for k in range(5)]
            for i in range(nb):
                for k in range(self.neq):
                    h = 1e-5 * (1.0 + u[:, i, k].abs().mean()).item()
                    d = torch.zeros_like(u)
                    d[:, i, k] = h * own[:, 0]
                    diff = ((self(u + d) - self(u - d)) / (2 * h)).reshape(E, bs)
                    for b in range(5):
                        J[rows[b], b, :, i * self.neq + k] = diff[rows[b]]
        return J.reshape(E * 5, bs, bs)[(nbr.t().reshape(-1) >= 0)]


def ns_parts(u):
    rho = u[..., 0]
    v = u[..., 1:3] / rho[..., None]
    e = u[..., 3] / rho
    p = (GAMMA - 1) * rho * (e - 0.5 * (v * v).sum(-1))
    return rho, v, e, p, torch.sqrt(GAMMA * p / rho)


def ns_stress(u, g):
    """velocity, gradient of velocity [i, j], of total energy [j], and stress"""
    rho, v, e, p, _ = ns_parts(u)
    gv = (g[..., 1:3, :] - v[..., :, None] * g[..., None, 0, :]) / rho[..., None, None]
    ge = (g[..., 3, :] - e[..., None] * g[..., 0, :]) / rho[..., None]
    div = gv[..., 0, 0] + gv[..., 1, 1]
    eye = torch.eye(2, dtype=u.dtype, device=u.device)
    tau = MU * (gv + gv.transpose(-1, -2)) - (2.0 / 3.0) * MU * div[..., None, None] * eye
    return v, gv, ge, tau, p


def ns_flux(u, g):
    """the physical flux [..., eq, d]"""
    v, gv, ge, tau, p = ns_stress(u, g)
    mom = u[..., 1:3]
    eye = torch.eye(2, dtype=u.dtype, device=u.device)
    fm = mom[..., :, None] * v[..., None, :] + p[..., None, None] * eye - tau
    heat = MU * GAMMA / PR * (ge - (v[..., :, None] * gv).sum(-2))
    fe = v * (u[..., 3] + p)[..., None] - heat - (v[..., :, None] * tau).sum(-2)
    return torch.cat([mom[..., None, :], fm, fe[..., None, :]], -2)


def ns_viscous(u, g, n):
    """the normal viscous flux; its energy row takes the gradient of the total energy"""
    v, _, ge, tau, _ = ns_stress(u, g)
    tn = (tau * n[..., None, :]).sum(-1)
    fe = MU * GAMMA / PR * (ge * n).sum(-1) + (v * tn).sum(-1)
    return torch.cat([torch.zeros_like(fe)[..., None], tn, fe[..., None]], -1)


def ns_normal(u, n):
    rho, v, e, p, c = ns_parts(u)
    vn = (v * n).sum(-1)
    f = torch.cat([(rho * vn)[..., None], u[..., 1:3] * vn[..., None] + p[..., None] * n,
                   (vn * (u[..., 3] + p))[..., None]], -1)
    return f, rho, v, e, p, c, vn


def ns_vanleer(uL, uR, n):
    out = 0.0
    for u, sg in ((uL, 1.0), (uR, -1.0)):
        f, rho, v, e, p, c, vn = ns_normal(u, n)
        m = vn / c
        fm = sg * rho * c * (m + sg) ** 2 / 4
        t = (GAMMA - 1) * vn + sg * 2 * c
        sub = torch.cat([fm[..., None], fm[..., None] * (v + n * ((-vn + sg * 2 * c) / GAMMA)[..., None]),
                         (fm * (((v * v).sum(-1) - vn * vn) / 2 + t * t / (2 * (GAMMA * GAMMA - 1))))[..., None]], -1)
        sm = (sg * m)[..., None]
        out = out + torch.where(sm > 1, f, torch.where(sm < -1, torch.zeros_like(f), sub))
    return out


def ns_roe(uL, uR, n):
    fL, rL, vL, eL, pL, _, vnL = ns_normal(uL, n)
    fR, rR, vR, eR, pR, _, vnR = ns_normal(uR, n)
    sL, sR = torch.sqrt(rL), torch.sqrt(rR)
    mean = lambda a, b: (sL * a + sR * b) / (sL + sR)  # noqa: E731
    ut = torch.stack([mean(vL[..., d], vR[..., d]) for d in range(2)], -1)
    Ht, rt = mean(eL + pL / rL, eR + pR / rR), sL * sR
    qq = (ut * ut).sum(-1)
    c2 = (GAMMA - 1) * (Ht - 0.5 * qq)
    c = torch.sqrt(c2)
    un = (ut * n).sum(-1)
    dun, dp = vnR - vnL, pR - pL
    fix = lambda l: torch.where(l < 0.1 * c, (l * l + 0.01 * c2) / (0.2 * c), l)  # noqa: E731
    s1 = fix((un - c).abs()) * (dp - rt * c * dun) / (2 * c2)
    s2 = un.abs() * (rR - rL - dp / c2)
    s4 = fix((un + c).abs()) * (dp + rt * c * dun) / (2 * c2)
    ss, st = un.abs() * rt, vR - vL - dun[..., None] * n
    k = lambda a: a[..., None]  # noqa: E731
    d = torch.cat([k(s1 + s2 + s4),
                   k(s1) * (ut - k(c) * n) + k(s2) * ut + k(s4) * (ut + k(c) * n) + k(ss) * st,
                   k(s1 * (Ht - c * un) + 0.5 * s2 * qq + s4 * (Ht + c * un) + ss * (ut * st).sum(-1))], -1)
    return 0.5 * (fL + fR) - 0.5 * d


def ilu_solve(A, x, nx, ny, tile):
    """(L U)^-1 x of the block-ILU(0) of A in natural order, blocks across tiles dropped, one anti-diagonal at a time"""
    nbr = torch.as_tensor(stencil(nx, ny), device=A.device)
    E, bs = nx * ny, A.shape[1]
    has = nbr >= 0
    pos = torch.cumsum(has.t().reshape(-1).long(), 0).reshape(E, 5).t() - 1
    e = torch.arange(E, device=A.device)
    i, j = e % nx, e // nx
    t = tile if tile else max(nx, ny)
    x = x.reshape(E, bs)
    for k in range(5):
        o = nbr[k].clamp(min=0)
        nbr[k] = torch.where(has[k] & (i // t == o % nx // t) & (j // t == o // nx // t), nbr[k], -1)
    level = i % t + j % t
    last = int(level.max())
    inv, f, y = torch.empty(E, bs, bs, dtype=A.dtype, device=A.device), x.clone(), torch.empty_like(x)
    for lv in range(last + 1):
        at = torch.nonzero(level == lv)[:, 0]
        D, fa = A[pos[2][at]], x[at].clone()
        for k in (0, 1):  # the lower neighbours: L = A inv(U), and the diagonal's update through the opposite block
            m = torch.nonzero(nbr[k][at] >= 0)[:, 0]
            o = nbr[k][at[m]]
            L = A[pos[k][at[m]]] @ inv[o]
            D[m] -= L @ A[pos[4 - k][o]]
            fa[m] -= (L @ f[o][..., None])[..., 0]
        f[at], inv[at] = fa, torch.linalg.inv(D)
    for lv in range(last, -1, -1):
        at = torch.nonzero(level == lv)[:, 0]
        fa = f[at].clone()
        for k in (3, 4):
            m = torch.nonzero(nbr[k][at] >= 0)[:, 0]
            fa[m] -= (A[pos[k][at[m]]] @ y[nbr[k][at[m]]][..., None])[..., 0]
        y[at] = (inv[at] @ fa[..., None])[..., 0]
    return y.reshape(-1)


def exact(case, seed):
    c = case
    if c["kind"] in ("pset", "mdg"):
        return None  # a set of sparse solves, and differences over the geometry: too much for plain torch
    if c["kind"] in ("spmv", "factor", "apply"):
        A, x = matrix(c, seed)
        if c["kind"] != "spmv":
            return ilu_solve(A, x, c["nx"], c["ny"], c["tile"])
        nbr = torch.as_tensor(stencil(c["nx"], c["ny"]), device=A.device).t()
        rows, ks = torch.nonzero(nbr >= 0, as_tuple=True)
        X = x.reshape(len(nbr), -1)
        y = torch.zeros_like(X)
        for k in range(5):
            y[rows[ks == k]] += torch.einsum("bij,bj->bi", A[ks == k], X[nbr[:, k][nbr[:, k] >= 0]])
        return y.reshape(-1)
    xy, u = grid_problem(c, seed)
    R = Plain(c, xy, DEV)
    u = torch.as_tensor(u, device=DEV)
    if c["kind"] == "residual":
        return R(u).reshape(-1)
    if c["kind"] == "jacobian":
        return {"res": R(u).reshape(-1), "vals": R.jacobian(u).reshape(-1)}
    if c["pde"] == "ns" or u.numel() > 12000:
        return None  # the dense linearisation of exact_newton() would not fit
    return exact_newton(R, u)


def exact_newton(R, u):
    """the root of R by Newton steps on the dense Jacobian"""
    E, n = u.shape[0], u.numel()
    bs = n // E
    nbr = torch.as_tensor(stencil(R.nx, R.ny), device=u.device)
    r = R(u)
    for _ in range(20):
        J = R.jacobian(u)
        dense = torch.zeros(n, n, dtype=torch.float64, device=u.device)
        view = dense.reshape(E, bs, E, bs)
        rows, ks = torch.nonzero(nbr.t() >= 0, as_tuple=True)
        view[rows, :, nbr[ks, rows], :] = J
        du = torch.linalg.solve(dense, r.reshape(-1)).reshape(u.shape)
        alpha = 1.0
        while R(u - alpha * du).norm() > r.norm() and alpha > 1e-3 and r.norm() > 1e-9:
            alpha *= 0.5
        u = u - alpha * du
        r = R(u)
        if r.norm() < 1e-13 or du.norm() < 1e-14 * u.norm():
            break
    return u.reshape(-1)
