"""What is timed: the work that programs have this framework do, through its public entry points.

    solve      one pressure solve from a zero guess (FP32, FP64, or FP32 cycles in FP64 refinement)
    project    one projection of a MAC velocity (divergence, pressure solve, gradient)
    flow       one Boussinesq time step: stable step size, advection, diffusion, projection
    stencils   one evaluation of the explicit terms: self-advection, scalar advection, diffusion
    ensemble   many independent pressure solves of uneven sizes in one persistent launch
    chain      the differentiable advection + projection chain, forward and gradients

`listed` holds the sizes of the repository's own benchmark and tests; `draw` gives others of the
same kinds, up to 256 cells along an axis, odd multiples of powers of two among them, with every
boundary type and both precisions.  `exact` restates each path in plain 64-bit torch.
"""
import math

import torch

import opencurrent_b200 as ocu
from opencurrent_b200.autograd import AdvectProject, AdvectProjectChain

_DTYPE = {"f32": ocu.F32, "f64": ocu.F64, "mixed": ocu.F64}
_TORCH = {ocu.F32: torch.float32, ocu.F64: torch.float64}


def listed():
    return [
        # a small box solved inside some other program's loop: launches and latency only
        dict(name="solve_f32_32", kind="solve", type="f32", nx=32, ny=32, nz=32, bc="closed", rhs="noise", tol=1e-6),
        # the benchmark's plain FP32 solve
        dict(name="solve_f32_64", kind="solve", type="f32", nx=64, ny=64, nz=64, bc="closed", rhs="noise", tol=1e-6),
        # FP64 on an uneven grid open at top and bottom, to near the precision of the type
        dict(name="solve_f64_96x80x112", kind="solve", type="f64", nx=96, ny=80, nz=112, bc="open", rhs="noise",
             tol=1e-10),
        # refinement on an uneven grid, one periodic axis
        dict(name="solve_mixed_192x160x144", kind="solve", type="mixed", nx=192, ny=160, nz=144, bc="duct",
             rhs="noise", tol=1e-10),
        # the benchmark's headline pair: the same 256^3 problem by refinement and in plain FP64
        dict(name="solve_mixed_256", kind="solve", type="mixed", nx=256, ny=256, nz=256, bc="closed", rhs="modes",
             tol=1e-10),
        dict(name="solve_f64_256", kind="solve", type="f64", nx=256, ny=256, nz=256, bc="closed", rhs="modes",
             tol=1e-10),
        # a velocity field made divergence-free in a closed box, as an application's own step does
        dict(name="project_f32_128x96x64", kind="project", type="f32", nx=128, ny=96, nz=64, bc="closed", tol=2e-5),
        # the benchmark's Rayleigh-Benard flow, pressure by refinement (every step converges) ...
        dict(name="flow_f32_128x128x64", kind="flow", type="f32", nx=128, ny=128, nz=64, refined=True, ab2=False),
        # ... and by the plain FP32 solver, which runs to its cycle limit; Adams-Bashforth
        dict(name="flow_f32_plain_128x128x64", kind="flow", type="f32", nx=128, ny=128, nz=64, refined=False, ab2=True),
        # the explicit terms alone on a grid larger than the L2 cache
        dict(name="stencils_f32_256x256x128", kind="stencils", type="f32", nx=256, ny=256, nz=128, centred=False),
        # the benchmark's ensemble: 512 members drawn from 32^3, 48^3, 64^3, 96^3
        dict(name="ensemble_512", kind="ensemble", members=512, tol=1e-6, sizes=1),
        # the benchmark's differentiable flow: 32 steps, checkpoints every 8
        dict(name="chain_f32_96", kind="chain", type="f32", nx=96, ny=96, nz=96, steps=32, tol=3e-5),
    ]


def _box(rng, top, coarse):
    """Axes m 2^p with one p, m in 3..9 without 8: the longest near a length spread over the
    logarithm of [16, top], at most `coarse` cells where halving stops."""
    want = math.exp(rng.uniform(math.log(16), math.log(top)))
    while True:
        p = rng.randint(2, 6)
        m = [rng.choice((3, 4, 5, 6, 7, 9)) for _ in range(3)]
        n = max(m) << p
        if math.prod(m) <= coarse and 0.75 * want < n < 1.33 * want and 16 <= n <= top:
            return [q << p for q in m]


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "project", "flow", "stencils", "ensemble", "chain"])
    if kind == "solve":
        t = rng.choice(["f32", "f64", "mixed"])
        n = _box(rng, 256, 256)
        return dict(kind=kind, type=t, nx=n[0], ny=n[1], nz=n[2], bc=rng.choice(["closed", "open", "duct"]),
                    rhs=rng.choice(["noise", "modes"]), tol=rng.choice([1e-4, 1e-5] if t == "f32" else [1e-6, 1e-8, 1e-10]))
    if kind == "project":
        t = rng.choice(["f32", "f64"])
        n = _box(rng, 192, 150)
        return dict(kind=kind, type=t, nx=n[0], ny=n[1], nz=n[2], bc=rng.choice(["closed", "channel", "periodic"]),
                    tol=rng.choice([1e-4, 2e-5] if t == "f32" else [1e-6, 1e-9]))
    if kind == "flow":
        n = _box(rng, 160, 80)
        return dict(kind=kind, type="f32", nx=n[0], ny=n[1], nz=n[2], refined=rng.random() < 0.7, ab2=rng.random() < 0.5)
    if kind == "stencils":  # any size: nothing is coarsened
        n = [int(math.exp(rng.uniform(math.log(16), math.log(257)))) for _ in range(3)]
        return dict(kind=kind, type=rng.choice(["f32", "f64"]), nx=n[0], ny=n[1], nz=n[2], centred=rng.random() < 0.3)
    if kind == "ensemble":
        return dict(kind=kind, members=int(math.exp(rng.uniform(math.log(8), math.log(512)))), tol=rng.choice([1e-6, 1e-8]),
                    sizes=rng.randrange(2, 1000))
    n = _box(rng, 96, 80)
    return dict(kind=kind, type="f32", nx=n[0], ny=n[1], nz=n[2], steps=rng.randint(4, 16), tol=3e-5)


# ---- inputs ---------------------------------------------------------------------------------


class _Memory:
    def __init__(self, grid):
        self.grid = grid  # tensors made of this keep the grid, and the solver that lends it
        L = grid.layout
        self.__cuda_array_interface__ = dict(shape=(int(L.allocated),), typestr="<f8" if grid.dtype == ocu.F64 else "<f4",
                                             data=(grid.device_ptr, False), version=3)


def _flat(grid):
    """The grid's whole padded buffer as a CUDA tensor (no copy; the grid owns the memory)."""
    return torch.as_tensor(_Memory(grid), device="cuda")


def _cells(grid, lo=0, n=None):
    """The cells lo .. lo + n - 1 along each axis (default: the interior) as a strided view."""
    L = grid.layout
    n = n or (L.nx, L.ny, L.nz)
    return _flat(grid).as_strided(n, (L.xstride, L.ystride, 1), int(L.shift) + lo * (L.xstride + L.ystride + 1))


def _grid(dtype, shape, pad=(0, 0, 0)):
    g = ocu.Grid3DDevice(dtype)
    g.init(*shape, 1, 1, 1, *pad)
    return g


def _mac(dtype, n):
    """u, v, w and a cell grid of one padded layout."""
    x, y, z = n
    return (_grid(dtype, (x + 1, y, z), (0, 1, 1)), _grid(dtype, (x, y + 1, z), (1, 0, 1)),
            _grid(dtype, (x, y, z + 1), (1, 1, 0)), _grid(dtype, n, (1, 1, 1)))


def _rng(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _noise(g, shape):
    return torch.rand(shape, generator=g, device="cuda", dtype=torch.float64) * 2 - 1


def _modes(g, shape, count=16, top=16, phase=False):
    """A sum of `count` cosine modes, wavenumbers 1..top (below the grid's), amplitudes N(0, 1)."""
    out = torch.zeros(shape, device="cuda", dtype=torch.float64)
    k = [torch.randint(1, min(top, n // 2) + 1, (count,), generator=g, device="cuda") for n in shape]
    a = torch.randn(count, generator=g, device="cuda", dtype=torch.float64)
    s = torch.rand((3, count), generator=g, device="cuda", dtype=torch.float64) * (2 * math.pi if phase else 0)
    for m in range(count):
        x, y, z = (torch.cos(k[d][m] * math.pi * (torch.arange(n, device="cuda", dtype=torch.float64) + 0.5) / n + s[d, m])
                   for d, n in enumerate(shape))
        out += a[m] * x[:, None, None] * y[None, :, None] * z[None, None, :]
    return out


def _bcs(name):
    neu, dirich, per = (ocu.BoundaryCondition(t) for t in (ocu.BC_NEUMANN, ocu.BC_DIRICHELET, ocu.BC_PERIODIC))
    return {"closed": ocu.BoundaryConditionSet(neu),                                 # Neumann all round
            "open": ocu.BoundaryConditionSet(neu, zpos=dirich, zneg=dirich),         # fixed pressure at both ends of z
            "duct": ocu.BoundaryConditionSet(neu, xpos=per, xneg=per, zpos=dirich)}[name]


def _flow_bcs(name):
    wall = ocu.BoundaryCondition(ocu.BC_FORCED_INFLOW_VARIABLE_SLIP, 0.0, 1.0)
    per = ocu.BoundaryCondition(ocu.BC_PERIODIC)
    return {"closed": ocu.BoundaryConditionSet(wall), "periodic": ocu.BoundaryConditionSet(per),
            "channel": ocu.BoundaryConditionSet(per, zpos=wall, zneg=wall)}[name]


_AXES = {"closed": ("neumann",) * 3, "open": ("neumann", "neumann", "dirichlet"), "duct": ("periodic", "neumann", "outlet"),
         "periodic": ("periodic",) * 3, "channel": ("periodic", "periodic", "neumann")}


def _size(case):
    return case["nx"], case["ny"], case["nz"]


def _spacing(case):
    return 1.0 / max(_size(case))  # cubic cells, the longest side of length 1


def _rhs(case, seed):
    g = _rng(seed)
    b = _noise(g, _size(case)) if case["rhs"] == "noise" else _modes(g, _size(case))
    if case["bc"] == "closed":
        b -= b.mean()
    return b.to(_TORCH[_DTYPE[case["type"]]])


def _velocity(case, seed):
    """A velocity to project: smooth motion with a rough part, at the faces."""
    g, (x, y, z) = _rng(seed), _size(case)
    return [(_modes(g, s, 6, 4, True) * 0.4 + 0.2 * _noise(g, s)).to(_TORCH[_DTYPE[case["type"]]])
            for s in ((x + 1, y, z), (x, y + 1, z), (x, y, z + 1))]


def _flow_start(case, seed):
    """Conduction profile with a finite perturbation, and a matching slow motion."""
    g, (x, y, z) = _rng(seed), _size(case)
    zc = (torch.arange(z, device="cuda", dtype=torch.float64) + 0.5) / z
    t = (1 - zc) + 0.05 * torch.sin(math.pi * zc) * _modes(g, (x, y, z), 6, 6, True)
    u, v, w = (5.0 * _modes(g, s, 6, 4, True) for s in ((x + 1, y, z), (x, y + 1, z), (x, y, z + 1)))
    return [f.to(_TORCH[_DTYPE[case["type"]]]) for f in (u, v, w, t)]


def _chain_start(case, seed):
    """Velocity = discrete curl of a smooth periodic potential, max 1; a scalar blob; a target."""
    g, n = _rng(seed), _size(case)
    at = [torch.arange(m, device="cuda", dtype=torch.float64) * (2 * math.pi / m) for m in n]

    def potential():
        f = torch.zeros(n, device="cuda", dtype=torch.float64)
        for _ in range(12):
            k = torch.randint(0, 6, (3,), generator=g, device="cuda")
            s = torch.rand(3, generator=g, device="cuda", dtype=torch.float64) * 2 * math.pi
            a = torch.randn(1, generator=g, device="cuda", dtype=torch.float64)
            f += a * (torch.cos(k[0] * at[0] + s[0])[:, None, None] * torch.cos(k[1] * at[1] + s[1])[None, :, None]
                      * torch.cos(k[2] * at[2] + s[2])[None, None, :])
        return f

    def d(f, axis):
        return torch.roll(f, -1, axis) - f

    a, b, c = potential(), potential(), potential()
    vel = [d(c, 1) - d(b, 2), d(a, 2) - d(c, 0), d(b, 0) - d(a, 1)]
    top = max(float(f.abs().max()) for f in vel)

    def blob():
        e = 0
        for axis, m in enumerate(n):
            x = (torch.arange(m, device="cuda", dtype=torch.float64) + 0.5) / m
            r = (x - (0.3 + 0.4 * torch.rand(1, generator=g, device="cuda", dtype=torch.float64))).abs()
            r = torch.minimum(r, 1 - r)
            e = e + (r * r).reshape([-1 if q == axis else 1 for q in range(3)])
        return torch.exp(-e / (2 * 0.1 ** 2))

    return [(f / top).float() for f in vel] + [blob().float(), blob().float()]


def _chain_dt(case):
    return 0.5 * _spacing(case)  # CFL 0.5 at velocity 1


def _member_sizes(case):
    g = torch.Generator().manual_seed(case["sizes"])
    return [(32, 48, 64, 96)[i] for i in torch.randint(0, 4, (case["members"],), generator=g).tolist()]


def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed)


def run(state):
    return state["run"](state)


def _prepare_solve(case, seed):
    n, h, dt = _size(case), _spacing(case), _DTYPE[case["type"]]
    rhs = _grid(dt, n)
    b = _rhs(case, seed)
    _cells(rhs).copy_(b)
    s = ocu.Sol_MultigridPressureMixed3DDeviceD() if case["type"] == "mixed" else ocu.Sol_MultigridPressure3DDevice(dt)
    s.bc = _bcs(case["bc"])
    s.initialize_storage(*n, h, h, h, rhs)
    p = s.pressure()
    return dict(run=_run_solve, solver=s, p=p, view=_cells(p), tol=case["tol"] * float(b.double().square().mean().sqrt()))


def _run_solve(st):
    st["p"].clear_zero()
    ok, _ = st["solver"].solve(st["tol"], 20)
    return {"converged": ok, "p": st["view"]}


def _prepare_project(case, seed):
    n, h, dt = _size(case), _spacing(case), _DTYPE[case["type"]]
    given, work = _mac(dt, n)[:3], _mac(dt, n)[:3]
    for g, f in zip(given, _velocity(case, seed)):
        _cells(g).copy_(f)
    s = ocu.Sol_ProjectDivergence3DDevice(dt)
    s.bc = _flow_bcs(case["bc"])
    s.initialize_storage(*n, h, h, h, *work)
    return dict(run=_run_project, solver=s, p=s.pressure_solver.pressure(), given=given, work=work,
                views=[_cells(g) for g in work], tol=case["tol"] / h)


def _run_project(st):
    for g, f in zip(st["work"], st["given"]):  # the step's provisional velocity
        g.copy_all_data(f)
    st["p"].clear_zero()
    ok = st["solver"].solve(st["tol"])
    return {"converged": ok, "uvw": st["views"]}


def _prepare_flow(case, seed):
    n, dt = _size(case), _DTYPE[case["type"]]
    p = ocu.Eqn_IncompressibleNS3DParams(dt)
    p.init_grids(*n)
    p.hx = p.hy = p.hz = 1.0 / n[2]
    p.max_divergence = 1e-5
    p.flow_bc = _flow_bcs("channel")
    per = ocu.BoundaryCondition(ocu.BC_PERIODIC)
    p.temp_bc = ocu.BoundaryConditionSet(per, zpos=ocu.BoundaryCondition(ocu.BC_DIRICHELET, 0.0),
                                         zneg=ocu.BoundaryCondition(ocu.BC_DIRICHELET, 1.0))
    p.vertical_direction = ocu.DIR_ZPOS
    p.gravity, p.bouyancy, p.thermal_diffusion, p.viscosity = -1.0, _RA * _PR, 1.0, _PR
    p.advection_scheme = ocu.IT_FIRST_ORDER_UPWIND
    p.time_step = ocu.TS_ADAMS_BASHFORD2 if case["ab2"] else ocu.TS_FORWARD_EULER
    p.cfl_factor = _CFL
    p.mixed_pressure = case["refined"]
    for c, buf, f in zip("uvwt", (p.init_u, p.init_v, p.init_w, p.init_temp), _flow_start(case, seed)):
        L = p.layouts[c]
        torch.from_numpy(buf).as_strided(f.shape, (L.xstride, L.ystride, 1), int(L.shift)).copy_(f)
    e = ocu.Eqn_IncompressibleNS3D(dt)
    e.set_parameters(p)
    return dict(run=_run_flow, eqn=e)


def _run_flow(st):
    e = st["eqn"]
    dt = e.get_max_stable_timestep()
    e.advance_one_step(dt)
    return {"dt": dt, "uvwt": [_cells(g) for g in (e.get_u(), e.get_v(), e.get_w(), e.get_temperature())]}


def _stencil_fields(case, seed):
    """u, v, w and the scalar with one layer of ghosts all round."""
    g, (x, y, z) = _rng(seed), _size(case)
    return [(_modes(g, s, 6, 6, True) + 0.1 * _noise(g, s)).to(_TORCH[_DTYPE[case["type"]]])
            for s in ((x + 3, y + 2, z + 2), (x + 2, y + 3, z + 2), (x + 2, y + 2, z + 3), (x + 2, y + 2, z + 2))]


def _prepare_stencils(case, seed):
    n, h, dt = _size(case), _spacing(case), _DTYPE[case["type"]]
    ins, outs = _mac(dt, n), _mac(dt, n)
    for g, f in zip(ins, _stencil_fields(case, seed)):
        _cells(g, -1, f.shape).copy_(f)
    sch = ocu.IT_SECOND_ORDER_CENTERED if case["centred"] else ocu.IT_FIRST_ORDER_UPWIND
    own, scalar, lap = ocu.Sol_SelfAdvection3DDevice(), ocu.Sol_PassiveAdvection3DDevice(), ocu.Sol_LaplacianCentered3DDevice()
    own.interp_type = scalar.interp_type = sch
    lap.coefficient = _KAPPA * h
    own.initialize_storage(*n, h, h, h, *ins[:3], *outs[:3])
    scalar.initialize_storage(*n, h, h, h, *ins[:3], ins[3], outs[3])
    lap.initialize_storage(*n, h, h, h, ins[3], outs[3])
    return dict(run=_run_stencils, parts=(own, scalar, lap), views=[_cells(g, 0, n) for g in outs])


def _run_stencils(st):
    for s in st["parts"]:
        s.solve()
    return st["views"]


def _prepare_ensemble(case, seed):
    sizes = _member_sizes(case)
    # the launch shape and schedule that PersistentEnsemble.autotune picks for these sizes
    e = ocu.PersistentEnsemble([(n,) * 3 for n in sizes], [(1.0 / n,) * 3 for n in sizes], threads=1024, cycles=3, nu1=2,
                               nu2=1)
    g, tol = _rng(seed), []
    for m, n in enumerate(sizes):
        b = _noise(g, (n,) * 3)
        b -= b.mean()
        _cells(e.rhs(m)).copy_(b)
        tol.append(b.square().mean().sqrt())
    tol = (torch.stack(tol) * case["tol"]).tolist()
    p = [e.pressure(m) for m in range(len(sizes))]
    groups = [[_cells(p[m]) for m, s in enumerate(sizes) if s == n] for n in sorted(set(sizes))]
    return dict(run=_run_ensemble, ens=e, tol=tol, p=p, flats=[_flat(q) for q in p], groups=groups)


def _run_ensemble(st):
    torch._foreach_zero_(st["flats"])
    conv = st["ens"].solve(st["tol"])
    return {"converged": conv, "p": [torch.stack(q) for q in st["groups"]]}


def _prepare_chain(case, seed):
    h = _spacing(case)
    ch = AdvectProjectChain(_size(case), (h, h, h), case["steps"], _chain_dt(case), checkpoint_every=8, dtype=ocu.F32,
                            proj_tol=case["tol"])
    *start, target = _chain_start(case, seed)
    ins = []
    for which, f in zip("uvwt", start):
        t = ch.empty(which)
        ch.interior(t, which).copy_(f)
        ins.append(t.requires_grad_(True))
    return dict(run=_run_chain, chain=ch, ins=ins, target=target)


def _run_chain(st):
    ch = st["chain"]
    out = AdvectProject.apply(*st["ins"], ch)
    phi = ch.interior(out, "t")
    loss = 0.5 * (phi - st["target"]).square().sum()
    grads = torch.autograd.grad(loss, st["ins"])
    return {"phi": phi.detach(), "grads": [ch.interior(g, w) for g, w in zip(grads, "uvwt")]}


_RA, _PR, _CFL, _KAPPA = 1e6, 0.71, 0.5, 0.1


# ---- what a pass cannot do without ----------------------------------------------------------


def work(case):
    """Each input read once and each output written once; a multigrid solve's arithmetic as ten
    V-cycles of 60 operations a cell."""
    kind = case["kind"]
    if kind == "ensemble":
        cells = sum(n ** 3 for n in _member_sizes(case))
        return {"bytes": 16 * cells, "flops": 600 * cells}
    cells = case["nx"] * case["ny"] * case["nz"]
    b = 4 if case["type"] == "f32" else 8
    words, ops = {"solve": (2, 600), "project": (6, 620), "flow": (8, 800), "stencils": (8, 130), "chain": (9, 0)}[kind]
    if kind == "chain":
        ops = 2 * 900 * case["steps"]
    return {"bytes": words * b * cells, "flops": ops * cells}


def tolerance(case):
    """About four times what two correct ways of computing the same differed by."""
    kind, f32 = case["kind"], case.get("type") == "f32"
    if kind == "ensemble" or kind == "solve" and case["bc"] == "closed":
        # the constant that a closed box leaves free: 2.7e-5 between the refinement's two inner
        # solvers and 3.0e-5 between refinement and plain FP64 at 256^3 (5e-15 without the mean)
        return {"rel": max(1e-4, (40 if f32 else 1600) * case["tol"])} if kind == "solve" else {"rel": 1e-4}
    if kind == "solve":  # the error that the residual tolerance leaves: 130 to 390 times it in FP64
        return {"rel": (40 if f32 else 1600) * case["tol"]}
    if kind == "project":
        return {"rel": (4 if f32 else 40) * case["tol"]}
    if kind == "flow":  # the plain FP32 solver stops at its cycle limit, 1.4e-5 from the 64-bit step
        return {"rel": 1e-5 if case["refined"] else 1e-4}
    if kind == "stencils":
        return {"rel": 2e-6 if f32 else 4e-15}
    return {"rel": 2e-5}  # chain


# ---- the same in plain 64-bit torch ---------------------------------------------------------


def exact(case, seed):
    return globals()["_exact_" + case["kind"]](case, seed)


def _poisson(b, h, axes):
    """Solution of the 7-point Laplace equation lap p = b with homogeneous boundary values, by
    diagonalising each axis; the null space's part is zero."""
    vs, ls = [], []
    for n, t in zip(b.shape, axes):
        a = torch.diag(torch.full((n,), -2.0, dtype=torch.float64))
        a += torch.diag(torch.ones(n - 1, dtype=torch.float64), 1) + torch.diag(torch.ones(n - 1, dtype=torch.float64), -1)
        if t == "periodic":
            a[0, -1] += 1
            a[-1, 0] += 1
        else:
            a[0, 0] += -1 if t == "dirichlet" else 1
            a[-1, -1] += -1 if t in ("dirichlet", "outlet") else 1
        val, vec = torch.linalg.eigh(a.cuda() / (h * h))
        ls.append(val)
        vs.append(vec)
    f = torch.einsum("ijk,ia,jb,kc->abc", b.double(), *vs)
    d = ls[0][:, None, None] + ls[1][None, :, None] + ls[2][None, None, :]
    f = torch.where(d.abs() > 1e-9 * d.abs().max(), f / d, torch.zeros_like(f))
    return torch.einsum("abc,ia,jb,kc->ijk", f, *vs)


def _exact_solve(case, seed):
    if case["bc"] == "closed":  # fixed up to a constant, which the iteration is free to choose
        return None
    return {"converged": None, "p": _poisson(_rhs(case, seed), _spacing(case), _AXES[case["bc"]])}


def _close(f, axis, kind):
    """Normal velocities: zero on walls, the two ends equal where periodic."""
    n = f.shape[axis] - 1
    a, b = f.select(axis, 0), f.select(axis, n)
    if kind == "periodic":
        b.copy_(a)
    else:
        a.zero_()
        b.zero_()


def _project(vel, h, axes):
    vel = [f.clone() for f in vel]
    for a, f in enumerate(vel):
        _close(f, a, axes[a])
    p = _poisson(sum(torch.diff(f, dim=a) for a, f in enumerate(vel)) / h, h, axes)
    for a, f in enumerate(vel):
        n = p.shape[a]
        f.narrow(a, 1, n - 1).sub_(torch.diff(p, dim=a) / h)
        if axes[a] == "periodic":
            f.select(a, 0).sub_((p.select(a, 0) - p.select(a, n - 1)) / h)
        _close(f, a, axes[a])
    return vel


def _exact_project(case, seed):
    return {"converged": None,
            "uvw": _project([f.double() for f in _velocity(case, seed)], _spacing(case), _AXES[case["bc"]])}


def _up(c, x0, x1, centred):
    return 0.5 * (x0 + x1) if centred else torch.where(c < 0, x1, x0)


def _flux_terms(at, h, centred):
    """Time derivatives of u, v, w and of a scalar from their advection; at(f, di, dj, dk) is
    field f (0, 1, 2 the velocity, 3 the scalar) at a cell's neighbour."""
    e = ((1, 0, 0), (0, 1, 0), (0, 0, 1))

    def nb(f, *steps):
        o = [0, 0, 0]
        for axis, s in steps:
            o[axis] += s
        return at(f, *o)

    out = []
    for c in range(3):
        q, total = nb(c), 0
        for a in range(3):
            hi = 0.5 * (nb(a, (a, 1)) + nb(a, (a, 1), (c, -1))) if a != c else 0.5 * (q + nb(c, (c, 1)))
            lo = 0.5 * (nb(a) + nb(a, (c, -1)))
            total = total + hi * _up(hi, q, nb(c, (a, 1)), centred) - lo * _up(lo, nb(c, (a, -1)), q, centred)
        out.append(-total / h)
    q, total = nb(3), 0
    for a in range(3):
        hi, lo = nb(a, (a, 1)), nb(a)
        total = total + hi * _up(hi, q, nb(3, (a, 1)), centred) - lo * _up(lo, nb(3, (a, -1)), q, centred)
    out.append(-total / h)
    return out


def _window(fields, n):
    """at() over fields with one ghost layer (index 0 is cell -1)."""
    return lambda f, i, j, k: fields[f][1 + i:1 + i + n[0], 1 + j:1 + j + n[1], 1 + k:1 + k + n[2]]


def _lap(at, f, h):
    return (at(f, 1, 0, 0) + at(f, -1, 0, 0) + at(f, 0, 1, 0) + at(f, 0, -1, 0) + at(f, 0, 0, 1) + at(f, 0, 0, -1)
            - 6 * at(f, 0, 0, 0)) / (h * h)


def _exact_stencils(case, seed):
    h = _spacing(case)
    at = _window([f.double() for f in _stencil_fields(case, seed)], _size(case))
    out = _flux_terms(at, h, case["centred"])
    out[3] = out[3] + _KAPPA * h * _lap(at, 3, h)
    return out


def _exact_flow(case, seed):
    """One forward-Euler step (the first Adams-Bashforth step is one)."""
    n = _size(case)
    h = 1.0 / n[2]
    u, v, w, t = (f.double() for f in _flow_start(case, seed))
    for a, f in enumerate((u, v, w)):
        _close(f, a, _AXES["channel"][a])
    dt = _CFL * min(h / float(f.abs().max()) for f in (u, v, w))
    dt = min(dt, h * h / 6, h * h / (6 * _PR))
    ext = []
    for c, f in enumerate((u, v, w, t)):
        f = f[:n[0], :n[1]]  # the periodic faces once
        f = torch.cat((f[-1:], f, f[:1]), 0)
        f = torch.cat((f[:, -1:], f, f[:, :1]), 1)
        lo, hi = f[:, :, :1], f[:, :, -1:]
        ends = (torch.zeros_like(lo), torch.zeros_like(hi)) if c == 2 else (2 - lo, -hi) if c == 3 else (-lo, -hi)
        ext.append(torch.cat((ends[0], f, ends[1]), 2))
    at = _window(ext, n)
    d = _flux_terms(at, h, False)
    for c in range(3):
        d[c] = d[c] + _PR * _lap(at, c, h)
    d[2] = d[2] + 0.5 * _RA * _PR * (at(3, 0, 0, 0) + at(3, 0, 0, -1))
    d[3] = d[3] + _lap(at, 3, h)
    vel = [f.clone() for f in (u, v, w)]
    for f, g in zip(vel, d):
        f[:n[0], :n[1], :n[2]] += dt * g
    return {"dt": dt, "uvwt": _project(vel, h, _AXES["channel"]) + [t + dt * d[3]]}


def _exact_ensemble(case, seed):
    return None  # closed boxes: each pressure is fixed up to a constant


def _exact_chain(case, seed):
    h, dt, n = _spacing(case), _chain_dt(case), _size(case)
    *start, target = [f.double() for f in _chain_start(case, seed)]
    start = [f.requires_grad_(True) for f in start]
    eig = 0
    for a, m in enumerate(n):
        k = torch.arange(m, device="cuda", dtype=torch.float64)
        eig = eig + ((2 * torch.cos(2 * math.pi * k / m) - 2) / (h * h)).reshape([-1 if q == a else 1 for q in range(3)])
    inv = torch.where(eig.abs() > 1e-9, 1 / eig, torch.zeros_like(eig))
    f = list(start)
    for _ in range(case["steps"]):
        d = _flux_terms(lambda q, i, j, k: torch.roll(f[q], (-i, -j, -k), (0, 1, 2)), h, False)
        new = [x + dt * y for x, y in zip(f, d)]
        div = sum(torch.roll(new[a], -1, a) - new[a] for a in range(3)) / h
        p = torch.fft.ifftn(torch.fft.fftn(div) * inv).real
        f = [new[a] - (p - torch.roll(p, 1, a)) / h for a in range(3)] + [new[3]]
    grads = torch.autograd.grad(0.5 * (f[3] - target).square().sum(), start)
    return {"phi": f[3].detach(), "grads": list(grads)}
