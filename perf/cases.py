"""The work that users of intfadv have it do, as cases for timing and for comparing outputs.

Five kinds of call, each through the package's public entry points:

* ``step``        one ``sim_step`` of a ``TwoPhaseSimulation`` (coupled momentum / VOF advection, forcing, two
                  pressure projections), from a stored mid-run state, as a run restarted from it takes it;
* ``advect``      one ``advect`` (VOF advection alone) in a deformation or vortex field whose sign alternates from
                  pass to pass, so that the interface stays near where it began;
* ``poisson``     one ``ia_poisson_solve`` of a bubbly pressure system from a zero guess;
* ``redistance``  ``LevelSet`` + ``redistaning`` of a droplet field;
* ``net``         the learned preconditioner's network: a training gradient, or a tensor-core forward pass.

The pressure and the Poisson solution are defined up to a constant, so they are returned with their mean taken out.
Step cases solve the pressure to 1e-12 (the large one to 1e-10), so that the outputs are the discretisation's and
not the stopping point's.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "interfaceadvection.jl_gb300"))

import intfadv as ia  # noqa: E402
from intfadv import learned, workloads  # noqa: E402
from intfadv.fields import fzeros, ptr  # noqa: E402

F64 = torch.float64
EPS = 2.220446049250313e-16


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # 2D dam break between walls with the default FP64 solver: the smallest step, bound by latency
        dict(name="dam_2d", kind="step", flow="dam", nx=128, ny=64, nz=0, poisson="fp64", tol=1e-12, normal="WH",
             limiter="Koren"),
        # a 2D droplet with surface tension in a box of odd sizes, mixed solver
        dict(name="droplet_2d_odd", kind="step", flow="droplet", nx=161, ny=97, nz=0, poisson="mixed", tol=1e-12,
             normal="WH", limiter="Koren"),
        # a small rising bubble (periodic x and z, walls in y): parameter sweeps, tests of a set-up
        dict(name="bubble_3d_small", kind="step", flow="bubble", nx=32, ny=64, nz=32, poisson="mixed", tol=1e-12,
             normal="WH", limiter="Koren"),
        # a medium rising bubble in the default all-FP64 mode, at a round size that is no power of two
        dict(name="bubble_3d_fp64", kind="step", flow="bubble", nx=100, ny=200, nz=100, poisson="fp64", tol=1e-12,
             normal="WH", limiter="Koren"),
        # a closed tank of ragged sizes, mixed solver, another normal scheme and limiter
        dict(name="tank_3d_ragged", kind="step", flow="dam", nx=41, ny=35, nz=30, poisson="mixed", tol=1e-12,
             normal="MYC", limiter="vanAlbada1"),
        # the benchmark's grid: the largest step
        dict(name="bubble_3d_large", kind="step", flow="bubble", nx=256, ny=512, nz=256, poisson="mixed", tol=1e-10,
             normal="WH", limiter="Koren"),
        # VOF advection alone: a 2D vortex (latency), and the 3D deformation test at its usual size
        dict(name="advect_2d", kind="advect", nx=100, ny=100, nz=0, normal="WH"),
        dict(name="advect_3d", kind="advect", nx=256, ny=256, nz=256, normal="WH"),
        # the pressure solve by itself, as a program with its own velocity step calls it
        dict(name="poisson_3d", kind="poisson", nx=128, ny=192, nz=160, poisson="mixed", tol=1e-10),
        # level-set reinitialisation over five cells
        dict(name="redistance_3d", kind="redistance", nx=160, ny=128, nz=96, d=5.0, dtau=0.5),
        # the network of the learned preconditioner: one gradient of its training, one forward of its use
        dict(name="net_train", kind="net", job="grad", batch=4, nx=64, ny=64, nz=64),
        dict(name="net_forward", kind="net", job="forward", batch=1, nx=128, ny=256, nz=128),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _even(n):
    return n + (n & 1)


def _affordable(nx, ny, nz):
    """The sizes, made multiples of 2, 4, ... until a solve is no longer dominated by sizes that do not halve: where
    one is odd the multigrid stops, and a grid costs about its cells times its longest side on that last level."""
    m = 1
    while True:
        n = [-(-v // m) * m for v in (nx, ny, nz)]
        last = [v for v in n if v]
        while all(v % 2 == 0 and v >= 4 for v in last) and math.prod(last) > 512:
            last = [v // 2 for v in last]
        if math.prod(last) * max(last) <= 2_000_000:
            return n
        m *= 2


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "advect", "advect", "poisson", "redistance", "net"])
    two_d = rng.random() < 0.35
    if kind == "step":
        flow = rng.choice(["bubble", "dam", "droplet"])
        poisson = rng.choice(["mixed", "mixed", "fp64"])
        hi2, hi3 = (400, 160) if poisson == "mixed" else (300, 110)
        nx, ny = (_log_int(rng, 40, hi2), _log_int(rng, 40, hi2)) if two_d else (_log_int(rng, 24, hi3),
                                                                                 _log_int(rng, 24, hi3))
        nz = 0 if two_d else _log_int(rng, 24, hi3)
        if flow == "bubble":             # periodic dimensions
            nx, nz = _even(nx), _even(nz)
        nx, ny, nz = _affordable(nx, ny, nz)
        return dict(kind="step", flow=flow, nx=nx, ny=ny, nz=nz, poisson=poisson, tol=1e-12,
                    normal=rng.choice(["WH", "WH", "WY", "MYC", "Y"]),
                    limiter=rng.choice(["Koren", "Koren", "minmod", "vanAlbada1", "superbee"]))
    if kind == "advect":
        a, b = (40, 1500) if two_d else (24, 256)
        return dict(kind="advect", nx=_log_int(rng, a, b), ny=_log_int(rng, a, b), nz=0 if two_d else _log_int(rng, a, b),
                    normal=rng.choice(["WH", "WH", "MYC", "WY", "Column"]))
    if kind == "poisson":
        m = 16
        return dict(kind="poisson", nx=m * rng.randint(2, 10), ny=m * rng.randint(2, 12), nz=m * rng.randint(2, 10),
                    poisson=rng.choice(["mixed", "fp64"]), tol=1e-10)
    if kind == "redistance":
        return dict(kind="redistance", nx=_log_int(rng, 24, 200), ny=_log_int(rng, 24, 200),
                    nz=0 if two_d else _log_int(rng, 24, 160), d=float(rng.choice([2, 4, 5])), dtau=0.5)
    job = rng.choice(["grad", "forward"])
    hi = 16 if job == "grad" else 32
    return dict(kind="net", job=job, batch=rng.randint(1, 4) if job == "grad" else 1, nx=4 * rng.randint(4, hi),
                ny=4 * rng.randint(4, hi), nz=4 * rng.randint(4, hi))


# ------------------------------------------------------------------------------------------------ inputs
def _dims(case):
    return (case["nx"], case["ny"]) + ((case["nz"],) if case["nz"] else ())


def _gen(seed):
    return np.random.Generator(np.random.PCG64(seed))


def _fraction(sdf_values):
    """Fraction of the dark fluid (sdf < 0) with a one-cell transition."""
    return torch.clamp(0.5 - sdf_values, 0.0, 1.0)


def _centres(dims, device="cuda"):
    """Cell-centre coordinates of the ghost-inclusive grid, broadcastable in the order (x, y[, z])."""
    D = len(dims)
    return [(torch.arange(n + 2, dtype=F64, device=device) - 0.5).view([-1 if e == d else 1 for e in range(D)])
            for d, n in enumerate(dims)]


def _ball(dims, rng, rel=0.15, at=0.35, jitter=0.05):
    c = [n * (at + jitter * rng.uniform(-1, 1)) for n in dims]
    r = rel * min(dims) * (1 + 0.1 * rng.uniform(-1, 1))

    def sdf(x):
        return torch.sqrt(sum((xi - ci) ** 2 for xi, ci in zip(x, c))) - r
    return sdf


def _stirred(dims, periodic, amp):
    """Face velocities of a single cell of stirring in x and y (nothing through a wall)."""
    nx, ny = dims[0], dims[1]
    kx = (2 if 0 in periodic else 1) * math.pi / nx
    ky = (2 if 1 in periodic else 1) * math.pi / ny

    def u0(i, x):
        if i == 0:
            return amp * torch.sin(kx * x[0]) * torch.cos(ky * x[1])
        if i == 1:
            return -amp * kx / ky * torch.cos(kx * x[0]) * torch.sin(ky * x[1])
        return 0.0 * x[0]
    return u0


def _prepare_step(case, seed):
    rng, dims = _gen(seed), _dims(case)
    D = len(dims)
    kw = dict(poisson=case["poisson"], poisson_tol=case["tol"], poisson_itmx=400, normalScheme=case["normal"],
              λ=case["limiter"])
    down = lambda G: tuple(-G if e == 1 else 0.0 for e in range(D))   # noqa: E731
    if case["flow"] == "dam":
        # a water column beside a wall, run a few steps from a weak stirring
        a, b = dims[0] * (0.25 + 0.05 * rng.uniform(-1, 1)), dims[1] * (0.5 + 0.05 * rng.uniform(-1, 1))
        L, per = float(min(dims)), ()
        kw.update(λρ=1e-3, λμ=1 / 55, ν=L / 1000, g=down(1 / L),
                  InterfaceSDF=lambda x: torch.maximum(x[0] - a, x[1] - b) + 0.0 * sum(x))
    elif case["flow"] == "droplet":
        # a heavy droplet in light fluid, closed box, surface tension, no gravity
        L, per = float(min(dims)), ()
        kw.update(λρ=1e-2, λμ=1e-2, ν=0.02, η=0.02, InterfaceSDF=_ball(dims, rng, rel=0.2, at=0.45))
    else:
        # the benchmark's rising bubble (Eo = 10, Mo = 1e-3) at this size
        p = workloads.bubble_params(min(dims))
        L, per = float(dims[0]), tuple(d for d in (0, 2) if d < D)
        ball = _ball(dims, rng, rel=0.125, at=0.5)
        kw.update(λρ=p["lrho"], λμ=p["lmu"], ν=p["mu"], η=p["sigma"], g=down(p["G"]), InterfaceSDF=lambda x: -ball(x))
    amp = 0.2 * (1 + 0.2 * rng.uniform(-1, 1))
    sim = ia.TwoPhaseSimulation(dims, (0.0,) * D, L, U=1.0, perdir=per, u0=_stirred(dims, per, amp), **kw)
    for _ in range(2):
        ia.sim_step(sim)
    fl, it = sim.flow, sim.intf
    return dict(sim=sim, u=fl.u.clone(), f=it.f.clone(), p=fl.p.clone(), dts=list(fl.Δt))


def _run_step(s):
    sim = s["sim"]
    fl, it = sim.flow, sim.intf
    fl.u.copy_(s["u"])
    it.f.copy_(s["f"])
    fl.p.copy_(s["p"])
    fl.Δt[:] = s["dts"]
    ia.sim_step(sim)
    return dict(u=fl.u, f=it.f, p=_mean_free(fl.p), dt=fl.Δt[-1])


def _mean_free(a):
    b = a[tuple(slice(1, -1) for _ in a.shape)]
    return b - b.mean()


def _deformation(dims, device="cuda"):
    """Divergence-free face velocities, zero through every wall, largest component 1: the curl of a vector potential
    (3D, LeVeque's deformation) or of a stream function (2D, the single vortex) sampled on edges."""
    D = len(dims)

    def axis(d, face):
        n = dims[d]
        x = (torch.arange(n + 3, dtype=F64, device=device) - (1.0 if face else 0.5)) / n
        return x.view([-1 if e == d else 1 for e in range(D)])

    def S(d):
        x = axis(d, True)
        v = torch.sin(math.pi * x) ** 2
        return torch.where((x == 0) | (x == 1), torch.zeros_like(v), v)

    def T(d):
        return torch.sin(2 * math.pi * axis(d, False))

    def diff(a, d):
        n = a.shape[d] - 1
        return a.narrow(d, 1, n) - a.narrow(d, 0, n)

    def cut(a):
        for d in range(D):
            a = a.narrow(d, 0, dims[d] + 2)
        return a
    if D == 2:
        psi = S(0) * S(1) * min(dims)
        comps = [diff(psi, 1), -diff(psi, 0)]
    else:
        A2 = -S(0) * T(1) * S(2) * min(dims)
        A3 = S(0) * S(1) * T(2) * min(dims)
        comps = [cut(diff(A3, 1)) - cut(diff(A2, 2)), -diff(A3, 0), diff(A2, 0)]
    comps = [cut(c) for c in comps]
    top = max(float(c.abs().max()) for c in comps)
    return [c / top for c in comps]


def _advect_inputs(case, seed):
    rng, dims = _gen(seed), _dims(case)
    f = _fraction(_ball(dims, rng)(_centres(dims)))
    # zero-gradient ghosts of a field that is empty near the walls are the field itself
    U = _deformation(dims)
    t = 0.3 * rng.uniform()
    return f, U, (math.cos(math.pi * t), math.cos(math.pi * (t + 0.01))), 0.45


def _prepare_advect(case, seed):
    dims = _dims(case)
    f, U, (c0, c1), dt = _advect_inputs(case, seed)
    flow = ia.Flow(dims, (0.0,) * len(dims), Δt=dt)
    intf = ia.cVOF(dims, lrho=1e-3, normalScheme=case["normal"])
    intf.f.copy_(f)
    fields = []
    for sign in (1.0, -1.0):
        for c in ((c0, c1) if sign > 0 else (c1, c0)):
            a = fzeros(flow.u.shape)
            for d, comp in enumerate(U):
                a[..., d].copy_(sign * c * comp)
            fields.append(a)
    return dict(flow=flow, intf=intf, fields=fields, k=0)


def _run_advect(s):
    k, flow, intf = s["k"], s["flow"], s["intf"]
    s["k"] = 1 - k
    ia.advect(flow, intf, u1=s["fields"][2 * k], u2=s["fields"][2 * k + 1])
    return dict(f=intf.f, rhouf=intf.rhouf, cbar=intf.cbar)


def _poisson_inputs(case, seed):
    """Face coefficients 1/ρ of a few bubbles and the divergence of a smooth and slightly noisy velocity: x and z
    periodic, walls in y.  Arrays over the ghost-inclusive grid, index order (x, y, z[, component])."""
    dims, rng = _dims(case), _gen(seed)
    lrho = 1e-3
    x = _centres(dims)
    sdf = None
    for _ in range(4):
        c = [n * rng.uniform(0.2, 0.8) for n in dims]
        r = rng.uniform(0.08, 0.15) * min(dims)
        s = r - torch.sqrt(sum((xi - ci) ** 2 for xi, ci in zip(x, c)))
        sdf = s if sdf is None else torch.maximum(sdf, s)
    rho = lrho + (1 - lrho) * _fraction(sdf)
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    L = torch.zeros(tuple(n + 2 for n in dims) + (3,), dtype=F64, device="cuda")
    z = torch.zeros(tuple(n + 2 for n in dims), dtype=F64, device="cuda")
    inner = (slice(1, -1),) * 3
    ri = rho[inner]
    for d in range(3):
        Ld = 2.0 / (ri + ri.roll(1, d))
        v = 0.1 * torch.randn(ri.shape, generator=gen, dtype=F64, device="cuda")
        for e in range(3):
            v = v + torch.sin(2 * math.pi * (x[e][tuple(slice(1, -1) if q == e else slice(None) for q in range(3))]
                                             / dims[e] * (1 + d) + rng.uniform()))
        v = 0.01 * v
        if d == 1:
            Ld.narrow(1, 0, 1).zero_()
            v.narrow(1, 0, 1).zero_()
        L[..., d][inner] = Ld
        hi = L[..., d].narrow(d, dims[d] + 1, 1)
        hi[tuple(slice(None) if q == d else slice(1, -1) for q in range(3))] = Ld.narrow(d, 0, 1)
        z[inner] += v.roll(-1, d) - v
    return L, z


def _prepare_poisson(case, seed):
    L, z = _poisson_inputs(case, seed)
    h = ia.Handle(ia.make_config(_dims(case), perdir=(0, 2), lrho=1e-3, poisson=case["poisson"]))
    fL, fz, fx = fzeros(L.shape), fzeros(z.shape), fzeros(z.shape)
    fL.copy_(L)
    fz.copy_(z)
    return dict(h=h, L=fL, z=fz, x=fx, tol=case["tol"])


def _run_poisson(s):
    s["x"].zero_()
    it, res = ctypes.c_int32(), ctypes.c_double()
    code = s["h"].call("ia_poisson_solve", ptr(s["x"]), ptr(s["z"]), ptr(s["L"]), s["tol"], 400, ctypes.byref(it),
                       ctypes.byref(res))
    if code != 0:
        raise RuntimeError(f"ia_poisson_solve: code {code}, residual {res.value}")
    return dict(x=_mean_free(s["x"]))


def _levelset_f(case, seed):
    dims = _dims(case)
    return _fraction(0.5 * _ball(dims, _gen(seed), rel=0.3, at=0.5)(_centres(dims)))


def _prepare_redistance(case, seed):
    dims = _dims(case)
    sim = ia.TwoPhaseSimulation(dims, (0.0,) * len(dims), float(dims[0]), U=1.0, perdir=(0,))
    sim.intf.f.copy_(_levelset_f(case, seed))
    return dict(sim=sim, d=case["d"], dtau=case["dtau"])


def _run_redistance(s):
    ls = ia.LevelSet(s["sim"])
    ia.redistaning(ls, s["d"], s["dtau"])
    return dict(phi=ls.ϕ)


CIN, COUT = (4, 16, 32, 32, 32, 16), (16, 32, 32, 32, 16, 1)


def _net_weights(rng):
    w = []
    for ci, co in zip(CIN, COUT):
        w += [rng.normal(0.0, math.sqrt(2.0 / (27 * ci)), 27 * co * ci), rng.normal(0.0, 0.02, co)]
    return np.concatenate(w).astype(np.float32)


def _net_inputs(case, seed):
    """A residual scaled to 1 and face coefficients λρ/ρ of a bubble (channels), and a smooth correction (target)."""
    B, dims = case["batch"], (case["nz"], case["ny"], case["nx"])
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    rng = _gen(seed)
    x0 = torch.zeros((B,) + tuple(n + 2 for n in dims) + (4,), device="cuda")
    tgt = torch.zeros(x0.shape[:-1], device="cuda")
    x = [c[tuple(slice(1, -1) if q == e else slice(None) for q in range(3))] for e, c in enumerate(_centres(dims))]
    inner = (slice(1, -1),) * 3
    for b in range(B):
        f = _fraction(-_ball(dims, rng, rel=0.25, at=0.5)(x))
        x0[b][inner][..., 0] = (torch.randn(dims, generator=gen, device="cuda") / 5).clamp(-1, 1)
        for d in range(3):
            x0[b][inner][..., 1 + d] = (1e-3 / (1e-3 + 0.999 * 0.5 * (f + f.roll(1, 2 - d)))).float()
        ph = rng.uniform(0, 1, 3)
        tgt[b][inner] = sum(torch.cos(2 * math.pi * (x[e] / dims[e] + ph[e])) for e in range(3)).float() / 3
    return x0, tgt, _net_weights(rng)


def _prepare_net(case, seed):
    x0, tgt, w = _net_inputs(case, seed)
    net = learned.Net()
    net.set_params(w)
    return dict(net=net, x0=x0, tgt=tgt, job=case["job"])


def _run_net(s):
    if s["job"] == "grad":
        loss, grad = s["net"].loss_grad(s["x0"], s["tgt"])
        return dict(loss=loss, grad=grad)
    return dict(out=s["net"].forward(s["x0"], tensor_cores=True))


_PREPARE = dict(step=_prepare_step, advect=_prepare_advect, poisson=_prepare_poisson, redistance=_prepare_redistance,
                net=_prepare_net)
_RUN = dict(step=_run_step, advect=_run_advect, poisson=_run_poisson, redistance=_run_redistance, net=_run_net)


def prepare(case, seed):
    s = _PREPARE[case["kind"]](case, seed)
    s["kind"] = case["kind"]
    return s


def run(state):
    return _RUN[state["kind"]](state)


def work(case):
    """Each input read once and each output written once; the operations of the discrete formulas applied once (a
    solve counts one application of its operator, an iteration count is the solver's business)."""
    dims = _dims(case)
    D, n = len(dims), math.prod(dims)
    kind = case["kind"]
    if kind == "step":       # u, f, p in and out, restored from the stored state
        return dict(bytes=8.0 * n * 4 * (D + 2), flops=2.0 * n * (60 * D * D + 60))
    if kind == "advect":     # f and both velocities in, ρuf and c̄ out, the changed fractions are few
        return dict(bytes=n * (8.0 + 16 * D + 8 * D + 1), flops=6.0 * n * D)
    if kind == "poisson":
        return dict(bytes=8.0 * n * (D + 2), flops=n * (4.0 * D + 2))
    if kind == "redistance":
        return dict(bytes=16.0 * n, flops=3.0 * round(case["d"] / case["dtau"]) * n * (16 * D + 12))
    cells = n * case["batch"]
    macs = sum(27 * ci * co / s for ci, co, s in zip(CIN, COUT, (1, 8, 64, 8, 1, 1)))
    if case["job"] == "grad":
        return dict(bytes=20.0 * cells, flops=6.0 * macs * cells)
    return dict(bytes=20.0 * cells, flops=2.0 * macs * cells)


# ------------------------------------------------------------------------------------------------ in 64 bits
def exact(case, seed):
    """The outputs in plain torch FP64; None for a whole step (it would restate the whole framework) and for VOF
    advection with another normal scheme than the default."""
    kind = case["kind"]
    if kind == "poisson":
        return dict(x=_exact_poisson(*_poisson_inputs(case, seed)))
    if kind == "redistance":
        return dict(phi=_exact_redistance(_levelset_f(case, seed), case["d"], case["dtau"], periodic=(0,)))
    if kind == "net":
        return _exact_net(case, seed)
    if kind == "advect" and case["normal"] == "WH":
        return _exact_advect(case, seed)
    return None


def _exact_poisson(L, z):
    """Jacobi-preconditioned CG on A x = z, (A x)_I = Σ_d L_d(I)(x(I-d) - x(I)) + L_d(I+d)(x(I+d) - x(I))."""
    inner = (slice(1, -1),) * 3
    Li = [L[..., d][inner].contiguous() for d in range(3)]
    z = z[inner].contiguous()
    # the lower wall face has no coefficient, and it stands for the upper one too: rolling wraps on all three

    def A(v):
        out = torch.zeros_like(v)
        for d in range(3):
            flux = Li[d] * (v.roll(1, d) - v)
            out += flux - flux.roll(-1, d)
        return out
    diag = -sum(l + l.roll(-1, d) for d, l in enumerate(Li))
    z = z - z.mean()
    x, r = torch.zeros_like(z), z.clone()
    p, rho = None, None
    goal = 1e-14 * float(z.norm())
    for it in range(20000):
        s = r / diag
        rho, old = (r * s).sum(), rho
        p = s if p is None else s + (rho / old) * p
        q = A(p)
        a = rho / (p * q).sum()
        x += a * p
        r -= a * q
        if it % 50 == 49 and float(r.norm()) <= goal:
            break
    return x - x.mean()


def _exact_redistance(f, d, dtau, periodic):
    D = f.dim()
    phi = 2 * f - 1
    ini = phi.clone()
    inner = (slice(1, -1),) * D

    def ghosts(a):
        for e in range(D):
            n = a.shape[e]
            lo, hi = (n - 2, 1) if e in periodic else (1, n - 2)
            a.narrow(e, 0, 1).copy_(a.narrow(e, lo, 1).clone())
            a.narrow(e, n - 1, 1).copy_(a.narrow(e, hi, 1).clone())

    def minmod(a, b):
        return torch.where(a.abs() <= b.abs(), a, b)

    def grad2(a, e, s):
        """ENO2 upwind square of the derivative along e of the interior cells."""
        m = a[tuple(slice(None) if q == e else slice(1, -1) for q in range(D))]
        n = m.shape[e]
        at = m.narrow
        below = at(e, n - 3, 1) if e in periodic else at(e, 0, 1)
        above = at(e, 2, 1) if e in periodic else at(e, n - 1, 1)
        m = torch.cat([below, m, above], e)
        a_, b, c, d_, e_ = (m.narrow(e, k, n - 2) for k in range(5))
        mid = minmod(d_ - 2 * c + b, c - 2 * b + a_)
        dR = d_ - c - minmod(e_ - 2 * d_ + c, d_ - 2 * c + b) / 2
        dL = c - b + mid / 2
        wR, wL = dR * s, dL * s
        return torch.where((wR < 0) & (wR + wL < 0), dR * dR,
                           torch.where((wL > 0) & (wR + wL > 0), dL * dL, torch.zeros_like(dR)))
    si = torch.sign(ini[inner])
    for _ in range(round(d / dtau)):
        phi0 = phi.clone()
        for alpha in (0.0, 3 / 4, 1 / 3):
            g = sum(grad2(phi, e, si) for e in range(D))
            rhs = ini[inner] * (1 - torch.sqrt(g))
            phi[inner] = alpha * phi0[inner] + (1 - alpha) * (phi[inner] + dtau * rhs)
            ghosts(phi)
    return phi


def _exact_net(case, seed):
    x0, tgt, w = _net_inputs(case, seed)
    params, o = [], 0
    for ci, co in zip(CIN, COUT):
        n = 27 * co * ci
        params.append(torch.tensor(w[o:o + n], dtype=F64, device="cuda").view(27, co, ci))
        params.append(torch.tensor(w[o + n:o + n + co], dtype=F64, device="cuda"))
        o += n + co
    grad = case["job"] == "grad"
    for p in params:
        p.requires_grad_(grad)

    def conv(v, l):
        W, b = params[2 * l], params[2 * l + 1]
        n = v.shape[1:4]
        v = torch.nn.functional.pad(v, (0, 0, 1, 1, 1, 1, 1, 1))
        out = b
        for t in range(27):
            dz, dy, dx = t // 9, t // 3 % 3, t % 3
            out = out + v[:, dz:dz + n[0], dy:dy + n[1], dx:dx + n[2]] @ W[t].T
        return out

    def pool(v):
        B, nz, ny, nx, c = v.shape
        return v.view(B, nz // 2, 2, ny // 2, 2, nx // 2, 2, c).mean((2, 4, 6))

    def up(v):
        for e in (1, 2, 3):
            v = v.repeat_interleave(2, e)
        return v

    def forward(x):
        a1 = conv(x, 0).relu()
        a2 = conv(pool(a1), 1).relu()
        a3 = conv(pool(a2), 2).relu()
        a4 = conv(up(a3) + a2, 3).relu()
        return conv(conv(up(a4), 4).relu() + a1, 5)[..., 0]
    inner = (slice(None),) + (slice(1, -1),) * 3
    x, y = x0[inner].double(), tgt[inner].double()
    if not grad:
        out = torch.zeros(x0.shape[:-1], dtype=F64, device="cuda")
        out[inner] = forward(x)
        return dict(out=out)
    total, n = 0.0, y.numel()
    for b in range(x.shape[0]):     # one sample at a time: the saved activations of 27 taps are large
        loss = ((forward(x[b:b + 1]) - y[b:b + 1]) ** 2).sum() / n
        loss.backward()
        total += float(loss)
    return dict(loss=total, grad=torch.cat([p.grad.reshape(-1) for p in params]))


# ---- one split VOF step with Huang-Weymouth normals and the Scardovelli-Zaleski plane relations
def _plane_constant(m, v):
    """α of the plane Σ m x = α that cuts the fraction v <= 1/2 off the unit cell; m sorted, Σ m = 1, [k, 3]."""
    m1, m2, m3 = m.unbind(1)
    m12 = m1 + m2
    p = 6 * m1 * m2 * m3
    v1 = torch.where(m2 == 0, torch.ones_like(m2), m1 / m2) * m1 / (6 * m3)
    v2 = v1 + (m2 - m1) / (2 * m3)
    low = m3 < m12
    v3 = torch.where(low, (m3 * m3 * (3 * m12 - m3) + m1 * m1 * (m1 - 3 * m3) + m2 * m2 * (m2 - 3 * m3)) / p,
                     m12 / (2 * m3))

    def root(c0, c1, c2, c3):
        a0, a1, a2 = c0 / c3, c1 / c3, c2 / c3
        p0 = a1 / 3 - a2 * a2 / 9
        q0 = (a1 * a2 - 3 * a0) / 6 - a2 ** 3 / 27
        a = q0 / torch.sqrt(-p0 ** 3)
        a = torch.where(a * a <= 1, a, torch.zeros_like(a))
        t = torch.acos(a) / 3
        return torch.sqrt(-p0) * (math.sqrt(3.0) * torch.sin(t) - torch.cos(t)) - a2 / 3
    one = torch.ones_like(v)
    out = torch.where(low, root(m1 ** 3 + m2 ** 3 + m3 ** 3 - p * v, -3 * (m1 * m1 + m2 * m2 + m3 * m3), 3 * one,
                                -2 * one), m3 * v + m12 / 2)
    out = torch.where(v < v3, root(m1 ** 3 + m2 ** 3 - p * v, -3 * (m1 * m1 + m2 * m2), 3 * m12, -one), out)
    out = torch.where(v < v2, (m1 + torch.sqrt(m1 * m1 + 8 * m2 * m3 * (v - v1).clamp(min=0))) / 2, out)
    return torch.where(v < v1, (p * v).clamp(min=0) ** (1 / 3), out)


def _plane_volume(m, a):
    """The fraction below Σ m x = a <= 1/2 of the unit cell; m sorted, Σ m = 1, [k, 3]."""
    m1, m2, m3 = m.unbind(1)
    m12 = m1 + m2
    p6 = 6 * m1 * m2 * m3
    c12 = m1 * m1 * (m1 - 3 * a) + m2 * m2 * (m2 - 3 * a)
    out = torch.where(m3 < m12, (a * a * (3 - 2 * a) + c12 + m3 * m3 * (m3 - 3 * a)) / p6, (2 * a - m12) / (2 * m3))
    out = torch.where(a < torch.minimum(m3, m12), (a * a * (3 * m12 - a) + c12) / p6, out)
    r = torch.where(m2 == 0, torch.ones_like(m2), m1 / m2)
    out = torch.where(a < m2, a * (a - m1) / (2 * m2 * m3) + r * m1 / (6 * m3), out)
    return torch.where(a < m1, a ** 3 / p6, out)


def _wh_normal(f, cells, D):
    """Huang-Weymouth normals of the listed cells ([k, D] coordinates) of the ghosted field f."""
    k = torch.arange(len(cells), device=f.device)

    def at(off):
        return f[tuple((cells[:, e] + off[:, e]) for e in range(D))]

    def unit(axis, s):     # [k, D] offset of s along the axis of each cell
        o = torch.zeros((len(cells), D), dtype=torch.long, device=f.device)
        o[k, axis] = s
        return o

    def col3(off, axis):
        one = unit(axis, 1)
        return at(off) + at(off - one) + at(off + one)

    def axis(d):
        return torch.full((len(cells),), d, dtype=torch.long, device=f.device)
    n = torch.stack([at(unit(axis(d), -1)) - at(unit(axis(d), 1)) for d in range(D)], 1)
    dom = (n * n).argmax(1)
    flat = torch.zeros((len(cells), D), dtype=torch.long, device=f.device)
    cols = []
    for d in range(D):
        ax = axis(d)
        v = (col3(unit(ax, -1), dom) - col3(unit(ax, 1), dom)) / 2
        cols.append(torch.where(dom == d, torch.where(n[:, d] >= 0, 1.0, -1.0).to(F64), v))
    n = torch.stack(cols, 1)
    ad = (n * n).argmax(1)
    big = n[k, ad].abs()
    big = torch.where(big == 0, torch.ones_like(big), big)
    dstep = torch.where(torch.signbit(n[k, ad]), -1, 1)
    n = n / big[:, None]
    for d in range(D):
        ax = axis(d)
        slope, neg = n[:, d].abs(), torch.signbit(n[:, d])
        step = torch.where(neg, -1, 1)
        hl, hc, hr = col3(unit(ax, -step), ad), col3(flat, ad), col3(unit(ax, step), ad)
        sh, tri = hl + hc + hr, 4.5 * slope
        lim = torch.minimum(1 / (2 * slope), tri)
        sgn = torch.where(neg, -1.0, 1.0).to(F64)
        wb, wt = col3(unit(ad, -dstep), ax), col3(unit(ad, dstep), ax)
        v = n[:, d]
        v = torch.where((sh < tri) & (wb > lim), torch.copysign((hl - 0.5) / (wb - 0.5), sgn), v)
        v = torch.where((sh > 9 - tri) & (wt < 3 - lim), torch.copysign((2.5 - hr) / (2.5 - wt), sgn), v)
        keep = (ad == d) | ((tri <= sh) & (sh <= 9 - tri))
        n = torch.cat([n[:, :d], torch.where(keep, n[:, d], v)[:, None], n[:, d + 1:]], 1)
    return n


def _sorted_m(n):
    m = n.abs()
    t = m.sum(1)
    m = m / t[:, None]
    if m.shape[1] == 2:        # a 2D cell is a 3D one with no slope along the third axis
        m = torch.cat([torch.zeros_like(m[:, :1]), m], 1)
    return m.sort(1).values, t


def _exact_advect(case, seed):
    dims = _dims(case)
    D = len(dims)
    f, U, (c0, c1), dt = _advect_inputs(case, seed)
    f = f.expand(tuple(n + 2 for n in dims)).clone()
    lrho, clean = 1e-3, 10 * EPS
    rhouf = torch.zeros(f.shape + (D,), dtype=F64, device=f.device)
    cbar = (f >= 0.5).to(torch.int8)
    for i in range(1, D + 1):
        d = (1 + i) % D
        u = U[d].expand(f.shape)
        dl = dt / 2 * (c0 * u + c1 * u)
        dl[tuple(slice(0, 1) if e == d else slice(None) for e in range(D))] = 0
        donor = torch.where(dl > 0, f.roll(1, d), f)
        F = donor * dl
        face = torch.ones_like(f, dtype=torch.bool)
        for e in range(D):
            face.narrow(e, 0, 1).zero_()
            if e != d:
                face.narrow(e, dims[e] + 1, 1).zero_()
        mixed = (face & (dl != 0) & (donor > 0) & (donor < 1)).nonzero()
        if len(mixed):
            cells = mixed.clone()
            dlm, g = dl[tuple(mixed.T)], donor[tuple(mixed.T)]
            cells[:, d] -= (dlm > 0).long()
            n = _wh_normal(f, cells, D)
            m, t = _sorted_m(n)
            v = torch.minimum(g, 1 - g)
            a = torch.where(g == 0.5, torch.full_like(g, 0.5), _plane_constant(m, v))
            alpha = torch.where(g < 0.5, a, 1 - a) * t + n.clamp(max=0).sum(1)
            b = torch.where(dlm > 0, alpha - n[:, d] * (1 - dlm), alpha)
            n = n.clone()
            n[:, d] *= dlm.abs()
            m, t = _sorted_m(n)
            a = (b - n.clamp(max=0).sum(1)) / t
            w = torch.minimum(a, 1 - a)
            vol = _plane_volume(m, w)
            vol = torch.where(a < 0.5, vol, 1 - vol)
            vol = torch.where((a <= 0) | (a == 0.5) | (a >= 1), a.clamp(0, 1), vol)
            F[tuple(mixed.T)] = torch.where(n.abs().sum(1) == 0, g, vol) * dlm
        F = torch.where(face, F, torch.zeros_like(F))
        rhouf[..., d] = torch.where(face, dl * lrho + (1 - lrho) * F, torch.zeros_like(F))
        du = (c0 + c1) * (u.roll(-1, d) - u)
        inner = (slice(1, -1),) * D
        new = f + ((F - F.roll(-1, d)) + cbar.to(F64) * du * dt / 2)
        new = torch.where(new < clean, torch.zeros_like(new), torch.where(new > 1 - clean, torch.ones_like(new), new))
        f[inner] = new[inner]
        for e in range(D):
            f.narrow(e, 0, 1).copy_(f.narrow(e, 1, 1).clone())
            f.narrow(e, dims[e] + 1, 1).copy_(f.narrow(e, dims[e], 1).clone())
    return dict(f=f, rhouf=rhouf, cbar=cbar)
