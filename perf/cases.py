"""The work that a user of this package has it do, as measurable cases.

A registration is a loop of a few device calls: certify a displacement, evaluate a line-search trial against its base,
form the gradient (and, once per outer step, the joint outer gradients), apply the DST-I Poisson preconditioner, and
once per subproblem build its metric.  The component cases are these calls, each as a program (the solver loop, or a
host loop that drives the package) makes it, on states like those of a running solve: smooth displacements of a
voxel or two, with a region of strongly compressed cells where the localized barrier is active.  The whole calls are
the registrations themselves: the certified solve from u = 0 in both forms, and the pyramid route from host images.

Grids are those that the package's configurations, tests and benchmark use (32^3, 48^3, 96^3, 128x144x128,
160x192x224, 256^3) and uneven ones between them; voxels are 1 mm or anisotropic.
"""
import math

import numpy as np
import torch

from seq_vp_3d_b200 import certificate, preopt, solver
from seq_vp_3d_b200.grid import grid_from_shape
from seq_vp_3d_b200.pair import DevicePair
from seq_vp_3d_b200.synthetic import default_weights

F64 = torch.float64
ISO, ANISO = (1., 1., 1.), (.9, 1., 1.25)
ACTIVATION = .05
LARGEST = 255 ** 3      # cells of the largest grid in use


def _case(name, kind, shape, **more):
    nz, ny, nx = shape
    c = dict(kind=kind, nz=nz, ny=ny, nx=nx, aniso=False, form="plain", steps=0)
    if name:
        c["name"] = name
    c.update(more)
    return c


def listed():
    return [
        # the smallest certificate: every trial of a 32^3 registration pays it, launches and the record's read-back
        _case("certify_32", "certify", (32, 32, 32)),
        # the whole-cell certificate of a head-sized field, as every trial and every exported field takes it
        _case("certify_head", "certify", (224, 192, 160)),
        # a line-search trial of a small request (warp, energies, differences, activity mask)
        _case("trial_48", "trial", (48, 48, 48)),
        # the same on the largest grid in use
        _case("trial_256", "trial", (256, 256, 256)),
        # the gradient of one PG step on a head-sized pair
        _case("gradient_head", "gradient", (224, 192, 160)),
        # the outer step's joint gradients (F, D, E) on an uneven odd grid with anisotropic voxels
        _case("outer_ragged", "outer", (131, 97, 113), aniso=True),
        # the preconditioned direction of one PG step, float64 tensor-core passes
        _case("direction_head", "direction", (224, 192, 160)),
        # the same in the mixed form (3xTF32 passes) on an uneven odd grid with anisotropic voxels
        _case("direction_ragged_mixed", "direction", (119, 165, 141), aniso=True, form="mixed"),
        # the metric of one subproblem: image shift, GGN diagonal, node JD measure, scale
        _case("metric_128", "metric", (128, 144, 128)),
        # a small registration: certified outer steps on 32^3, where host decisions and launches count
        _case("solve_32", "solve", (32, 32, 32), steps=4),
        # outer steps of the head-sized registration in the mixed form
        _case("solve_head_mixed", "solve", (224, 192, 160), form="mixed", steps=2),
        # the pyramid route end to end from host images: pre-optimizer, certified transfer, certified solve
        _case("register_96", "register", (96, 96, 96), steps=3),
    ]


def draw(rng):
    """Another call of the same ranges: axis lengths spread over their logarithm, odd ones among them."""
    kind = rng.choice(["certify", "trial", "gradient", "outer", "direction", "metric", "solve", "register"])
    lo, hi = {"solve": (24, 192), "register": (40, 160)}.get(kind, (24, 256))
    size = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    shape = [min(256, max(20, int(round(size * math.exp(rng.uniform(-.25, .25)))))) for _ in range(3)]
    if kind == "register":       # its coarsest level (an eighth) needs five nodes per axis
        shape = [max(36, n) for n in shape]
    form = "mixed" if kind in ("direction", "solve", "register") and rng.random() < .4 else "plain"
    steps = rng.randint(1, 2) if kind in ("solve", "register") else 0
    return _case(None, kind, shape, aniso=rng.random() < .4, form=form, steps=steps)


# ------------------------------------------------------------------------------------------------------- inputs
def _grid(c):
    return grid_from_shape((c["nz"], c["ny"], c["nx"]), ANISO if c["aniso"] else ISO)


def _weights(c):
    return default_weights((c["nz"], c["ny"], c["nx"]), ANISO if c["aniso"] else ISO)


def _bumps(shape, gen, count, sigma):
    """Per bump its three axis profiles exp(-(k - c)^2 / (2 s^2)), (count, n) each, centres in the middle 60%."""
    out = []
    s = sigma[0] + (sigma[1] - sigma[0]) * torch.rand(count, 1, generator=gen, device="cuda", dtype=F64)
    for n in shape:
        ctr = n * (.2 + .6 * torch.rand(count, 1, generator=gen, device="cuda", dtype=F64))
        out.append((ctr, s, torch.arange(n, device="cuda", dtype=F64)))
    return out


def _sum(bumps, amp, shift=None):
    p = [torch.exp(-(k - c - (0. if shift is None else shift[:, a:a + 1])) ** 2 / (2 * s * s))
         for a, (c, s, k) in enumerate(bumps)]
    return torch.einsum("b,bz,by,bx->zyx", amp, *p)


def _images(c, gen):
    """Fixed: Gaussian blobs normalised to [0, 1] with 1% noise; moving: the blobs moved by about a voxel."""
    shape = (c["nz"], c["ny"], c["nx"])
    w = max(2., min(shape) / 12)
    b = _bumps(shape, gen, 24, (w, 2.5 * w))
    amp = .2 + .8 * torch.rand(24, generator=gen, device="cuda", dtype=F64)
    shift = .8 * torch.randn(24, 3, generator=gen, device="cuda", dtype=F64).clamp(-2, 2)
    noise = .01 * torch.randn(2, *shape, generator=gen, device="cuda", dtype=F64)
    f, m = _sum(b, amp), _sum(b, amp, shift)
    top = f.max()
    return (f / top + noise[0]).contiguous(), (m / top + noise[1]).contiguous()


def _smooth(c, gen, peak):
    """A smooth displacement of six Gaussian vector bumps (peak in voxels), zero on the faces."""
    shape = (c["nz"], c["ny"], c["nx"])
    w = max(4., min(shape) / 10)
    b = _bumps(shape, gen, 6, (w, 2 * w))
    amp = peak * torch.randn(3, 6, generator=gen, device="cuda", dtype=F64).clamp(-1, 1)
    h = _grid(c).spacing
    u = torch.stack([_sum(b, amp[r]) * h[r] for r in range(3)], -1)
    win = 1.
    for a, n in enumerate(shape):
        k = torch.arange(n, device="cuda", dtype=F64)
        p = torch.clamp(torch.minimum(k, n - 1 - k) / 6., 0., 1.)
        win = win * p.reshape([-1 if j == a else 1 for j in range(3)])
    return u * win[..., None]


def _compressed(c, gen, floor):
    """A feasible displacement with a region of cells compressed along x to J near `floor` (times 1 +- 0.15): the x
    map sums positive cell increments per line; y and z move smoothly where x moves alone, so J stays a product."""
    nz, ny, nx = shape = (c["nz"], c["ny"], c["nx"])
    h = _grid(c).spacing
    w = max(3., min(shape) / 8)
    region = _sum(_bumps(shape, gen, 8, (w, 2 * w)), torch.ones(8, device="cuda", dtype=F64))[:, :, 1:]
    x = torch.arange(nx - 1, device="cuda", dtype=F64) / (nx - 2)
    waves = torch.sigmoid(12. * (torch.sin(2 * math.pi * x * max(2., nx / 24.)) - .55))      # thin slabs across x
    ends = [torch.clamp(torch.minimum(k, n - 1 - k) / 4., 0., 1.) for n in (nz, ny)
            for k in [torch.arange(n, device="cuda", dtype=F64)]]
    k = torch.arange(nx - 1, device="cuda", dtype=F64)
    inner = torch.clamp((torch.minimum(k, nx - 2 - k) - 6.) / 2., 0., 1.)                    # where y and z move freely
    m = torch.clamp(region, 0., 1.) * waves * inner * ends[0][:, None, None] * ends[1][None, :, None]
    inc = 1. - (1. - floor) * m
    inc = inc * ((nx - 1) / inc.sum(2, keepdim=True))
    u = torch.zeros(shape + (3,), device="cuda", dtype=F64)
    u[:, :, 1:, 0] = (torch.cumsum(inc, 2) - torch.arange(1, nx, device="cuda", dtype=F64)) * h[0]
    s = _smooth(c, gen, .5)
    win = torch.clamp(torch.minimum(torch.arange(nx, device="cuda"), nx - 1 - torch.arange(nx, device="cuda")) / 6., 0., 1.)
    u[..., 1] = s[:, :, nx // 2, 1][:, :, None] * win
    u[..., 2] = (s[:, ny // 2, nx // 2, 2][:, None, None] * win
                 * torch.clamp(torch.minimum(torch.arange(ny, device="cuda"), ny - 1 - torch.arange(ny, device="cuda")) / 6., 0., 1.)[None, :, None])
    u[[0, -1]] = 0.
    u[:, [0, -1]] = 0.
    u[:, :, [0, -1]] = 0.
    return u


def _rough(c, gen):
    """A feasible field with voxel-scale roughness, as late in a solve: about a third of the cells need more than the
    edge-hull proof.  Roughness is halved around the cells that it nearly folds."""
    smooth = _compressed(c, gen, .9) + _smooth(c, gen, .25)
    h = _grid(c).spacing
    noise = ((torch.rand(smooth.shape, generator=gen, device="cuda", dtype=F64) - .5) * .58
             * torch.tensor(h, device="cuda", dtype=F64))
    noise[[0, -1]] = 0.
    noise[:, [0, -1]] = 0.
    noise[:, :, [0, -1]] = 0.
    closed = [(i / 2, j / 2, k / 2) for k in range(3) for j in range(3) for i in range(3)]
    for _ in range(3):
        v = _vertices(smooth + noise)
        low = None
        for p in closed:
            J = _det(_deformation(v, h, p))
            low = J if low is None else torch.minimum(low, J)
        damp = torch.nn.functional.max_pool3d((low < .02).to(F64)[None, None], 2, 1, 1)[0, 0]
        noise = noise * (1. - .5 * damp)[..., None]
    return (smooth + noise).contiguous()


def _state(c, seed):
    """The images and three states of a running solve: the proximal reference, the base and a trial."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    fixed, moving = _images(c, gen)
    base = _compressed(c, gen, .03)
    ref = base - _smooth(c, gen, .006)
    trial = base + _smooth(c, gen, .004)
    return gen, fixed, moving, ref.contiguous(), base.contiguous(), trial.contiguous()


def prepare(case, seed):
    c, grid = case, _grid(case)
    kind = c["kind"]
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    if kind == "certify":
        return dict(kind=kind, grid=grid, u=_rough(c, gen))
    if kind == "solve":
        fixed, moving = _images(c, gen)
        return dict(kind=kind, grid=grid, case=c, fixed=fixed, moving=moving,
                    reg=solver.Registration(grid, fixed, moving, **_weights(c), precision=c["form"]))
    if kind == "register":
        fixed, moving = (t.cpu().pin_memory() for t in _images(c, gen))
        return dict(kind=kind, grid=grid, case=c, fixed=fixed, moving=moving)
    gen, fixed, moving, ref, base, trial = _state(c, seed)
    if kind == "metric":
        reg = solver.Registration(grid, fixed, moving, **_weights(c), u_ref=ref, precision=c["form"])
        s = reg.prepare_base(reg.pair.restrict(base))
        s.active = reg.pair.trial_energy(s.u, s.warped, s.u)[5]
        return dict(kind=kind, reg=reg, base=s, config=solver.PGConfig3D())
    pair = DevicePair(grid, fixed, moving, ref, **_weights(c), activation=ACTIVATION, precision=c["form"])
    s = dict(kind=kind, pair=pair)
    if kind == "direction":
        n = 3 * grid.n_free_scalar
        s.update(a=_weights(c)["lam"] + .02, b=.03,
                 rhs=torch.randn(n, generator=gen, device="cuda", dtype=F64),
                 scale=.5 + torch.rand(n, generator=gen, device="cuda", dtype=F64))
        return s
    warped, grad = pair.warp(base, with_gradient=True)
    active = pair.trial_energy(trial, warped, base)[5]
    s.update(base=base, trial=trial, warped=warped, grad=grad, active=active)
    return s


# ------------------------------------------------------------------------------------------------------- the pass
def _record(r):
    num = lambda v: float("nan") if v is None else float(v)
    return dict(status=certificate.STATUS.index(r.status), reason=certificate.REASONS.index(r.reason),
                checked=r.n_cells_checked, uncertain=r.n_uncertain, infeasible=r.n_infeasible, boxes=r.n_boxes,
                depth=r.max_depth, fast=r.n_fast_cells, prescreened=r.n_prescreen_cells, fallback=r.n_fallback_cells,
                min_jd=num(r.min_jd_lower_bound), min_margin=num(r.min_margin_lower_bound),
                sampled=num(r.sampled_min_jd))


def _result(res):
    return dict(u=res.final_state.u, warped=res.final_state.warped, native_mse=res.native_mse,
                final_mse=res.final_mse, gf=res.GF_final, accepted=res.counts["outer_accepted"],
                trials=res.counts["trials"])


def run(state):
    s, kind = state, state["kind"]
    if kind == "certify":
        return _record(certificate.certify_map(s["u"], s["grid"], config=certificate.NATIVE_CERTIFICATE,
                                               with_hash=False))
    if kind == "trial":
        w, g, terms, bad, diff, act = s["pair"].trial_energy(s["base"], s["warped"], s["trial"],
                                                             base_active=s["active"])
        return dict(warped=w, image_grad=g, terms=terms, bad=bad, dE=diff[0], dF=diff[1], active=act)
    if kind == "gradient":
        return dict(g=s["pair"].gradient(s["base"], s["warped"], s["grad"], active=s["active"]))
    if kind == "outer":
        gF, gD, gE = s["pair"].outer_gradients(s["base"], s["warped"], s["grad"], s["active"])
        return dict(gF=gF, gD=gD, gE=gE)
    if kind == "direction":
        return dict(p=s["pair"].poisson_apply(s["a"], s["b"], s["rhs"], scale=s["scale"], sign=-1.))
    if kind == "metric":
        a, b, scale = s["reg"].metric(s["base"], s["config"])
        return dict(a=a, b=b, scale=scale)
    outer = solver.SequentialConfig3D(max_iterations=s["case"]["steps"])
    if kind == "solve":
        # a registration object is one problem: its proximal reference is where the solve starts
        s["reg"].pair.set_reference(torch.zeros(s["grid"].shape + (3,), dtype=F64, device="cuda"))
        return _result(solver.solve_sequential(s["reg"], config=outer))
    res, _ = preopt.register_pair(s["fixed"], s["moving"], s["grid"], _weights(s["case"]), outer=s["case"]["steps"],
                                  precision=s["case"]["form"])
    return _result(res)


# ------------------------------------------------------------------------------------------------------- the work
def work(case):
    """Bytes: each input read and each output written once.  Flops: what the mathematics needs at least: J of one
    field at 27 points of a cell about 500, a cofactor pass about 900, a 4x4x4 spline sample with its gradient
    about 350, a folded transform n per entry and axis."""
    nz, ny, nx = case["nz"], case["ny"], case["nx"]
    nodes, cells = nz * ny * nx, (nz - 1) * (ny - 1) * (nx - 1)
    free = 3 * (nz - 2) * (ny - 2) * (nx - 2)
    trial = (24 * 4 + 8 * 3 + 24) * nodes + 2 * cells, 350 * nodes + 2000 * cells
    cert = 24 * nodes, 600 * cells
    grad = (24 * 3 + 8 * 2) * nodes + 8 * free, 2400 * cells
    outer = grad[0] + 16 * free, grad[1] + 900 * cells
    poisson = 24 * free, 2. * (nz + ny + nx) * free
    metric = 48 * nodes + 8 * free, 4000 * cells
    step = [sum(v) for v in zip(trial, cert, grad, poisson)]
    per_outer = [5 * step[k] + outer[k] + metric[k] for k in (0, 1)]
    b, f = {"certify": cert, "trial": trial, "gradient": grad, "outer": outer, "direction": poisson,
            "metric": metric}.get(case["kind"], [max(1, case["steps"]) * v for v in per_outer])
    if case["kind"] == "register":      # the finest pyramid level alone: 60 float32 iterations
        b, f = b + 60 * 60 * nodes, f + 60 * 400 * nodes
    return dict(bytes=float(b), flops=float(f))


# ------------------------------------------------------------------------------------------------------- 64 bits
def _spline(axis_nodes):
    """(knots, inverse collocation matrix) of the not-a-knot cubic spline on uniform nodes 0 .. n-1."""
    n = axis_nodes
    t = torch.cat([torch.zeros(4, dtype=F64), torch.arange(2, n - 2, dtype=F64), torch.full((4,), n - 1., dtype=F64)])
    x = torch.arange(n, dtype=F64)
    s, B, _ = _basis(t.cuda(), n, x.cuda())
    A = torch.zeros(n, n, dtype=F64, device="cuda")
    A.scatter_add_(1, (s - 3)[:, None] + torch.arange(4, device="cuda"), B)
    return t.cuda(), A


def _basis(t, n, x):
    """Span, values and derivatives of the four cubic B-splines at x (Cox-de Boor)."""
    s = torch.clamp(torch.searchsorted(t, x, right=True) - 1, 3, n - 1)
    b = [torch.ones_like(x)]
    for d in range(1, 4):
        nb, saved = [], torch.zeros_like(x)
        for r in range(d):
            right, left = t[s + r + 1], t[s + 1 - d + r]
            temp = b[r] / (right - left)
            nb.append(saved + (right - x) * temp)
            saved = (x - left) * temp
        nb.append(saved)
        if d == 3:
            q = b
        b = nb
    dB, zero = [], torch.zeros_like(x)
    for k in range(4):
        i = s - 3 + k
        lo, hi = t[i + 3] - t[i], t[i + 4] - t[i + 1]
        left = 3 * q[k - 1] / torch.where(lo == 0, 1., lo) if k else zero
        right = 3 * q[k] / torch.where(hi == 0, 1., hi) if k < 3 else zero
        dB.append(left - right)
    return s, torch.stack(b, -1), torch.stack(dB, -1)


def _warp64(c, image, u):
    """Value and xyz gradient of the image's not-a-knot cubic spline at X + u."""
    shape, h = (c["nz"], c["ny"], c["nx"]), _grid(c).spacing
    coef, per = image, []
    for a, n in enumerate(shape):
        t, A = _spline(n)
        coef = torch.linalg.solve(A, coef.movedim(a, 0).reshape(n, -1)).reshape(coef.movedim(a, 0).shape).movedim(0, a)
        k = torch.arange(n, device="cuda", dtype=F64).reshape([-1 if j == a else 1 for j in range(3)])
        per.append(_basis(t, n, (k + u[..., 2 - a] / h[2 - a]).reshape(-1)))
    (sz, bz, dz), (sy, by, dy), (sx, bx, dx) = per
    coef = coef.reshape(-1)
    val, g = 0., [0., 0., 0.]
    for i in range(4):
        for j in range(4):
            for k in range(4):
                v = coef[((sz - 3 + i) * shape[1] + sy - 3 + j) * shape[2] + sx - 3 + k]
                val = val + v * bz[:, i] * by[:, j] * bx[:, k]
                g[0] = g[0] + v * bz[:, i] * by[:, j] * dx[:, k] / h[0]
                g[1] = g[1] + v * bz[:, i] * dy[:, j] * bx[:, k] / h[1]
                g[2] = g[2] + v * dz[:, i] * by[:, j] * bx[:, k] / h[2]
    return val.reshape(shape), torch.stack(g, -1).reshape(shape + (3,))


def _node_weights(c):
    w = float(np.prod(_grid(c).spacing))
    for a, n in enumerate((c["nz"], c["ny"], c["nx"])):
        p = torch.ones(n, device="cuda", dtype=F64)
        p[0] = p[-1] = .5
        w = w * p.reshape([-1 if j == a else 1 for j in range(3)])
    return w


def _vertices(u):
    sl = (slice(None, -1), slice(1, None))
    return [u[sl[(a >> 2) & 1], sl[(a >> 1) & 1], sl[a & 1]] for a in range(8)]


def _deformation(v, h, p):
    """I + grad u at the cell point p (x, y, z in [0, 1]) of every cell, as F[r][j]."""
    F = [[0., 0., 0.] for _ in range(3)]
    for a in range(8):
        bit = (a & 1, (a >> 1) & 1, (a >> 2) & 1)
        f = [p[j] if bit[j] else 1 - p[j] for j in range(3)]
        for j in range(3):
            d = (1. if bit[j] else -1.) / h[j] * f[(j + 1) % 3] * f[(j + 2) % 3]
            if d:
                for r in range(3):
                    F[r][j] = F[r][j] + d * v[a][..., r]
    for r in range(3):
        F[r][r] = F[r][r] + 1.
    return F


def _det(F):
    return (F[0][0] * (F[1][1] * F[2][2] - F[1][2] * F[2][1]) + F[0][1] * (F[1][2] * F[2][0] - F[1][0] * F[2][2])
            + F[0][2] * (F[1][0] * F[2][1] - F[1][1] * F[2][0]))


def _curl(F):
    return F[2][1] - F[1][2], F[0][2] - F[2][0], F[1][0] - F[0][1]


def _points(c):
    """The Gauss points with their weights, and the closed points with theirs."""
    r, omega = math.sqrt(15.) / 10, float(np.prod(_grid(c).spacing))
    x, w = (.5 - r, .5, .5 + r), (5 / 18, 4 / 9, 5 / 18)
    three = range(3)
    gauss = [((x[i], x[j], x[k]), omega * w[i] * w[j] * w[k]) for k in three for j in three for i in three]
    closed = [((i / 2, j / 2, k / 2), omega / 27) for k in three for j in three for i in three]
    return gauss, closed


def _psi(J):
    """The localized barrier -r^2 log t below the activation (delta 0), zero above."""
    t = torch.clamp(J / ACTIVATION, max=1.)
    return -(1 - t) ** 2 * torch.log(t)


def _exact_trial(c, seed):
    _, fixed, moving, ref, base, trial = _state(c, seed)
    W, h, q = _weights(c), _grid(c).spacing, _node_weights(c)
    wa, _ = _warp64(c, moving, base)
    wb, gb = _warp64(c, moving, trial)
    img = .5 * (q * (wb - fixed) ** 2).sum()
    prox = .5 * W["lam"] * (q[..., None] * (trial - ref) ** 2).sum()
    dF = .5 * (q * (wb - wa) * (wb + wa - 2 * fixed)).sum()
    dE = .5 * W["lam"] * (q[..., None] * (trial - base) * (trial + base - 2 * ref)).sum()
    gauss, closed = _points(c)
    va, vb, vr = _vertices(base), _vertices(trial), _vertices(ref)
    jd = curl = bar = dB = 0.
    for p, w in gauss:
        Fa, Fb, Fr = (_deformation(v, h, p) for v in (va, vb, vr))
        Ja, Jb, Jr = _det(Fa), _det(Fb), _det(Fr)
        jd = jd + .5 * W["mu"] * w * ((Jb - Jr) ** 2).sum()
        dE = dE + .5 * W["mu"] * w * ((Jb - Ja) * (Jb + Ja - 2 * Jr)).sum()
        for a, b, r in zip(_curl(Fa), _curl(Fb), _curl(Fr)):
            curl = curl + .5 * W["nu"] * w * ((b - r) ** 2).sum()
            dE = dE + .5 * W["nu"] * w * ((b - a) * (b + a - 2 * r)).sum()
    for p, w in closed:
        Ja, Jb = _det(_deformation(va, h, p)), _det(_deformation(vb, h, p))
        bar = bar + W["kappa"] * w * _psi(Jb).sum()
        dB = dB + W["kappa"] * w * (_psi(Jb) - _psi(Ja)).sum()
    num = lambda v: float(v)
    return dict(warped=wb, image_grad=gb, terms=np.array([num(v) for v in (img, prox, jd, curl, bar)]), bad=None,
                dE=num(dE + dF + dB), dF=num(dF + dB), active=None)


def _exact_gradients(c, seed):
    """(image, proximity, JD + curl, barrier) gradients at the free nodes, component-major."""
    _, fixed, moving, ref, base, _ = _state(c, seed)
    W, h, q = _weights(c), _grid(c).spacing, _node_weights(c)
    w, g = _warp64(c, moving, base)
    vr = _vertices(ref)
    soft, bar = torch.zeros_like(base), torch.zeros_like(base)
    gauss, closed = _points(c)
    for points, out in ((gauss, soft), (closed, bar)):
        for p, wt in points:
            u = base.clone().requires_grad_(True)
            F = _deformation(_vertices(u), h, p)
            if out is soft:
                Fr = _deformation(vr, h, p)
                e = .5 * W["mu"] * wt * ((_det(F) - _det(Fr)) ** 2).sum()
                for a, r in zip(_curl(F), _curl(Fr)):
                    e = e + .5 * W["nu"] * wt * ((a - r) ** 2).sum()
            else:
                e = W["kappa"] * wt * _psi(_det(F)).sum()
            out += torch.autograd.grad(e, u)[0]
    free = lambda v: v[1:-1, 1:-1, 1:-1].movedim(-1, 0).reshape(-1)
    image = q[..., None] * (w - fixed)[..., None] * g
    return [free(v) for v in (image, W["lam"] * q[..., None] * (base - ref), soft, bar)]


def _exact_direction(c, seed):
    gen = _state(c, seed)[0]
    shape, h = (c["nz"] - 2, c["ny"] - 2, c["nx"] - 2), _grid(c).spacing
    n = 3 * math.prod(shape)
    rhs = torch.randn(n, generator=gen, device="cuda", dtype=F64)
    scale = .5 + torch.rand(n, generator=gen, device="cuda", dtype=F64)
    v, lam, mass = (scale * rhs).reshape((3,) + shape), [], []
    sines = []
    for a, m in enumerate(shape):
        k = torch.arange(1, m + 1, device="cuda", dtype=F64)
        sines.append(math.sqrt(2 / (m + 1)) * torch.sin(math.pi / (m + 1) * ((k[:, None] * k) % (2 * (m + 1)))))
        th = (math.pi * k / (m + 1)).reshape([-1 if j == a else 1 for j in range(3)])
        lam.append((2 * torch.sin(th / 2) / h[2 - a]) ** 2)
        mass.append((2 + torch.cos(th)) / 3)
    spectrum = lam[0] * mass[1] * mass[2] + mass[0] * lam[1] * mass[2] + mass[0] * mass[1] * lam[2]
    den = math.prod(h) * (_weights(c)["lam"] + .02 + .03 * spectrum)
    for sweep in range(2):
        for a in range(3):
            v = torch.movedim(torch.tensordot(sines[a], v, dims=([1], [a + 1])), 0, a + 1)
        if not sweep:
            v = v / den
    return dict(p=-scale * v.reshape(-1))


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "trial":
        return _exact_trial(c, seed)
    if kind in ("gradient", "outer"):
        image, prox, soft, bar = _exact_gradients(c, seed)
        if kind == "gradient":
            return dict(g=image + prox + soft + bar)
        return dict(gF=image + bar, gD=image, gE=image + prox + soft + bar)
    if kind == "direction":
        return _exact_direction(c, seed)
    if kind == "metric":
        _, _, moving, _, base, _ = _state(c, seed)
        _, g = _warp64(c, moving, base)
        W = _weights(c)
        return dict(a=W["lam"] + float((g[1:-1, 1:-1, 1:-1] ** 2).sum(-1).mean()) / 3, b=(W["mu"] + W["nu"]) / 2,
                    scale=None)
    return None
