"""The work that programs built on this package give it, as timed cases.

Each case is one pass through the public entry points (``Solver``, ``numerics_pc``, ``physics``,
``gcbc_go``, ``Ensemble``, ``Adjoint``): line solves, time steps of one box, time steps through the
reference-shaped call sequence, time steps of many boxes, and gradients.  ``listed`` names the
standing cases, ``draw`` gives further ones of the same ranges, ``prepare`` / ``run`` make and run a
case, ``work`` and ``tolerance`` say what a pass must move and how exactly two correct runs agree,
and ``exact`` is the same mathematics in plain FP64 torch with dense line operators, independent of
the package.
"""
import math
from fractions import Fraction

import torch

import compact_schemes_b200 as cs

GAM, PRANDTL = 1.4, 0.71
TWO_PI = 2.0 * math.pi
PERIODIC, NONREFLECTIVE, WALL = cs.BC_PERIODIC, cs.BC_NON_REFLECTIVE, cs.BC_WALL_VISCOUS

# One box's options, with their usual values.  kind: "lines" (derivative, and filter, of one field
# along x, y, z), "step" (one RK step of one box), "dropin" (the same step through the reference's
# call sequence), "ensemble" (one step of many boxes), "gradient" (d J / d q0 through checkpointed
# steps), "tangent" (one linearized step).
_DEFAULTS = {"f32": False, "open_x": False, "walls_y": False, "closed": False, "filter": False, "curved": False,
             "mixed": False, "tune": False, "viscous": True, "steps": 1, "every": 1, "boxes": 0, "box_seed": 0}


def _case(kind, lxi, let, lze, **opt):
    c = {"kind": kind, "lxi": lxi, "let": let, "lze": lze}
    c.update(_DEFAULTS)
    c.update(opt)
    return c


def listed():
    def named(name, *a, **k):
        return dict(_case(*a, **k), name=name)
    return [
        # the derivative-and-filter workload: one small field on a non-periodic grid, called line
        # family by line family, so that latency and launches count
        named("lines_64_closed", "lines", 64, 64, 64, closed=True, filter=True),
        # the derivative of one field of the headline box, as a user's own operators call it
        named("lines_256", "lines", 256, 256, 256),
        # single precision, lengths that fill neither chunks nor tiles
        named("lines_f32_ragged", "lines", 161, 130, 257, f32=True),
        # the reference driver's time step with per-point metrics, characteristic x faces and
        # viscous walls on y, on a small block: many short calls
        named("dropin_40_walls", "dropin", 40, 36, 33, open_x=True, walls_y=True),
        # the same call sequence on the headline box, periodic
        named("dropin_256", "dropin", 256, 256, 256),
        # the fused time step: a small box, where launches and latency count
        named("step_48", "step", 48, 48, 48),
        # the headline: 256^3 Taylor-Green, FP64
        named("step_256", "step", 256, 256, 256, tune=True),
        # odd sizes with every option of the FP64 step: curvilinear metrics, characteristic x faces,
        # filter after the step
        named("step_ragged_curved", "step", 150, 97, 131, open_x=True, filter=True, curved=True),
        # the mixed-precision step with characteristic x faces and 512-point lines
        named("mixed_512", "step", 512, 256, 256, open_x=True, mixed=True, tune=True),
        # 64 boxes with axes of 32 to 128 points advanced together
        named("ensemble_64", "ensemble", 0, 0, 0, boxes=64),
        # gradient of the kinetic energy on the 128^3 box, checkpointed every second step
        named("gradient_128", "gradient", 128, 128, 128, steps=4, every=2),
        # one linearized step (tangent) of an uneven box
        named("tangent_96", "tangent", 96, 80, 112),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["lines", "lines", "step", "step", "mixed", "dropin", "dropin", "ensemble", "gradient", "tangent"])
    if kind == "ensemble":
        return _case("ensemble", 0, 0, 0, boxes=_log_int(rng, 2, 64), box_seed=rng.randrange(1000))
    # per kind: the largest box drawn, in points; the box's size is spread over its logarithm and its
    # axes are uneven around it
    most = {"lines": 256 ** 3, "step": 256 ** 3, "mixed": 256 ** 3, "dropin": 256 ** 3, "gradient": 128 ** 3,
            "tangent": 128 ** 3}[kind]
    longest = 512
    while True:
        side = math.exp(rng.uniform(math.log(24.0), math.log(most ** (1.0 / 3.0))))
        dims = [int(round(side * math.exp(rng.uniform(-0.45, 0.45)))) for _ in range(3)]
        if rng.random() < 0.5:  # half of the boxes have even, 8-point sizes, as most users choose
            dims = [8 * max(2, int(round(d / 8.0))) for d in dims]
        dims = [max(16, min(longest, d)) for d in dims]
        if dims[0] * dims[1] * dims[2] <= most:
            break
    big = dims[0] * dims[1] * dims[2] > 1000000
    if kind == "lines":
        f32 = rng.random() < 0.3
        closed = not f32 and rng.random() < 0.5
        return _case("lines", *dims, f32=f32, closed=closed, filter=not f32 and rng.random() < 0.5)
    if kind == "step":
        curved = rng.random() < 0.3
        return _case("step", *dims, open_x=rng.random() < 0.4, filter=rng.random() < 0.3, curved=curved,
                     viscous=rng.random() < 0.85, tune=big)
    if kind == "mixed":
        return _case("step", *dims, mixed=True, open_x=rng.random() < 0.4, tune=big)
    if kind == "dropin":
        return _case("dropin", *dims, open_x=rng.random() < 0.5, walls_y=rng.random() < 0.4, viscous=rng.random() < 0.85)
    if kind == "gradient":
        steps = rng.choice([2, 3, 4])
        return _case("gradient", *dims, steps=steps, every=rng.choice([1, 2]), open_x=rng.random() < 0.3)
    return _case("tangent", *dims, open_x=rng.random() < 0.3)


# --------------------------------------------------------------------------- inputs
def _dims(case):
    return case["lxi"], case["let"], case["lze"]


def _nbc(case):
    b = [PERIODIC] * 3
    if case["closed"]:
        b = [NONREFLECTIVE] * 3
    if case["open_x"]:
        b[0] = NONREFLECTIVE
    if case["walls_y"]:
        b[1] = WALL
    return [b, list(b)]


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _axes(dims):
    lxi, let, lze = dims
    ax = [torch.arange(n, dtype=torch.float64, device="cuda") * (TWO_PI / n) for n in dims]
    return ax[0].view(1, 1, lxi), ax[1].view(1, let, 1), ax[2].view(lze, 1, 1)


def _field(case, seed):
    """One smooth field with a little noise."""
    g = _generator(seed)
    x, y, z = _axes(_dims(case))
    ph = torch.rand(3, generator=g, device="cuda", dtype=torch.float64) * TWO_PI
    f = torch.sin(3 * x + ph[0]) * torch.cos(2 * y + ph[1]) + 0.5 * torch.sin(5 * z + ph[2])
    f = f + 1e-3 * torch.randn(f.shape, generator=g, device="cuda", dtype=torch.float64)
    return (f.float() if case["f32"] else f).reshape(-1).contiguous()


def _flow(dims, mach, seed):
    """Taylor-Green state in the package's units, with a seeded large-scale perturbation and noise: [5 * points]."""
    g = _generator(seed)
    x, y, z = _axes(dims)
    ph = torch.rand(3, generator=g, device="cuda", dtype=torch.float64) * TWO_PI
    u = mach * (torch.sin(x) * torch.cos(y) * torch.cos(z) + 0.05 * torch.sin(2 * y + ph[0]))
    v = mach * (-torch.cos(x) * torch.sin(y) * torch.cos(z) + 0.05 * torch.sin(2 * z + ph[1]))
    w = mach * 0.1 * torch.sin(x + ph[2]) * torch.cos(y) + 0.0 * z
    p = 1.0 / GAM + mach * mach / 16.0 * (torch.cos(2 * x) + torch.cos(2 * y)) * (torch.cos(2 * z) + 2.0)
    rho = 1.0 + 1e-4 * (2.0 * torch.rand(p.shape, generator=g, device="cuda", dtype=torch.float64) - 1.0)
    e = p / (GAM - 1.0) + 0.5 * rho * (u * u + v * v + w * w)
    return torch.stack([rho, rho * u, rho * v, rho * w, e]).reshape(-1).contiguous()


def _metrics(case):
    """Metrics [3][points] x 3 and Jacobian of the wavy grid x = xi + A sin(eta) sin(zeta) (and cyclic)."""
    dims = _dims(case)
    h = [TWO_PI / n for n in dims]
    x, y, z = _axes(dims)
    one = torch.ones(dims[2], dims[1], dims[0], dtype=torch.float64, device="cuda")
    A = 0.1
    r = [[h[0] * one, h[0] * A * torch.sin(z) * torch.cos(x) * one, h[0] * A * torch.cos(x) * torch.sin(y) * one],
         [h[1] * A * torch.cos(y) * torch.sin(z) * one, h[1] * one, h[1] * A * torch.sin(x) * torch.cos(y) * one],
         [h[2] * A * torch.sin(y) * torch.cos(z) * one, h[2] * A * torch.cos(z) * torch.sin(x) * one, h[2] * one]]

    def cross(a, b):
        return [a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]]
    m = [cross(r[1], r[2]), cross(r[2], r[0]), cross(r[0], r[1])]
    yaco = 1.0 / (r[0][0] * m[0][0] + r[0][1] * m[0][1] + r[0][2] * m[0][2])
    return [torch.stack(a).reshape(-1).contiguous() for a in m] + [yaco.reshape(-1).contiguous()]


_MACH, _RE, _CFL, _ALPHA = 0.1, 1600.0, 0.5, 0.45
_UMF = (0.01, -0.02, 0.005)  # frame velocity of the call-sequence cases
_ACC = (0.002, 0.001, -0.001)


def _dt(dims, mach=_MACH, cfl=0.4):
    """A stable time step of the uniform box (the gradient and tangent cases hold dt fixed)."""
    return cfl / ((1.0 + mach) * sum(n / TWO_PI for n in dims))


def _config(case):
    return cs.tgv_config(None, mach=_MACH, re=_RE, cfl=_CFL, dims=_dims(case), nbc=_nbc(case), gcbc=case["open_x"],
                         viscous=case["viscous"], precision=cs.solver.PREC_MIXED_F32 if case["mixed"] else 0,
                         filter=cs.solver.FILTER_STEP if case["filter"] else 0, alpha_f=_ALPHA)


def _boxes(case):
    return cs.draw_boxes(case["boxes"], case["box_seed"])


def _sbcc(case, yaco):
    """1/J on the characteristic and wall face planes, 0 elsewhere."""
    lxi, let, lze = _dims(case)
    s = torch.zeros(lze, let, lxi, dtype=torch.float64, device="cuda")
    inv = (1.0 / yaco).view(lze, let, lxi)
    if case["open_x"]:
        s[:, :, 0], s[:, :, -1] = inv[:, :, 0], inv[:, :, -1]
    if case["walls_y"]:
        s[:, 0], s[:, -1] = inv[:, 0], inv[:, -1]
    return s.reshape(-1).contiguous()


def _normals(case, met):
    """Unit face normals per axis [2][3][F], face index along the axis' line families."""
    lxi, let, lze = _dims(case)
    out = []
    for a in range(3):
        m = met[a].view(3, lze, let, lxi)
        f = [m[:, :, :, i].reshape(3, -1) if a == 0 else (m[:, :, i].reshape(3, -1) if a == 1 else m[:, i].reshape(3, -1))
             for i in (0, -1)]
        out.append(torch.stack([v / v.norm(dim=0) for v in f]).reshape(-1).contiguous())
    return out


def prepare(case, seed):
    dims, kind = _dims(case), case["kind"]
    n = dims[0] * dims[1] * dims[2]
    st = {"case": case, "dims": dims}
    new = lambda k, dt=torch.float64: torch.empty(k, dtype=dt, device="cuda")  # noqa: E731
    if kind == "lines":
        f = _field(case, seed)
        nm = cs.numerics_pc(dims, _nbc(case))
        nm.deriv_setup()
        st.update(nm=nm, f=f, out=[torch.empty_like(f) for _ in range(6 if case["filter"] else 3)])
        return st
    if kind == "ensemble":
        boxes = _boxes(case)
        ens = cs.Ensemble(cs.ensemble_tgv(boxes, cfl=_CFL))
        q0 = torch.zeros(ens.state_size(), dtype=torch.float64, device="cuda")
        for b, (d, mach, _) in enumerate(boxes):
            ens.box_view(q0, b).copy_(_flow(d, mach, seed * 1000 + b))
        st.update(ens=ens, q0=q0, q=torch.empty_like(q0), nb=len(boxes))
        return st
    q0 = _flow(dims, _MACH, seed)
    st.update(q0=q0)
    if kind == "step":
        s = cs.Solver(_config(case))
        if case["curved"]:
            s.set_metrics(*_metrics(case))
        if case["tune"]:
            s.autotune(q0, 2)
        st.update(s=s, q=torch.empty_like(q0))
    elif kind == "dropin":
        met = _metrics(case)
        nm = cs.numerics_pc(dims, _nbc(case))
        nm.deriv_setup()
        ph = cs.physics(dims, case["viscous"])
        ph.umf = _UMF
        npex = torch.ones(dims[2], dims[1], dims[0], dtype=torch.int32, device="cuda")
        npex[:, 0], npex[:, -1] = 0, 0
        faces = [dims[1] * dims[2], dims[0] * dims[2], dims[0] * dims[1]]
        st.update(nm=nm, ph=ph, met=met, ssk=torch.full((n,), _MACH / _RE, dtype=torch.float64, device="cuda"),
                  sbcc=_sbcc(case, met[3]), cm=_normals(case, met), npex=npex.reshape(-1), de=new(5 * n), p=new(n),
                  drva=[nm.buffers(a)[0] for a in range(3)], drvb=[torch.zeros(10 * F, dtype=torch.float64, device="cuda") for F in faces],
                  qa=new(5 * n))
    elif kind == "gradient":
        st.update(adj=cs.Adjoint(_config(case)), dts=[_dt(dims)] * case["steps"], g=torch.empty_like(q0))
    else:
        st.update(adj=cs.Adjoint(_config(case)), dt=_dt(dims), stages=[torch.empty_like(q0) for _ in range(4)],
                  dq=_flow(dims, _MACH, seed + 77) - q0, out=torch.empty_like(q0))
        st["adj"].stages(q0, st["dt"], st["stages"])
    return st


def run(st):
    case, dims, kind = st["case"], st["dims"], st["case"]["kind"]
    if kind == "lines":
        nm, f, out = st["nm"], st["f"], st["out"]
        for a in range(3):
            nm.deriv1d(a, f, out[a], nm.ndf[0][a], nm.ndf[1][a], nm.dcomp, 0, halo=cs.HALO_SELF)
        if case["filter"]:
            src = f
            for a in range(3):
                nm.filter(a, src, out[3 + a], _ALPHA, nm.dcomp)
                src = out[3 + a]
        return out
    if kind == "step":
        st["q"].copy_(st["q0"])  # restart from the saved state, then one step in place
        st["s"].step(st["q"])
        return st["q"]
    if kind == "ensemble":
        st["q"].copy_(st["q0"])
        st["ens"].step(st["q"])
        return [st["ens"].box_view(st["q"], b) for b in range(st["nb"])]
    if kind == "gradient":
        J = st["adj"].gradient(st["q0"], st["dts"], case["every"], st["g"])
        return {"J": J, "grad": st["g"]}
    if kind == "tangent":
        st["adj"].step_jvp(st["stages"], st["dt"], st["dq"], st["out"])
        return st["out"]
    # the reference driver's loop over the four stages of a step
    nm, ph, (X, E, Z, Y), qn, qa, de, p = st["nm"], st["ph"], st["met"], st["q0"], st["qa"], st["de"], st["p"]
    nbc = _nbc(case)
    n = Y.numel()
    qa.copy_(qn)
    for k in range(4):
        cs.thermo(qa, de, p)
        if k == 0:
            dt = ph.calc_time_step(X, E, Z, de, Y, st["ssk"], _CFL, n)
        if case["viscous"]:
            ph.calc_viscous_shear_stress(de, st["ssk"], X, E, Z, Y, nm.dcomp, None, nm)
            cs.thermo(qa, de, p)
        ph.calc_fluxes(qa, p, de, X, E, Z, nm.dcomp, None, nm)
        if case["open_x"] or case["walls_y"]:
            cs.gcbc_go(st["drva"], st["cm"], st["drvb"], qa, de, p, Y, st["sbcc"], _UMF, _ACC, nm.dcomp, 1.0 / dt, nbc)
        cs.rk_update(qn, de, Y, dt / (4 - k), qa)
        if case["walls_y"]:
            cs.wall_condition_update(qa, st["npex"], dims, nbc, _UMF)
    return {"dt": dt, "q": qa, "rhs": de}


# --------------------------------------------------------------------------- work and tolerance
def work(case):
    kind = case["kind"]
    lxi, let, lze = _dims(case)
    n = lxi * let * lze
    solve = 12.0  # operations per row of one line solve with its right-hand side
    stage = (27 * solve + 3 * 90 + 60) if case["viscous"] else (15 * solve + 3 * 35 + 20)
    if kind == "lines":
        b = 4 if case["f32"] else 8
        outs = 6 if case["filter"] else 3
        return {"bytes": n * b * (1 + outs), "flops": n * outs * (solve + 6)}
    if kind == "ensemble":
        n = sum(math.prod(d) for d, _, _ in _boxes(case))
        return {"bytes": 80 * n, "flops": 4 * stage * n}
    if kind == "step":
        return {"bytes": n * (80 + (80 if case["curved"] else 0)), "flops": n * (4 * stage + (90 * 3 if case["filter"] else 0))}
    if kind == "dropin":  # state, metrics, Jacobian and viscosity in; state and right-hand side out
        return {"bytes": n * 8 * (5 + 9 + 1 + 1 + 5 + 5), "flops": 4 * n * (stage + 250)}
    if kind == "gradient":
        k = case["steps"]
        return {"bytes": 80 * n, "flops": n * 4 * k * (2 * stage + 3 * stage)}
    return {"bytes": n * 8 * 5 * (4 + 2), "flops": n * 4 * 3 * stage}


def tolerance(case):
    # about four times the distance measured to `exact`: derivatives 2e-15 (FP32 2.6e-7), steps
    # 1.2e-15 with the filter, gradients 7e-16, the mixed step 1e-9 of the state, and 1e-12 for a
    # right-hand side by itself (the boundary rows' weights cancel the fluxes' mean, which amplifies
    # rounding a few hundred times)
    if case["kind"] == "lines":
        return {"rel": 1e-6, "max": 1e-4} if case["f32"] else {"rel": 1e-14, "max": 1e-12}
    if case["mixed"]:
        return {"rel": 5e-9, "max": 5e-7}
    if case["kind"] == "dropin":
        return {"rel": 5e-12, "max": 5e-10}
    return {"rel": 1e-14, "max": 1e-12}


# --------------------------------------------------------------------------- the same in plain FP64
def _interface_weights():
    """Rows 8 and 9 of P~ P^-1 Q of the two-block 16-row system, in exact fractions, as (pbco, pbci) floats."""
    n = 16
    P = [[Fraction(0)] * n for _ in range(n)]
    Q = [[Fraction(0)] * n for _ in range(n)]
    al, a01, a10 = Fraction(1, 3), Fraction(2), Fraction(1, 4)
    aa, bb, b00, b01, b02, b10 = Fraction(7, 9), Fraction(1, 36), Fraction(-5, 2), Fraction(2), Fraction(1, 2), Fraction(3, 4)
    for i in range(n):
        P[i][i] = Fraction(1)
    P[0][1] = P[n - 1][n - 2] = a01
    P[1][0] = P[1][2] = P[n - 2][n - 1] = P[n - 2][n - 3] = a10
    Q[0][0], Q[0][1], Q[0][2], Q[1][0], Q[1][2] = b00, b01, b02, -b10, b10
    # the last row's weights in the scheme's own order (it only shapes the far, decayed end)
    Q[n - 1][n - 1], Q[n - 1][n - 2], Q[n - 1][n - 3] = -b02, -b01, -b00
    Q[n - 2][n - 1], Q[n - 2][n - 3] = b10, -b10
    for i in range(2, n - 2):
        P[i][i - 1] = P[i][i + 1] = al
        Q[i][i - 2], Q[i][i - 1], Q[i][i + 1], Q[i][i + 2] = -bb, -aa, aa, bb
    M = [P[i][:] + Q[i][:] for i in range(n)]
    for i in range(n):
        piv = next(r for r in range(i, n) if M[r][i] != 0)
        M[i], M[piv] = M[piv], M[i]
        f = M[i][i]
        M[i] = [v / f for v in M[i]]
        for r in range(n):
            if r != i and M[r][i] != 0:
                f = M[r][i]
                M[r] = [v - f * w for v, w in zip(M[r], M[i])]
    T = [row[n:] for row in M]  # P^-1 Q
    P[8][7] = P[8][6] = P[9][7] = Fraction(0)
    rows = [[sum(P[r][k] * T[k][c] for k in range(n)) for c in range(n)] for r in (8, 9)]
    pbco = [[float(r[7 - k]) for k in range(8)] for r in rows]
    pbci = [[float(r[8 + k]) for k in range(8)] for r in rows]
    return pbco, pbci


def _deriv_matrix(n, interface):
    A = torch.eye(n, dtype=torch.float64)
    B = torch.zeros(n, n, dtype=torch.float64)
    for i in range(n):
        for j in (i - 1, i + 1):
            if 0 <= j < n:
                A[i, j] = 1.0 / 3.0
    for i in range(2, n - 2):
        B[i, i - 2], B[i, i - 1], B[i, i + 1], B[i, i + 2] = -1.0 / 36.0, -7.0 / 9.0, 7.0 / 9.0, 1.0 / 36.0
    if interface:
        pbco, pbci = _interface_weights()
        for r in range(2):
            for k in range(8):
                B[r, k] += pbci[r][k]
                B[r, n - 1 - k] += pbco[r][k]
                B[n - 1 - r, n - 1 - k] -= pbci[r][k]
                B[n - 1 - r, k] -= pbco[r][k]
    else:
        A[0, 1] = A[n - 1, n - 2] = 2.0
        A[1, 0] = A[1, 2] = A[n - 2, n - 1] = A[n - 2, n - 3] = 0.25
        B[0, 0], B[0, 1], B[0, 2] = -2.5, 2.0, 0.5
        B[n - 1, n - 1], B[n - 1, n - 2], B[n - 1, n - 3] = 2.5, -2.0, -0.5
        B[1, 0], B[1, 2] = -0.75, 0.75
        B[n - 2, n - 1], B[n - 2, n - 3] = 0.75, -0.75
    return torch.linalg.solve(A, B).cuda()


def _filter_matrix(n, cyclic, af):
    a6 = [(11 + 10 * af) / 16, (15 + 34 * af) / 64, (-3 + 6 * af) / 32, (1 - 2 * af) / 64]
    a4 = [(5 + 6 * af) / 8, (1 + 2 * af) / 4, (-1 + 2 * af) / 16]
    a2 = [(1 + 2 * af) / 2, (1 + 2 * af) / 4]
    A = torch.eye(n, dtype=torch.float64)
    B = torch.zeros(n, n, dtype=torch.float64)
    for i in range(n):
        dist = n if cyclic else min(i, n - 1 - i)
        w = [1.0] if dist == 0 else (a2 if dist == 1 else (a4 if dist == 2 else a6))
        if dist > 0:
            A[i, (i - 1) % n] = A[i, (i + 1) % n] = af
        for m, c in enumerate(w):
            for j in ({i} if m == 0 else {(i - m) % n, (i + m) % n}):
                B[i, j] += c
    return torch.linalg.solve(A, B).cuda()


class _Operators:
    """Dense line operators of one box, applied to fields [..., lze, let, lxi]."""

    def __init__(self, dims, nbc, af=None):
        per = [nbc[0][a] == PERIODIC for a in range(3)]
        self.D = [_deriv_matrix(n, p) for n, p in zip(dims, per)]
        self.Fm = [_filter_matrix(n, p, af) for n, p in zip(dims, per)] if af is not None else None

    @staticmethod
    def along(M, axis, f):
        if axis == 0:
            return f @ M.T
        if axis == 1:
            return torch.matmul(M, f)
        s = f.shape
        return torch.matmul(M, f.reshape(s[:-3] + (s[-3], s[-2] * s[-1]))).reshape(s)

    def d(self, axis, f):
        return self.along(self.D[axis], axis, f)

    def filter(self, q):
        for a in range(3):
            q = self.along(self.Fm[a], a, q)
        return q


def _primitive(q):
    u = [q[1] / q[0], q[2] / q[0], q[3] / q[0]]
    p = (GAM - 1.0) * (q[4] - 0.5 * (q[1] * u[0] + q[2] * u[1] + q[3] * u[2]))
    return u, p, GAM * p / q[0]


def _char_matrix(c, u, a, hv2):
    """Columns of the characteristic-to-conservative transformation for unit normals c [3, F]: [F, 5, 5]."""
    S = torch.zeros(c[0].numel(), 5, 5, dtype=torch.float64, device="cuda")
    vn = c[0] * u[0] + c[1] * u[1] + c[2] * u[2]
    d = [a * c[0], a * c[1], a * c[2]]
    for k in range(3):
        k1, k2 = (k + 1) % 3, (k + 2) % 3
        S[:, 0, k] = c[k]
        S[:, 1 + k, k] = c[k] * u[k]
        S[:, 1 + k, k1] = c[k1] * u[k] - d[k2]
        S[:, 1 + k, k2] = c[k2] * u[k] + d[k1]
        S[:, 1 + k, 3], S[:, 1 + k, 4] = 0.5 * (u[k] + d[k]), 0.5 * (u[k] - d[k])
        S[:, 4, k] = hv2 * c[k] + d[k2] * u[k1] - d[k1] * u[k2]
    S[:, 0, 3] = S[:, 0, 4] = 0.5
    h = hv2 + a * a / (GAM - 1.0)
    S[:, 4, 3], S[:, 4, 4] = 0.5 * (h + a * vn), 0.5 * (h - a * vn)
    return S


def _characteristic(q, src, J, cm, ip, umf, wall=None):
    """Change of the right-hand side at face points from the characteristic closure: q, src, [5, F] (src the
    derivative terms), J [F], cm [3, F]; wall: None (non-reflective) or (frame acceleration, 1/dt)."""
    u, p, _ = _primitive(q)
    a = torch.sqrt(GAM * p / q[0])
    hv2 = 0.5 * (u[0] ** 2 + u[1] ** 2 + u[2] ** 2)
    S = _char_matrix(cm, u, a, hv2)
    cha = torch.linalg.solve(S, (J * src).T.unsqueeze(-1)).squeeze(-1)
    vn = sum(cm[k] * u[k] for k in range(3)) + sum(cm[k] * umf[k] for k in range(3))
    sgn = 1.0 - 2.0 * ip
    zero = torch.zeros_like(vn)
    if wall is None:
        d3 = torch.where(sgn * (vn + a) > 0, -cha[:, 3], zero)
        d4 = torch.where(sgn * (vn - a) > 0, -cha[:, 4], zero)
    else:
        acc, dtwi = wall
        w = 2.0 * sgn * q[0] / a * (sum(cm[k] * acc[k] for k in range(3)) + dtwi * vn)
        d3 = cha[:, 4] + w - cha[:, 3] if ip == 0 else zero
        d4 = cha[:, 3] + w - cha[:, 4] if ip == 1 else zero
    return (S[:, :, 3] * d3[:, None] + S[:, :, 4] * d4[:, None]).T


def _rhs(op, q, met, J, mu, umf, viscous, open_x):
    """Right-hand side [5, lze, let, lxi] of the state q; met[a][c] and J are fields or numbers."""
    u, p, T = _primitive(q)
    if viscous:
        prim = torch.stack([u[0], u[1], u[2], T])
        G = [op.d(a, prim) for a in range(3)]
        dx = [[sum(met[b][k] * G[b][c] for b in range(3) if not (isinstance(met[b][k], float) and met[b][k] == 0.0))
               for k in range(3)] for c in range(4)]
        del G
        muj = mu * J
        div = 2.0 / 3.0 * (dx[0][0] + dx[1][1] + dx[2][2])
        tau = [[None] * 3 for _ in range(3)]
        for i in range(3):
            for k in range(i, 3):
                t = muj * (2.0 * dx[i][i] - div) if i == k else muj * (dx[i][k] + dx[k][i])
                tau[i][k] = tau[k][i] = t
        kap = muj / ((GAM - 1.0) * PRANDTL)
        heat = [kap * dx[3][k] + u[0] * tau[0][k] + u[1] * tau[1][k] + u[2] * tau[2][k] for k in range(3)]
    out = None
    for a in range(3):
        ss = sum(met[a][k] * (u[k] + umf[k]) for k in range(3))
        fl = [q[0] * ss]
        for m in range(3):
            f = q[1 + m] * ss + met[a][m] * p
            if viscous:
                f = f - sum(met[a][k] * tau[m][k] for k in range(3))
            fl.append(f)
        f = (q[4] + p) * ss - p * sum(met[a][k] * umf[k] for k in range(3))
        if viscous:
            f = f - sum(met[a][k] * heat[k] for k in range(3))
        fl.append(f)
        d = op.d(a, torch.stack(fl))
        if a == 0 and open_x:
            add = torch.zeros_like(d)
            for ip, i in ((0, 0), (1, d.shape[-1] - 1)):
                field = torch.is_tensor(J)
                Jf = J[:, :, i].reshape(-1) if field else torch.full((d[0, :, :, i].numel(),), J, dtype=torch.float64, device="cuda")
                cm = [met[0][k][:, :, i].reshape(-1) if field else torch.full_like(Jf, met[0][k]) for k in range(3)]
                nrm = torch.sqrt(cm[0] ** 2 + cm[1] ** 2 + cm[2] ** 2)
                dq = _characteristic(q[..., i].reshape(5, -1), d[..., i].reshape(5, -1), Jf, [c / nrm for c in cm], ip, umf)
                sel = torch.zeros(d.shape[-1], dtype=torch.float64, device="cuda")
                sel[i] = 1.0
                add = add + (dq / Jf).reshape(5, d.shape[1], d.shape[2], 1) * sel
            d = d + add
        out = d if out is None else out + d
    return out


def _uniform(dims):
    h = [TWO_PI / n for n in dims]
    met = [[0.0] * 3 for _ in range(3)]
    met[0][0], met[1][1], met[2][2] = h[1] * h[2], h[0] * h[2], h[0] * h[1]
    return met, 1.0 / (h[0] * h[1] * h[2])


def _time_step(q, met, J, mu, umf, cfl):
    u, _, T = _primitive(q)
    r1 = sum(met[a][k] * met[a][k] for a in range(3) for k in range(3))
    r2 = sum((sum(met[a][k] * (u[k] + umf[k]) for k in range(3))).abs() for a in range(3))
    Ja = J.abs() if torch.is_tensor(J) else abs(J)
    m1 = ((torch.sqrt(T * r1) + r2) * Ja).max()
    m2 = (mu / q[0] * r1 * Ja * Ja).max()
    return float(torch.minimum(cfl / m1, 0.5 / m2))


def _exact_step(dims, q, nbc, met, J, mu, viscous, open_x, af):
    op = _Operators(dims, nbc, af)
    zero = (0.0, 0.0, 0.0)
    q0 = q.view(5, dims[2], dims[1], dims[0])
    dt = _time_step(q0, met, J, mu, zero, _CFL)
    cur = q0
    for k in range(4):
        cur = q0 - dt / (4 - k) * J * _rhs(op, cur, met, J, mu, zero, viscous, open_x)
    if af is not None:
        cur = op.filter(cur)
    return cur.reshape(-1)


def exact(case, seed):
    dims, kind = _dims(case), case["kind"]
    shape = (dims[2], dims[1], dims[0])
    mu = _MACH / _RE
    with torch.no_grad():
        if kind == "lines":
            op = _Operators(dims, _nbc(case), _ALPHA if case["filter"] else None)
            f = _field(case, seed).double().view(shape)
            out = [op.d(a, f).reshape(-1) for a in range(3)]
            if case["filter"]:
                for a in range(3):
                    f = op.along(op.Fm[a], a, f)
                    out.append(f.reshape(-1))
            return out
        if kind == "ensemble":
            out = []
            for b, (d, mach, re) in enumerate(_boxes(case)):
                met, J = _uniform(d)
                out.append(_exact_step(d, _flow(d, mach, seed * 1000 + b), [[PERIODIC] * 3] * 2, met, J, mach / re, True, False, None))
            return out
        q0 = _flow(dims, _MACH, seed)
        met, J = _uniform(dims)
        if kind == "dropin" or case["curved"]:
            arr = _metrics(case)
            met = [[arr[a].view((3,) + shape)[k] for k in range(3)] for a in range(3)]
            J = arr[3].view(shape)
        if kind == "step":
            return _exact_step(dims, q0, _nbc(case), met, J, mu, case["viscous"], case["open_x"], _ALPHA if case["filter"] else None)
        if kind == "dropin":
            return _exact_dropin(case, dims, q0, met, J, mu)
    op = _Operators(dims, _nbc(case))
    zero = (0.0, 0.0, 0.0)
    rhs = lambda q: _rhs(op, q, met, J, mu, zero, case["viscous"], case["open_x"])  # noqa: E731
    dt = _dt(dims)

    def stages(q):
        got = [q]
        with torch.no_grad():
            for k in range(4):
                got.append(q - dt / (4 - k) * J * rhs(got[-1]))
        return got
    q0 = q0.view((5,) + shape)
    if kind == "tangent":
        st = stages(q0)
        dq = (_flow(dims, _MACH, seed + 77) - q0.reshape(-1)).view_as(q0)
        cur = dq
        for k in range(4):
            cur = dq - dt / (4 - k) * J * _linear(rhs, st[k], cur)
        return cur.reshape(-1)
    starts = [q0]
    for _ in range(case["steps"]):
        starts.append(stages(starts[-1])[4])
    qe = starts[-1].clone().requires_grad_(True)
    energy = 0.5 * ((qe[1] ** 2 + qe[2] ** 2 + qe[3] ** 2) / qe[0]).sum() / J
    lam, = torch.autograd.grad(energy, qe)
    for s in reversed(range(case["steps"])):
        st = stages(starts[s])
        total, cur = lam.clone(), lam
        for k in (3, 2, 1, 0):
            x = st[k].detach().requires_grad_(True)
            g, = torch.autograd.grad(rhs(x), x, cur)
            cur = -dt / (4 - k) * J * g
            total += cur
        lam = total
    return {"J": float(energy.detach()), "grad": lam.reshape(-1)}


def _linear(f, x, dx):
    """Directional derivative of f at x along dx, as the gradient of <f'(x)^T v, dx> with respect to v."""
    x = x.detach().requires_grad_(True)
    y = f(x)
    v = torch.zeros_like(y, requires_grad=True)
    g, = torch.autograd.grad(y, x, v, create_graph=True)
    out, = torch.autograd.grad((g * dx).sum(), v)
    return out


def _exact_dropin(case, dims, q0, met, J, mu):
    op = _Operators(dims, _nbc(case))
    shape = (5, dims[2], dims[1], dims[0])
    q0 = q0.view(shape)
    dt = _time_step(q0, met, J, mu, _UMF, _CFL)
    cur = q0
    for k in range(4):
        de, dx_flux = _rhs_terms(op, cur, met, J, mu, _UMF, case["viscous"])
        base = de.clone()
        faces = ([(0, None)] if case["open_x"] else []) + ([(1, (_ACC, 1.0 / dt))] if case["walls_y"] else [])
        for axis, wall in faces:
            for ip in (0, 1):
                i = -ip
                at = (lambda f: f[..., i]) if axis == 0 else (lambda f: f[..., i, :])
                src = at(dx_flux) if wall is None else at(base)
                cm = [at(met[axis][c]).reshape(-1) for c in range(3)]
                nrm = torch.sqrt(cm[0] ** 2 + cm[1] ** 2 + cm[2] ** 2)
                Jf = at(J).reshape(-1)
                dq = _characteristic(at(cur).reshape(5, -1), src.reshape(5, -1), Jf, [c / nrm for c in cm], ip, _UMF, wall)
                _planes(case, de, dq, J, axis, ip)
        cur = q0 - dt / (4 - k) * J * de
        if case["walls_y"]:
            cur = cur.clone()
            for i in (0, -1):
                rho = cur[0, :, i].clone()
                for c in range(3):
                    cur[1 + c, :, i] = -rho * _UMF[c]
                cur[4, :, i] = rho / (GAM * (GAM - 1.0)) + 0.5 * rho * sum(v * v for v in _UMF)
    return {"dt": dt, "q": cur.reshape(-1), "rhs": de.reshape(-1)}


def _planes(case, de, dq, J, axis, ip):
    """de += sbcc dq on the four planes next to a face (sbcc is 1/J on the closed faces' planes, 0 elsewhere)."""
    s = _sbcc(case, J.reshape(-1)).view(J.shape)
    for ii in range(4):
        i = ii if ip == 0 else -1 - ii
        if axis == 0:
            de[..., i] += s[..., i] * dq.reshape(de[..., i].shape)
        else:
            de[..., i, :] += s[..., i, :] * dq.reshape(de[..., i, :].shape)


def _rhs_terms(op, q, met, J, mu, umf, viscous):
    """(right-hand side, its x-derivative term) without boundary closures."""
    class Split:
        first = None

        def d(self, axis, f):
            got = op.d(axis, f)
            if axis == 0 and f.shape[0] == 5:
                self.first = got
            return got
    split = Split()
    return _rhs(split, q, met, J, mu, umf, viscous, False), split.first
