"""Performance cases of the engine: the calls a host program makes, over the sizes it makes them at.

A case is a dict: `kind` is the entry point, `model` the flow, `nx`, `ny`, `nz` the cells, `scheme` the
reconstruction, `precision` the form (fp64 or mixed) and `steps` the time steps of one pass.

kind "rhs"     FillPatch + compute_dUdt_FV on the caller's arrays (a host that integrates in time itself)
     "step"    one TVD-RK3 step through the drop-in stage entry points (a host that owns its state arrays)
     "solve"   a level object: upload an initial state, advance `steps` steps, download the result
     "batch"   a box list of uneven independent boxes advanced together
     "amr"     the multi-level object: subcycled levels, refluxing and average-down

model "disc"    2D five-equation advected interface, periodic
      "bubble"  2D five-equation shock-bubble interaction, walls and outflow
      "droplet" 3D six-equation shock-droplet interaction, relaxation after every stage
      "triple"  2D N-phase five-equation triple point, three phases, walls

The flows are those of compas_b200.cases with a smooth velocity perturbation, drawn from the seed with
the flow's own parameters, so that no component of the state is zero by symmetry.
"""
import math
import random

import torch

import compas_b200 as cb
from compas_b200 import amr, cases

DEVICE = "cuda"
FIELDS = {"disc": 6, "bubble": 6, "droplet": 8, "triple": 9}  # conserved components
DIMS = {"disc": 2, "bubble": 2, "droplet": 3, "triple": 2}
TRIPLE_PHASES = 3


def _case(kind, model, nx, ny, nz, scheme, precision, steps, **more):
    c = dict(kind=kind, model=model, nx=nx, ny=ny, nz=nz, scheme=scheme, precision=precision, steps=steps)
    c.update(more)
    return c


def listed():
    out = [
        # the smallest call: one right-hand side of a small box, where launches and latency count
        ("rhs_disc_64_fp64", _case("rhs", "disc", 64, 64, 1, "WENO5", "fp64", 1)),
        # the CPU-runnable configuration: many short steps of a small level, replayed as a graph
        ("solve_disc_128_fp64", _case("solve", "disc", 128, 128, 1, "WENO5", "fp64", 20)),
        # a mid-sized level at odd sizes in the plain form
        ("solve_bubble_1021x509_fp64", _case("solve", "bubble", 1021, 509, 1, "WENO5B", "fp64", 2)),
        # the 2D configuration's full size in the mixed form
        ("solve_bubble_2048x1024_mixed", _case("solve", "bubble", 2048, 1024, 1, "WENO5B", "mixed", 4)),
        # a ragged 3D box (no side a multiple of a tile), the stages driven by the host program
        ("step_droplet_93x61x77_mixed", _case("step", "droplet", 93, 61, 77, "WENO5", "mixed", 1)),
        # the 3D configuration in the plain form, at a size a request has
        ("solve_droplet_96_fp64", _case("solve", "droplet", 96, 96, 96, "WENO5", "fp64", 1)),
        # the largest: the 3D configuration's full size in the mixed form
        ("solve_droplet_256_mixed", _case("solve", "droplet", 256, 256, 256, "WENO5", "mixed", 2)),
        # a shock-droplet request with the bounded scheme
        ("solve_droplet_128_weno5b_mixed", _case("solve", "droplet", 128, 128, 128, "WENO5B", "mixed", 2)),
        # an N-phase request
        ("solve_triple_896x384_mixed", _case("solve", "triple", 896, 384, 1, "WENO5", "mixed", 4)),
        # independent cases of uneven size in one box list
        ("batch_24_bubbles_mixed", _case("batch", "bubble", 0, 0, 1, "WENO5B", "mixed", 2, boxes=24, lo=64, hi=512)),
        # three refinement levels around the bubble
        ("amr_bubble_256x128_mixed", _case("amr", "bubble", 256, 128, 1, "WENO5B", "mixed", 1, grid=64)),
        # the regularised interface: a hyperbolic step and a Phase-Field step with its elliptic solve
        ("solve_bubble_512x256_cac_mixed", _case("solve", "bubble", 512, 256, 1, "WENO5B", "mixed", 4, cac=True)),
    ]
    return [dict(c, name=name) for name, c in out]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rhs", "step", "solve", "solve", "solve", "batch", "amr"])
    precision = rng.choice(["fp64", "mixed", "mixed"])
    scheme = rng.choice(["WENO5", "WENO5B"])
    if kind == "batch":
        lo = _log_uniform(rng, 48, 128)
        return _case("batch", "bubble", 0, 0, 1, scheme, precision, rng.randint(1, 3),
                     boxes=rng.randint(4, 32), lo=lo, hi=lo * rng.randint(2, 5))
    if kind == "amr":
        ny = 32 * rng.randint(2, 8)
        return _case("amr", "bubble", 2 * ny, ny, 1, "WENO5B", precision, 1, grid=rng.choice([32, 64, 128]))
    model = rng.choice(["disc", "bubble", "bubble", "droplet", "droplet", "triple"])
    if model == "disc":
        nx = ny = _log_uniform(rng, 48, 768)
        nz, scheme = 1, "WENO5"
    elif model == "bubble":
        ny, nz = _log_uniform(rng, 64, 1024), 1
        nx = int(ny * rng.uniform(1.0, 2.0))
    elif model == "triple":
        m = _log_uniform(rng, 16, 160)
        nx, ny, nz, scheme = 7 * m, 3 * m, 1, "WENO5"
    else:
        nx = _log_uniform(rng, 32, 192 if precision == "mixed" else 96)
        ny, nz = (max(16, int(nx * rng.uniform(0.6, 1.0))) for _ in range(2))
    cells = nx * ny * nz
    steps = 1 if kind in ("rhs", "step") else max(1, min(20, 400000 // cells))
    return _case(kind, model, nx, ny, nz, scheme, precision, steps)


# ---- inputs -------------------------------------------------------------------------------------

# velocity scale of the perturbation, a few per cent of the flow's sound speed
_PERTURB = {"disc": 5.0, "bubble": 0.05, "droplet": 20.0, "triple": 0.03}


def _perturb(model, U, dx, r):
    """Add a smooth velocity to the valid cells of the padded state U, momentum and energy alike."""
    dim, ng = DIMS[model], 3
    gz = ng if dim == 3 else 0
    V = U[:, gz:U.shape[1] - gz, ng:U.shape[2] - ng, ng:U.shape[3] - ng]
    nz, ny, nx = V.shape[1:]
    ax = [(torch.arange(n, dtype=torch.float64, device=U.device) + 0.5) * h for n, h in ((nx, dx[0]), (ny, dx[1]), (nz, dx[2]))]
    X, Y, Z = ax[0][None, None, :], ax[1][None, :, None], ax[2][:, None, None]
    first = 3 if model == "triple" else 2  # the momentum components follow the masses
    rho = V[:first].sum(0)
    amp = _PERTURB[model]
    du = []
    for d in range(dim):
        kx, ky, kz = (2.0 * math.pi * r.randint(1, 3) for _ in range(3))
        a, b, c = (r.uniform(0.0, 2.0 * math.pi) for _ in range(3))
        du.append(amp * torch.sin(kx * X + a) * torch.cos(ky * Y + b) * (torch.cos(kz * Z + c) if dim == 3 else 1.0))
    work = sum(V[first + d] * du[d] + 0.5 * rho * du[d] * du[d] for d in range(dim))  # change of the kinetic energy
    if model == "droplet":
        y1 = V[0] / rho
        V[first + dim] += y1 * work
        V[first + dim + 1] += (1.0 - y1) * work
    else:
        V[first + dim] += work
    for d in range(dim):
        V[first + d] += rho * du[d]
    return U


def _flow(case, r, nx=None, ny=None):
    """(physics, dim, inputs, geom kwargs, padded state) of the case's flow for the random.Random r."""
    model = case["model"]
    nx, ny, nz = nx or case["nx"], ny or case["ny"], case["nz"]
    kw = dict(quadrature=False, xp=torch, device=DEVICE)
    if model == "disc":
        phys, dim, inputs, geom, U = cases.advected_disc(n=nx, **kw)
    elif model == "bubble":
        radius = r.uniform(0.15, 0.25)
        phys, dim, inputs, geom, U = cases.shock_bubble(
            nx=nx, ny=ny, Ma=r.uniform(1.15, 1.5), rho_b=math.exp(r.uniform(math.log(0.1), math.log(5.0))), radius=radius,
            center=(0.3 + radius, r.uniform(0.45, 0.55)), scheme=case["scheme"], length=nx / ny, **kw)
    elif model == "triple":
        phys, dim, inputs, geom, U = cases.triple_point(m=ny // 3, **kw)
    else:
        n = max(nx, ny, nz)
        phys, dim, inputs, geom, U = cases.shock_droplet(n=n, Ma=r.uniform(2.0, 2.6), **kw)
        j, k = (n - ny) // 2, (n - nz) // 2  # a box that holds the shock and the droplet
        U = U[:, k:k + nz + 6, j:j + ny + 6, :nx + 6].contiguous()
        U[:, :3] = U[:, -3:] = 0.0
        U[:, :, :3] = U[:, :, -3:] = 0.0
        U[:, :, :, :3] = U[:, :, :, -3:] = 0.0
        geom = dict(geom, n=(nx, ny, nz))
    inputs = dict(inputs, **{"FiniteVolume.Scheme": case["scheme"]})
    return phys, dim, inputs, geom, _perturb(model, U, geom["dx"], r)


# largest wave speed that the initial flow can have (sets the step size of the "step" calls)
_SPEED = {"disc": 2200.0, "bubble": 5.0, "droplet": 3500.0, "triple": 3.0}


def _batch_flows(case, seed):
    r = random.Random(int(seed))
    sides = random.Random(int(case["boxes"]) * 1000 + int(case["lo"]))  # the sizes are the case's, not the seed's
    out = []
    for _ in range(case["boxes"]):
        ny = sides.randint(case["lo"], case["hi"])
        nx = int(ny * sides.uniform(1.0, 2.0))
        out.append(_flow(case, r, nx, ny))
    return out


def _amr_layout(case):
    """Level 0 and two nested refined regions in the proportions of the AMR configuration."""
    nx, ny = case["nx"], case["ny"]
    f = nx / 512.0
    regions = [((int(64 * f), int(96 * f), 0), (int(896 * f) - 1, int(416 * f) - 1, 0)),
               ((int(512 * f), int(256 * f), 0), (int(1408 * f) - 1, int(768 * f) - 1, 0))]
    return amr.hierarchy((nx, ny), 2, regions, case["grid"])


def _amr_flows(case, seed):
    boxes = _amr_layout(case)

    def flow(ng, xp, device, nx, ny):
        return _flow(case, random.Random(int(seed)), nx, ny)

    states = amr.box_states(flow, dict(nx=case["nx"], ny=case["ny"]), (case["nx"], case["ny"]), 2, boxes, xp=torch, device=DEVICE)
    return boxes, states


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case = case
    extra = {"compas_b200.precision": case["precision"]}
    if case.get("cac"):
        extra.update({"PhaseField.phase_field": "1", "PhaseField.Mechanism": "CAC-Adv"})
    if case["kind"] == "batch":
        flows = _batch_flows(case, seed)
        phys, dim = flows[0][:2]
        first = cb.make_parm(phys, dim, dict(flows[0][2], **extra))
        s.batch = cb.Batch(phys, dim, id_limiter=first.id_limiter, precision=first.precision)
        s.ids, s.outs, s.views = [], [], []
        for phys, dim, inputs, geom, U in flows:
            p, g = cb.make_parm(phys, dim, dict(inputs, **extra)), cb.make_geom(**geom)
            s.ids.append(s.batch.add(p, g, U))
            s.outs.append(torch.empty_like(U))
            s.views.append(cb.valid_view(s.outs[-1], p, g))
        return s
    if case["kind"] == "amr":
        boxes, states = _amr_flows(case, seed)
        phys, dim, inputs, geom, _ = _flow(case, random.Random(int(seed)))
        p = cb.make_parm(phys, dim, dict(inputs, **extra))
        s.amr = cb.Amr(p, cb.make_geom(**geom), boxes)
        for b, U in enumerate(states):
            s.amr.upload(b, U)
        s.outs = [torch.empty_like(U) for U in states]
        s.views = [o[:, :, 3:-3, 3:-3] for o in s.outs]
        return s
    phys, dim, inputs, geom, U = _flow(case, random.Random(int(seed)))
    s.p, s.g, s.U = cb.make_parm(phys, dim, dict(inputs, **extra)), cb.make_geom(**geom), U
    if case["kind"] == "solve":
        s.level = cb.Level(s.p, s.g)
        s.out = torch.empty_like(U)
    else:
        s.cmax = torch.zeros(1, dtype=torch.float64, device=DEVICE)
        s.err = torch.zeros(1, dtype=torch.int32, device=DEVICE)
        s.dt = torch.full((1,), 0.4 * min(geom["dx"][:dim]) / _SPEED[case["model"]], dtype=torch.float64, device=DEVICE)
        s.stages = [torch.zeros_like(U) for _ in range(1 if case["kind"] == "rhs" else 3)]
        s.out = s.stages[-1]
    s.view = cb.valid_view(s.out, s.p, s.g)
    return s


def run(s):
    kind = s.case["kind"]
    if kind == "batch":
        s.batch.advance(s.case["steps"])
        for i, o in zip(s.ids, s.outs):
            s.batch.download(i, out=o)
        return list(s.views)
    if kind == "amr":
        s.amr.advance(s.case["steps"])
        for b, o in enumerate(s.outs):
            s.amr.download(b, out=o)
        return list(s.views)
    if kind == "solve":
        s.level.upload(s.U)
        s.level.advance(s.case["steps"])
        s.level.download(out=s.out)
        return {"u%d" % n: s.view[n] for n in range(s.view.shape[0])}
    s.cmax.zero_()
    if kind == "rhs":
        cb.FillPatch(s.p, s.g, s.U)
        cb.compute_dUdt_FV(s.p, s.g, s.U, s.out, cmax=s.cmax, err=s.err)
    else:
        src = s.U
        for k in range(3):
            cb.FillPatch(s.p, s.g, src)
            cb.ThirdOrderSSPRK_stage(s.p, s.g, k, src, s.U, s.stages[k], s.dt, cmax=s.cmax, err=s.err)
            src = s.stages[k]
    return dict({"u%d" % n: s.view[n] for n in range(s.view.shape[0])}, cmax=s.cmax)


# ---- cost and tolerance -------------------------------------------------------------------------

def work(case):
    """Bytes: per stage the state that it reads and writes ((2 + 3 + 3)/3 states a stage), for a
    solve also the copies in and out. Operations: per cell and stage and direction, two fifth-order face values
    of every component (about 60 operations each) and the Riemann flux (about 30 a component)."""
    N, D = FIELDS[case["model"]], DIMS[case["model"]]
    state = 8.0 * N
    if case["kind"] == "batch":
        sides = random.Random(int(case["boxes"]) * 1000 + int(case["lo"]))
        cells = 0
        for _ in range(case["boxes"]):
            ny = sides.randint(case["lo"], case["hi"])
            cells += ny * int(ny * sides.uniform(1.0, 2.0))
        updates, copied = 3.0 * case["steps"] * cells, cells
    elif case["kind"] == "amr":
        cells = [0, 0, 0]
        for lev, lo, hi in _amr_layout(case):
            cells[lev] += (hi[0] - lo[0] + 1) * (hi[1] - lo[1] + 1)
        updates, copied = 3.0 * case["steps"] * sum(c << lev for lev, c in enumerate(cells)), sum(cells)
    else:
        copied = case["nx"] * case["ny"] * case["nz"]
        updates = copied * (1.0 if case["kind"] == "rhs" else 3.0 * case["steps"])
        if case["kind"] == "solve":
            updates += copied  # the wave speeds of the initial state set the first step
            copied *= 2
        else:
            copied = 0
    per_stage = state * (2.0 if case["kind"] == "rhs" else 8.0 / 3.0)
    return {"bytes": updates * per_stage + 2.0 * state * copied, "flops": updates * D * N * 150.0}


def tolerance(case):
    """The plain form carries 64 bits throughout, the mixed form reconstructs in 32. A right-hand side is a
    difference of fluxes: where velocity and pressure are uniform (the advected disc) its momentum part
    cancels to about a thousandth of the flux. The Phase-Field step adds an elliptic solve to a relative
    residual of 1e-10; the limiters switch on thresholds, hence the wide bound on single values."""
    if case["precision"] == "fp64":
        return {"rel": 2e-10, "max": 1e-7}
    if case["kind"] == "rhs":
        return {"rel": 1.2e-3 if case["model"] == "disc" else 2e-5, "max": 5e-2}
    return {"rel": 5e-6, "max": 5e-3}


# ---- the same results in 64 bits with plain torch ------------------------------------------------

class _Eos:
    """gamma and pinf of every phase as A = 1/(gamma - 1), B = gamma pinf/(gamma - 1)."""

    def __init__(self, model, inputs):
        if model == "triple":
            gam, pinf = inputs["prob.EOS.gamma"], inputs["prob.EOS.pinf"]
        else:
            gam = [inputs["prob.EOS.gamma_1"], inputs["prob.EOS.gamma_2"]]
            pinf = [inputs.get("prob.EOS.pinf_1", 0.0), inputs.get("prob.EOS.pinf_2", 0.0)]
        self.np = len(gam)
        self.A = [1.0 / (g - 1.0) for g in gam]
        self.B = [g * q / (g - 1.0) for g, q in zip(gam, pinf)]


def _fill(U, dim, codes_lo, codes_hi, mom):
    """Ghost cells direction by direction: 0 periodic, 2 outflow, 4 reflecting wall."""
    ng = 3
    for d in range(dim):
        axis = 3 - d
        n = U.shape[axis] - 2 * ng
        for side, code in ((0, codes_lo[d]), (1, codes_hi[d])):
            for g in range(ng):
                dst = g if side == 0 else ng + n + g
                if code == 0:
                    src = dst + n if side == 0 else dst - n
                elif code == 2:
                    src = ng if side == 0 else ng + n - 1
                else:
                    src = 2 * ng - 1 - dst if side == 0 else 2 * (ng + n) - 1 - dst
                U.select(axis, dst).copy_(U.select(axis, src))
                if code == 4:
                    U.select(axis, dst)[mom + d].neg_()


def _prims(model, U, e, dim):
    """Masses, velocities, pressure(s) and volume fractions in the order of the conserved state."""
    npm = e.np
    rho = U[:npm].sum(0)
    W = U.clone()
    for d in range(dim):
        W[npm + d] = U[npm + d] / rho
    k = sum(W[npm + d] ** 2 for d in range(dim))
    if model == "droplet":
        al = [U[-1], 1.0 - U[-1]]
        for q in range(2):
            W[npm + dim + q] = (U[npm + dim + q] - 0.5 * U[q] * k - al[q] * e.B[q]) / e.A[q]
    else:
        al = [U[npm + dim + 1 + q] for q in range(npm)] if model == "triple" else [U[-1], 1.0 - U[-1]]
        AP = sum(a * A for a, A in zip(al, e.A))
        BP = sum(a * B for a, B in zip(al, e.B))
        W[npm + dim] = (U[npm + dim] - 0.5 * rho * k - BP) / AP
    return W


def _cons(model, W, e, dim):
    npm = e.np
    rho = W[:npm].sum(0)
    U = W.clone()
    for d in range(dim):
        U[npm + d] = rho * W[npm + d]
    k = sum(W[npm + d] ** 2 for d in range(dim))
    if model == "droplet":
        al = [W[-1], 1.0 - W[-1]]
        for q in range(2):
            U[npm + dim + q] = e.A[q] * W[npm + dim + q] + al[q] * e.B[q] + 0.5 * W[q] * k
    else:
        al = [W[npm + dim + 1 + q] for q in range(npm)] if model == "triple" else [W[-1], 1.0 - W[-1]]
        AP = sum(a * A for a, A in zip(al, e.A))
        BP = sum(a * B for a, B in zip(al, e.B))
        U[npm + dim] = AP * W[npm + dim] + BP + 0.5 * rho * k
    return U


def _candidates(f, side):
    c, p, m = f[3] - f[2], f[4] - f[3], f[2] - f[1]
    g = f[1] - f[0]
    if side > 0:
        return (f[2] + 2.0 / 3.0 * c - 1.0 / 6.0 * p, f[2] + 1.0 / 6.0 * m + 1.0 / 3.0 * c, f[2] - 1.0 / 3.0 * g + 5.0 / 6.0 * m)
    return (f[2] - 5.0 / 6.0 * c + 1.0 / 3.0 * p, f[2] - 1.0 / 3.0 * m - 1.0 / 6.0 * c, f[2] + 1.0 / 6.0 * g - 2.0 / 3.0 * m)


def _weights(f, side):
    c, p, m, g = f[3] - f[2], f[4] - f[3], f[2] - f[1], f[1] - f[0]
    d = (0.3, 0.6, 0.1) if side > 0 else (0.1, 0.6, 0.3)
    s = [10.0 / 3.0 * c * c - 11.0 / 3.0 * c * p + 4.0 / 3.0 * p * p,
         4.0 / 3.0 * m * m - 5.0 / 3.0 * m * c + 4.0 / 3.0 * c * c,
         10.0 / 3.0 * m * m - 11.0 / 3.0 * g * m + 4.0 / 3.0 * g * g]

    def ratio(a, b):
        q = a / b
        return torch.where(torch.isnan(q), torch.ones_like(q), q)

    r01, r02, r12 = ratio(s[0], s[1]), ratio(s[0], s[2]), ratio(s[1], s[2])
    return (d[0] / (d[0] + r01 ** 2 * d[1] + r02 ** 2 * d[2]),
            d[1] / ((1.0 / r01) ** 2 * d[0] + d[1] + r12 ** 2 * d[2]),
            d[2] / ((1.0 / r02) ** 2 * d[0] + (1.0 / r12) ** 2 * d[1] + d[2]))


def _dot(w, q):
    return w[0] * q[0] + w[1] * q[1] + w[2] * q[2]


def _theta(c, fl, fr):
    """Largest factor that keeps the cell's two face values and its interior value non-negative."""
    inner = (c - fl / 12.0 - fr / 12.0) / (1.0 - 1.0 / 6.0)
    low = torch.minimum(inner, torch.minimum(fl, fr))
    th = torch.clamp(c, min=0.0) / torch.clamp(c - low, min=0.0)
    return torch.where(th < 1.0, th, torch.ones_like(th))


def _bounded_faces(masses, alphas):
    """Both faces (right, left) of every cell: bounded masses and volume fractions, one pass per phase and a common one."""
    R, L, aR, aL = [], [], [], []
    for fr, fa in zip(masses, alphas):
        face = []
        for side in (1, -1):
            w = _weights(fr, side)
            face.append((_dot(w, _candidates(fr, side)), _dot(w, _candidates(fa, side))))
        (r, a), (l, b) = face
        th = torch.minimum(_theta(fr[2], r, l), _theta(fa[2], a, b))
        R.append(fr[2] + th * (r - fr[2]))
        aR.append(fa[2] + th * (a - fa[2]))
        L.append(fr[2] + th * (l - fr[2]))
        aL.append(fa[2] + th * (b - fa[2]))
    sR, sL = sum(aR), sum(aL)
    th = torch.ones_like(sR)
    for k, (fr, fa) in enumerate(zip(masses, alphas)):
        R[k], aR[k], L[k], aL[k] = R[k] / sR, aR[k] / sR, L[k] / sL, aL[k] / sL
        th = torch.minimum(th, torch.minimum(_theta(fr[2], R[k], L[k]), _theta(fa[2], aR[k], aL[k])))
    at = [(fr[2], fa[2]) for fr, fa in zip(masses, alphas)]
    right = [(c + th * (r - c), a + th * (x - a)) for (c, a), r, x in zip(at, R, aR)]
    left = [(c + th * (r - c), a + th * (x - a)) for (c, a), r, x in zip(at, L, aL)]
    return right, left


def _consistent(W, C, npm, ia, h):
    """N-phase consistent limiting of the masses and volume fractions of the face values W, at the signed
    distance h from the cells of values C."""
    sa = [(W[ia + k] - C[ia + k]) / h for k in range(npm)]
    total = sum(sa)
    mag = torch.stack([a.abs() for a in sa])
    top = mag.argmax(0)
    smax = torch.gather(torch.stack(sa), 0, top[None])[0]
    rest = smax - total
    idle = (smax.abs() < 1e-10) | (total.abs() < 1e-10)
    one = torch.ones_like(total)
    t_other = torch.where(idle, one, torch.clamp(smax / rest, 0.0, 1.0))
    t_max = torch.where(idle, one, torch.clamp(rest / smax, 0.0, 1.0))
    for k in range(npm):
        th = torch.where(top == k, t_max, t_other)
        W[k] = C[k] + h * th * ((W[k] - C[k]) / h)
        W[ia + k] = C[ia + k] + h * th * sa[k]


def _faces(model, W, e, dim, d, scheme, dx):
    """Left and right primitive states of the n + 1 faces along d (W: primitives with ghosts along d only)."""
    axis = 3 - d
    n = W.shape[axis] - 6
    f = [W.narrow(axis, s, n + 1) for s in range(6)]
    npm, N = e.np, W.shape[0]
    WL, WR = torch.empty_like(f[0]), torch.empty_like(f[0])
    plain = range(N)
    if scheme == "WENO5B":
        plain = range(npm, N - 1)
        cells = [W.narrow(axis, s, n + 2) for s in range(5)]
        masses = [[c[k] for c in cells] for k in range(2)]
        alphas = [[c[N - 1] for c in cells], [1.0 - c[N - 1] for c in cells]]
        right, left = _bounded_faces(masses, alphas)
        ax = axis - 1
        for k in range(2):
            WL[k] = right[k][0].narrow(ax, 0, n + 1)
            WR[k] = left[k][0].narrow(ax, 1, n + 1)
        WL[N - 1] = right[0][1].narrow(ax, 0, n + 1)
        WR[N - 1] = left[0][1].narrow(ax, 1, n + 1)
    for c in plain:
        l, r = [x[c] for x in f[:5]], [x[c] for x in f[1:]]
        WL[c] = _dot(_weights(l, 1), _candidates(l, 1))
        WR[c] = _dot(_weights(r, -1), _candidates(r, -1))
    if model == "triple":
        _consistent(WL, f[2], npm, npm + dim + 1, 0.5 * dx)
        _consistent(WR, f[3], npm, npm + dim + 1, -0.5 * dx)
    return WL, WR


def _speed(model, W, e, dim):
    npm = e.np
    rho = W[:npm].sum(0)
    if model == "droplet":
        al = [W[-1], 1.0 - W[-1]]
        rc2 = sum(((A + 1.0) * W[npm + dim + q] + al[q] * B) / A for q, (A, B) in enumerate(zip(e.A, e.B)))
    else:
        p = W[npm + dim]
        al = [W[npm + dim + 1 + q] for q in range(npm)] if model == "triple" else [W[-1], 1.0 - W[-1]]
        rc2 = sum(a * ((A + 1.0) * p + B) for a, A, B in zip(al, e.A, e.B)) / sum(a * A for a, A in zip(al, e.A))
    return torch.sqrt(rc2 / rho)


def _hllc(model, WL, WR, e, dim, d):
    """Flux, the face values of the non-conservative terms, and the face wave speed."""
    npm = e.np
    six = model == "droplet"
    UL, UR = _cons(model, WL, e, dim), _cons(model, WR, e, dim)
    cL, cR = _speed(model, WL, e, dim), _speed(model, WR, e, dim)
    VL, VR = WL[npm + d], WR[npm + d]
    ie = npm + dim
    pL, pR = (WL[ie] + WL[ie + 1], WR[ie] + WR[ie + 1]) if six else (WL[ie], WR[ie])
    if six:
        SL, SR = torch.minimum(VL - cL, VR - cR), torch.maximum(VL + cL, VR + cR)
    else:
        SL, SR = torch.minimum(0.5 * (VL + VR) - 0.5 * (cL + cR), VL - cL), torch.maximum(0.5 * (VL + VR) + 0.5 * (cL + cR), VR + cR)
    Sm, Sp = torch.clamp(SL, max=0.0), torch.clamp(SR, min=0.0)
    rL, rR = WL[:npm].sum(0), WR[:npm].sum(0)
    S = (pR - pL + rL * VL * (SL - VL) - rR * VR * (SR - VR)) / (rL * (SL - VL) - rR * (SR - VR))
    sgn = torch.sign(S)
    F, nc = None, None
    for U, W, V, p, rho, Sk, Sb, h in ((UL, WL, VL, pL, rL, SL, Sm, 0.5 * (1.0 + sgn)), (UR, WR, VR, pR, rR, SR, Sp, 0.5 * (1.0 - sgn))):
        f = (Sk - V) / (Sk - S)
        flux, star = U * V, f * U
        flux[npm + d] += p
        star[npm + d] += f * rho * (S - V)
        face = [h * (V + Sb * (f - 1.0))]
        if six:
            for q in range(2):
                ap = W[ie + q]
                aps = ap + W[q] * (Sk - V) * (S - V)
                flux[ie + q] += ap * V
                star[ie + q] += (V * ap - S * aps) / (S - Sk)
                face.append(h * (V * ap + Sb * (V * ap - S * aps) / (S - Sk)))
        else:
            flux[ie] += p * V
            star[ie] += f * (S - V) * (rho * S + p / (Sk - V))
        part = h * (flux + Sb * (star - U))
        F = part if F is None else F + part
        nc = face if nc is None else [a + b for a, b in zip(nc, face)]
    speed = torch.maximum(cL + torch.sqrt(sum(WL[npm + c] ** 2 for c in range(dim))),
                          cR + torch.sqrt(sum(WR[npm + c] ** 2 for c in range(dim))))
    return F, nc, speed


def _rhs(model, U, e, dim, scheme, dx, fill):
    """(dU/dt of the valid cells, largest face wave speed) of the padded state U, whose ghosts are filled here."""
    fill(U)
    W = _prims(model, U, e, dim)
    ng, npm = 3, e.np
    core = [slice(None)] + [slice(ng, W.shape[a] - ng) if (a > 1 or dim == 3) else slice(None) for a in (1, 2, 3)]
    Wc = W[tuple(core)]
    div, nc_div, cmax = torch.zeros_like(Wc), None, 0.0
    for d in range(dim):
        axis = 3 - d
        cut = list(core)
        cut[axis] = slice(None)
        F, nc, speed = _hllc(model, *_faces(model, W[tuple(cut)], e, dim, d, scheme, dx[d]), e, dim, d)
        n = Wc.shape[axis]
        div += (F.narrow(axis, 1, n) - F.narrow(axis, 0, n)) / dx[d]
        parts = [(q.narrow(axis - 1, 1, n) - q.narrow(axis - 1, 0, n)) / dx[d] for q in nc]
        nc_div = parts if nc_div is None else [a + b for a, b in zip(nc_div, parts)]
        cmax = max(cmax, float(speed.narrow(axis - 1, 0, n).max()))
        del F, nc, speed
    L = -div
    if model == "droplet":
        rho = Wc[:2].sum(0)
        ie = npm + dim
        g1, g2 = nc_div[1] - Wc[ie] * nc_div[0], nc_div[2] - Wc[ie + 1] * nc_div[0]
        x = Wc[1] / rho * g1 - Wc[0] / rho * g2
        L[ie] += x
        L[ie + 1] -= x
        L[-1] += Wc[-1] * nc_div[0]
    else:
        for c in (range(npm + dim + 1, npm + dim + 1 + npm) if model == "triple" else [Wc.shape[0] - 1]):
            L[c] += Wc[c] * nc_div[0]
    return L, cmax


def _relax(U, e, dim):
    """Instantaneous pressure relaxation of the six-equation state: the closed-form equilibrium pressure."""
    W = _prims("droplet", U, e, dim)
    (A1, A2), (B1, B2) = e.A, e.B
    ie = 2 + dim
    a1, a2 = W[-1], 1.0 - W[-1]
    p1, p2 = W[ie], W[ie + 1]
    a = A1 * A2 + A1 * a1 + A2 * a2
    b = A1 * B2 * a1 + A2 * B1 * a2 - (A2 + 1.0) * A1 * p1 - (A1 + 1.0) * A2 * p2
    c = -B2 * A1 * p1 - B1 * A2 * p2
    p = (-b + torch.sqrt(b * b - 4.0 * a * c)) / (2.0 * a)
    r1 = (A1 * p1 + B1 * a1 + p * a1) / ((A1 + 1.0) * p + B1)
    r2 = (A2 * p2 + B2 * a2 + p * a2) / ((A2 + 1.0) * p + B2)
    r1, r2 = r1 / (r1 + r2), r2 / (r1 + r2)
    p = (A1 * p1 + A2 * p2 + B1 * (a1 - r1) + B2 * (a2 - r2)) / (A1 * r1 + A2 * r2)
    W[ie], W[ie + 1], W[-1] = r1 * p, r2 * p, r1
    return _cons("droplet", W, e, dim)


def _advance(case, phys, dim, inputs, geom, U, steps, dt=None):
    """`steps` TVD-RK3 steps of the padded state U (dt: a fixed step, else from the wave speeds): valid cells, cmax."""
    model, scheme = case["model"], case["scheme"]
    e = _Eos(model, inputs)
    dx = geom["dx"]
    ng = 3
    core = tuple([slice(None)] + [slice(ng, U.shape[a] - ng) if (a > 1 or dim == 3) else slice(None) for a in (1, 2, 3)])

    def fill(X):
        _fill(X, dim, geom["lo_bc"], geom["hi_bc"], e.np)

    fixed, cmax, last = dt, 0.0, None
    if fixed is None:
        cmax = _rhs(model, U.clone(), e, dim, scheme, dx, fill)[1]
    for _ in range(steps):
        if fixed is None:
            dt = min(inputs["run.cfl"] * h / cmax for h in dx[:dim])
            if last is not None and inputs.get("run.timestep_change_limiter", 1):
                dt = min(dt, 1.1 * last)
            last = dt
        cmax = 0.0
        old, cur = U[core].clone(), U
        for k, (a, b, c) in enumerate(((1.0, 0.0, 1.0), (0.25, 0.75, 0.25), (2.0 / 3.0, 1.0 / 3.0, 2.0 / 3.0))):
            L, cm = _rhs(model, cur, e, dim, scheme, dx, fill)
            cmax = max(cmax, cm)
            v = a * cur[core] + b * old + (c * dt) * L
            if model == "droplet":
                v = _relax(v, e, dim)
            cur = U if k == 2 else torch.zeros_like(U)
            cur[core] = v
    return U[core], cmax


def exact(case, seed):
    if case["kind"] == "amr" or case.get("cac"):
        return None  # a hierarchy driver and an elliptic solve of their own
    if case["kind"] == "batch":
        return [_advance(case, *flow, case["steps"])[0] for flow in _batch_flows(case, seed)]
    phys, dim, inputs, geom, U = _flow(case, random.Random(int(seed)))
    if case["kind"] == "rhs":
        e = _Eos(case["model"], inputs)
        L, cmax = _rhs(case["model"], U, e, dim, case["scheme"], geom["dx"], lambda X: _fill(X, dim, geom["lo_bc"], geom["hi_bc"], e.np))
        out = L
    elif case["kind"] == "step":
        dt = 0.4 * min(geom["dx"][:dim]) / _SPEED[case["model"]]
        out, cmax = _advance(case, phys, dim, inputs, geom, U, 1, dt=dt)
    else:
        out = _advance(case, phys, dim, inputs, geom, U, case["steps"])[0]
        return {"u%d" % n: out[n] for n in range(out.shape[0])}
    return dict({"u%d" % n: out[n] for n in range(out.shape[0])}, cmax=torch.tensor([cmax], dtype=torch.float64))
