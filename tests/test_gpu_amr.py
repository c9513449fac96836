"""Multi-level (AMR) advance on the CUDA path against the reference-header oracle's multi-level driver
(oracle/ref_amr.inc), and its invariants.

Both sides run the same fixed hierarchy (refinement ratio 2, subcycling, flux registers with the
five-equation non-conservative alpha1 source or the six-equation phase-energy and alpha1 terms and the
relaxation of the refluxed cells, average-down), the same coarse-fine interpolation and
the reference's own face arithmetic, so the plain FP64 form is compared to the bit (the asserted bound
is 1e-11 relative L-infinity per field and box). The coarse-fine operations follow
AMReX's documented semantics on both sides; AMReX itself is not in the image, so they are not pinned
by the reference. Also: one level of several boxes equals the single-box level; the composite-grid
totals of mass, momentum and energy are conserved to round-off on a periodic domain; every level's
boxes go through one box-list launch per RK stage; the mixed form's error.
"""
import numpy as np
import pytest

import compas_b200 as cb
from compas_b200 import amr, cases
from helpers import rel_linf
from oracle.oracle import Oracle, have_ref

pytestmark = pytest.mark.gpu

TOL = 1e-11


def _valid(U, lo, hi, dim, ng=3):
    if dim == 2:
        return U[:, 0, ng:ng + hi[1] - lo[1] + 1, ng:ng + hi[0] - lo[0] + 1]
    return U[:, ng:ng + hi[2] - lo[2] + 1, ng:ng + hi[1] - lo[1] + 1, ng:ng + hi[0] - lo[0] + 1]


def _run(case_fn, kw, domain, regions, mgs, steps, extra=None, precision="fp64"):
    phys, dim, inputs, geom, _ = case_fn(**kw)
    inputs = dict(inputs, **{"compas_b200.precision": precision}, **(extra or {}))
    p, g = cb.make_parm(phys, dim, inputs), cb.make_geom(**geom)
    boxes = amr.hierarchy(domain, dim, regions, mgs)
    states = amr.box_states(case_fn, kw, domain, dim, boxes)
    A = cb.Amr(p, g, boxes)
    for b, U in enumerate(states):
        A.upload(b, U)
    A.advance(steps)
    info = A.sync()
    got = [A.download(b) for b in range(len(boxes))]
    dts = A.dts(info.steps)
    launches = A.launches()
    A.close()
    return p, g, dim, boxes, states, got, dts, info, launches


def _compare(p, g, dim, boxes, states, got, dts, steps):
    if not have_ref(p.physics, p.dim, p.nphase):
        pytest.skip("reference-header oracle not built")
    ref = [U.copy() for U in states]
    _, dts_ref = Oracle("reference", p, g).amr_advance(boxes, ref, steps)
    np.testing.assert_array_equal(dts, dts_ref)
    worst = np.zeros(ref[0].shape[0])
    for (lev, lo, hi), a, r in zip(boxes, got, ref):
        worst = np.maximum(worst, rel_linf(_valid(a, lo, hi, dim), _valid(r, lo, hi, dim)))
    print(f"{len(boxes)} boxes, {1 + max(b[0] for b in boxes)} levels, {steps} steps: rel Linf per field "
          f"{np.array2string(worst, precision=2)}; bitwise equal: {all(np.array_equal(_valid(a, *b[1:], dim), _valid(r, *b[1:], dim)) for b, a, r in zip(boxes, got, ref))}")
    assert np.all(worst <= TOL), worst


def test_one_level_of_boxes_equals_single_box_level():
    kw = dict(nx=64, ny=32, scheme="WENO5B")
    p, g, dim, boxes, states, got, dts, info, _ = _run(cases.shock_bubble, kw, (64, 32), [], 16, 5)
    phys, _, inputs, geom, U = cases.shock_bubble(**kw)
    lv = cb.Level(p, g)
    lv.upload(U)
    lv.advance(5)
    ref = lv.download()
    lv.close()
    V = cb.valid_view(ref, p, g)
    for (lev, lo, hi), a in zip(boxes, got):
        np.testing.assert_array_equal(_valid(a, lo, hi, dim), V[:, 0, lo[1]:hi[1] + 1, lo[0]:hi[0] + 1])


@pytest.mark.parametrize("case_fn,kw,domain,regions,mgs,steps", [
    (cases.shock_bubble, dict(nx=64, ny=32, scheme="WENO5B"), (64, 32),
     [((40, 16, 0), (95, 47, 0)), ((96, 48, 0), (175, 79, 0))], 32, 4),
    (cases.shock_bubble, dict(nx=48, ny=24, scheme="WENO5"), (48, 24), [((24, 8, 0), (71, 39, 0))], 16, 4),
    (cases.advected_disc, dict(n=32), (32, 32), [((16, 16, 0), (47, 47, 0)), ((40, 40, 0), (87, 87, 0))], 16, 5),
    (cases.advected_interface, dict(n=16, dim=3, physics=cb.FIVEEQS), (16, 16, 16),
     [((8, 8, 8), (23, 23, 23))], 8, 3),
    (cases.advected_interface, dict(n=16, dim=2, physics=cb.SIXEQS), (16, 16),
     [((8, 8, 0), (23, 23, 0)), ((24, 24, 0), (39, 39, 0))], 8, 4),
    (cases.advected_interface, dict(n=16, dim=3, physics=cb.SIXEQS), (16, 16, 16),
     [((8, 8, 8), (23, 23, 23))], 8, 3),
    (cases.shock_droplet, dict(n=16), (16, 16, 16), [((8, 8, 8), (23, 23, 23))], 8, 3),
], ids=["bubble3lev_weno5b", "bubble2lev_weno5", "disc3lev_periodic", "sphere2lev_3d", "sixeq_disc3lev_periodic",
        "sixeq_sphere2lev_3d", "sixeq_droplet2lev_3d"])
def test_amr_matches_oracle(case_fn, kw, domain, regions, mgs, steps):
    p, g, dim, boxes, states, got, dts, info, launches = _run(case_fn, kw, domain, regions, mgs, steps)
    assert info.status == 0 and info.steps == steps
    _compare(p, g, dim, boxes, states, got, dts, steps)


def test_amr_composite_conservation_periodic():
    kw = dict(n=32)
    p, g, dim, boxes, states, got, dts, info, _ = _run(
        cases.advected_disc, kw, (32, 32), [((16, 16, 0), (47, 47, 0)), ((40, 40, 0), (87, 87, 0))], 16, 6)
    cov = amr.covered_mask_fn(boxes, 2)
    for c in range(5):  # masses, momenta, total energy
        s0 = amr.composite_sum(states, boxes, 2, 3, c, cov)
        s1 = amr.composite_sum(got, boxes, 2, 3, c, cov)
        print(f"component {c}: composite total relative change {abs(s1 - s0) / abs(s0):.1e}")
        assert abs(s1 - s0) <= 1e-13 * abs(s0)


def test_sixeq_amr_composite_conservation_periodic():
    kw = dict(n=16, dim=2, physics=cb.SIXEQS)
    p, g, dim, boxes, states, got, dts, info, _ = _run(
        cases.advected_interface, kw, (16, 16), [((8, 8, 0), (23, 23, 0)), ((24, 24, 0), (39, 39, 0))], 8, 6)
    assert info.status == 0
    cov = amr.covered_mask_fn(boxes, 2)

    def totals(st):
        s = [amr.composite_sum(st, boxes, 2, 3, c, cov) for c in range(6)]
        return s[:4] + [s[4] + s[5]]  # masses, momenta, total energy

    for c, (s0, s1) in enumerate(zip(totals(states), totals(got))):
        print(f"quantity {c}: composite total relative change {abs(s1 - s0) / abs(s0):.1e}")
        assert abs(s1 - s0) <= 1e-13 * abs(s0)


def test_amr_levels_use_one_list_launch_per_stage():
    # 3 levels x (1 + 2 + 4 substeps) x 3 stages of list launches plus fills, faces, reflux and average-down
    p, g, dim, boxes, states, got, dts, info, launches = _run(
        cases.shock_bubble, dict(nx=64, ny=32, scheme="WENO5B"), (64, 32),
        [((40, 16, 0), (95, 47, 0)), ((96, 48, 0), (175, 79, 0))], 16, 1)
    nbox = len(boxes)
    assert nbox > 10
    stage_launches = 3 * (1 + 2 + 4)
    print(f"{nbox} boxes, {launches} launches in one coarse step ({stage_launches} box-list stage launches)")
    assert launches < 10 * stage_launches + 20


@pytest.mark.parametrize("args", [
    (cases.shock_bubble, dict(nx=64, ny=32, scheme="WENO5B"), (64, 32),
     [((40, 16, 0), (95, 47, 0)), ((96, 48, 0), (175, 79, 0))], 32, 6),
    (cases.shock_droplet, dict(n=16), (16, 16, 16), [((8, 8, 8), (23, 23, 23))], 8, 6),
], ids=["fiveeq_bubble", "sixeq_droplet"])
def test_amr_mixed_error_vs_fp64(args):
    _, _, dim, boxes, _, a, _, ia, _ = _run(*args, precision="mixed")
    _, _, _, _, _, b, _, ib, _ = _run(*args, precision="fp64")
    assert ia.status == 0 and ib.status == 0
    num = np.zeros(a[0].shape[0])
    den = np.zeros(a[0].shape[0])
    for (lev, lo, hi), x, y in zip(boxes, a, b):
        X, Y = _valid(x, lo, hi, dim), _valid(y, lo, hi, dim)
        num += np.abs(X - Y).reshape(X.shape[0], -1).sum(axis=1)
        den += np.abs(Y).reshape(Y.shape[0], -1).sum(axis=1)
    e = num / den
    print("AMR mixed vs FP64 rel L1 per field:", np.array2string(e, precision=2))
    for c in (0, 1, a[0].shape[0] - 1):  # masses and volume fraction
        assert e[c] <= 1e-5, e


@pytest.mark.parametrize("case_fn,kw,domain,regions,mgs,steps,extra", [
    (cases.triple_point, dict(m=8), (56, 24), [((8, 8, 0), (47, 39, 0)), ((24, 24, 0), (71, 55, 0))], 16, 4,
     {"FiniteVolume.Scheme": "MUSCL-MC"}),
    (cases.triple_point, dict(m=8), (56, 24), [((16, 12, 0), (47, 35, 0))], 16, 4, {}),
    (cases.shock_bubble, dict(nx=48, ny=24, scheme="WENO5"), (48, 24), [((24, 8, 0), (71, 39, 0))], 16, 4,
     {"FiniteVolume.Scheme": "MUSCL-MC"}),
    (cases.shock_bubble, dict(nx=48, ny=24, scheme="WENO5B"), (48, 24), [((24, 8, 0), (71, 39, 0))], 16, 4,
     {"Physics.RiemannSolver": "HLL"}),
    (cases.shock_droplet, dict(n=16), (16, 16, 16), [((8, 8, 8), (23, 23, 23))], 8, 3,
     {"FiniteVolume.Scheme": "WENO3", "Physics.RiemannSolver": "LLF"}),
    (cases.shock_bubble, dict(nx=48, ny=24, scheme="WENO5"), (48, 24), [((24, 8, 0), (71, 39, 0))], 16, 4,
     {"FiniteVolume.Scheme": "WENO3B"}),
    (cases.triple_point, dict(m=8), (56, 24), [((16, 12, 0), (47, 35, 0))], 16, 4,
     {"FiniteVolume.Scheme": "WENO3B"}),
    (cases.shock_bubble, dict(nx=64, ny=32, scheme="WENO5B"), (64, 32),
     [((40, 16, 0), (95, 47, 0)), ((96, 48, 0), (175, 79, 0))], 32, 4, {"amr.Interpolater": "pc_interp"}),
    (cases.shock_droplet, dict(n=16), (16, 16, 16), [((8, 8, 8), (23, 23, 23))], 8, 3,
     {"amr.Interpolater": "pc_interp"}),
], ids=["triple_muscl_mc_3lev", "triple_weno5_2lev", "bubble_muscl_mc", "bubble_hll", "droplet_weno3_llf",
        "bubble_weno3b", "triple_weno3b", "bubble3lev_pc_interp", "droplet2lev_pc_interp"])
def test_amr_schemes_and_nphase_match_oracle(case_fn, kw, domain, regions, mgs, steps, extra):
    """The multi-level advance with the N-phase model (the triple point, as the reference's example runs
    it: MUSCL-MC on a hierarchy), the three-cell schemes, the LLF / HLL Riemann solvers and the
    piecewise-constant coarse-fine interpolation (amr.Interpolater = pc_interp), to the bit."""
    p, g, dim, boxes, states, got, dts, info, launches = _run(case_fn, kw, domain, regions, mgs, steps, extra)
    assert info.status == 0 and info.steps == steps
    _compare(p, g, dim, boxes, states, got, dts, steps)


# ---- fine regions at the domain boundary ---------------------------------------------------------
# The ghost cells are compared with a plain restatement over whole-domain arrays: a level's cells inside the
# domain are its boxes' values, elsewhere the lincc_interp value of the level below; the domain is then
# extended direction by direction with the boundary conditions, and a box takes its part.
def _extend(V, ng, lo_bc, hi_bc, m0, dim):
    """V (component, [z,] y, x) extended by ng cells per side along every direction."""
    for d in range(dim):
        ax = V.ndim - 1 - d
        n = V.shape[ax]
        parts = []
        for code, low in ((lo_bc[d], True), (hi_bc[d], False)):
            k = np.arange(-ng, 0) if low else np.arange(n, n + ng)
            if code == 0:
                src, odd = k % n, ()
            elif code == 2:
                src, odd = np.full(ng, 0 if low else n - 1), ()
            else:
                src = -1 - k if low else 2 * n - 1 - k
                odd = (m0 + d,) if code in (3, 4) else tuple(range(m0, m0 + dim))
            g = np.take(V, src, axis=ax)
            for c in odd:
                g[c] = -g[c]
            parts.append(g)
        V = np.concatenate([parts[0], V, parts[1]], axis=ax)
    return V


def _lincc(C, lo_bc, hi_bc, m0, dim):
    """The values of every fine cell from the coarse whole-domain array C."""
    E = _extend(C, 1, lo_bc, hi_bc, m0, dim)
    inner = (slice(None),) + (slice(1, -1),) * dim
    F = E[inner]
    for d in range(dim):
        F = np.repeat(F, 2, axis=F.ndim - 1 - d)
    for d in range(dim):
        ax = E.ndim - 1 - d
        sl = [list(inner) for _ in range(2)]
        sl[0][ax], sl[1][ax] = slice(0, -2), slice(2, None)
        um, uc, up = E[tuple(sl[0])], E[inner], E[tuple(sl[1])]
        dc, df, db = 0.5 * (up - um), 2.0 * (up - uc), 2.0 * (uc - um)
        sx = np.where(df * db >= 0.0, np.minimum(np.abs(df), np.abs(db)), 0.0)
        sx = np.copysign(1.0, dc) * np.minimum(sx, np.abs(dc))
        with np.errstate(all="ignore"):
            sf = np.minimum(1.0, np.where(dc != 0.0, sx / dc, 1.0).min(0))
        slope = dc * sf
        for e in range(dim):
            slope = np.repeat(slope, 2, axis=slope.ndim - 1 - e)
        off = np.where(np.arange(F.shape[ax]) % 2, 0.25, -0.25)
        F = F + off.reshape([-1 if a == ax else 1 for a in range(F.ndim)]) * slope
    return F


WALLS = {"walls": ((4, 3, 5), (3, 5, 4)), "outflow_slip": ((2, 4, 3), (4, 2, 2)), "noslip_periodic": ((5, 0, 2), (2, 0, 5))}


@pytest.mark.parametrize("bc", list(WALLS))
@pytest.mark.parametrize("name,domain,regions,mgs", [
    ("corner2d", (24, 20), [((0, 0, 0), (27, 23, 0)), ((0, 0, 0), (31, 17, 0))], 12),
    ("high_corner2d", (24, 20), [((20, 0, 0), (47, 39, 0)), ((64, 48, 0), (95, 79, 0))], 16),
    ("corner3d", (12, 12, 12), [((0, 0, 0), (11, 15, 7))], 8),
], ids=["corner2d", "high_corner2d", "corner3d"])
def test_ghost_cells_of_boundary_regions(name, domain, regions, mgs, bc):
    """Ghost cells of boxes at walls, outflow sides and corners: copies and interpolated cells mirrored through one
    or more sides with their signs, to the bit."""
    dim = len(domain)
    lo_bc, hi_bc = WALLS[bc]
    if name == "corner2d" and bc == "noslip_periodic":
        regions = regions[:1]  # the second region's wrapped ghost cells would not be nested in the first
    phys, _, inputs, geom, _ = cases.advected_interface(n=16, dim=dim, physics=cb.SIXEQS)
    p = cb.make_parm(phys, dim, inputs)
    n = domain + (1,) * (3 - dim)
    g = cb.make_geom(n=n, dx=(0.1, 0.1, 0.1), lo_bc=lo_bc[:dim] + (0,) * (3 - dim), hi_bc=hi_bc[:dim] + (0,) * (3 - dim))
    boxes = amr.hierarchy(domain, dim, regions, mgs)
    N, ng = cb.parm_nstate(p), 3
    rng = np.random.default_rng(7)
    level = {}
    for lev in range(1 + len(regions)):
        shape = (N,) + tuple(domain[d] << lev for d in reversed(range(dim)))
        level[lev] = 1.0 + rng.random(shape) * np.where(rng.random(shape) < 0.5, 1.0, 1e-3)
    A = cb.Amr(p, g, boxes)

    def part(lo, hi, pad):
        return (slice(None),) + tuple(slice(lo[d], hi[d] + 1 + 2 * pad) for d in reversed(range(dim)))

    for b, (lev, lo, hi) in enumerate(boxes):
        U = np.full((N,) + tuple(hi[d] - lo[d] + 1 + 2 * ng for d in reversed(range(dim))), np.nan)
        U[(slice(None),) + (slice(ng, -ng),) * dim] = level[lev][part(lo, hi, 0)]
        A.upload(b, U if dim == 3 else U[:, None])
    for lev in range(1 + len(regions)):
        whole = level[lev].copy()
        if lev:
            whole = _lincc(below, lo_bc, hi_bc, 2, dim)
            for l, lo, hi in boxes:
                if l == lev:
                    whole[part(lo, hi, 0)] = level[lev][part(lo, hi, 0)]
        below = whole
        E = _extend(whole, ng, lo_bc, hi_bc, 2, dim)
        A.fill(lev)
        for b, (l, lo, hi) in enumerate(boxes):
            if l == lev:
                got = A.download(b)
                np.testing.assert_array_equal(got if dim == 3 else got[:, 0], E[part(lo, hi, ng)], err_msg=f"box {b} of level {lev}")
    A.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_region_at_a_slip_wall_equals_the_mirrored_domain(precision):
    """Three levels whose fine regions lie on a slip wall (and on the outflow side left of it): the run on the domain
    doubled by its mirror image, in which the wall is an inner symmetry line, gives the same state. Ghost cells,
    fluxes for the registers, refluxing and averaging at the wall are those of the interior (the two runs
    add the halves' terms in mirrored order, 2^-53 each; FP32 face values 2^-24 in the mixed form)."""
    n = (32, 16)
    phys, dim, inputs, geom, _ = cases.shock_bubble(nx=n[0], ny=n[1])
    inputs = dict(inputs, **{"compas_b200.precision": precision})
    p = cb.make_parm(phys, dim, inputs)
    A_, B_ = (1.0 / 0.4, 1.0 / 0.648), (0.0, 0.0)

    def state(lev, lo, hi, y_wall):
        """Cell-centre values of a flow symmetric about the height y_wall (in level-0 cells)."""
        h = 1.0 / (1 << lev)
        x = (np.arange(lo[0] - 3, hi[0] + 4) + 0.5)[None, :] * h
        y = (np.arange(lo[1] - 3, hi[1] + 4) + 0.5)[:, None] * h - y_wall
        bump = np.exp(-((x - 9.0) ** 2 + y ** 2) / 20.0)
        rho, a1 = 1.0 + 0.5 * bump + 0 * y, 0.2 + 0.6 * bump
        vel = [0.5 + 0.3 * bump, 0.4 * np.tanh(y / 6.0) * bump + 0 * x]
        U = cases._cons_from_prims(phys, dim, a1 * rho, (1 - a1) * 0.3 * rho, vel, 1.0 + 0.4 * bump, a1, A_, B_, np)
        return np.stack([np.broadcast_to(u, rho.shape) for u in U])[:, None]

    def run(ny, y_wall, lo_y, regions):
        g = cb.make_geom(n=(n[0], ny, 1), dx=(1.0 / 16, 1.0 / 16, 1.0), lo_bc=(2, lo_y, 0), hi_bc=(2, 4, 0))
        boxes = amr.hierarchy((n[0], ny), 2, regions, 16)
        H = cb.Amr(p, g, boxes)
        for b, (lev, lo, hi) in enumerate(boxes):
            H.upload(b, state(lev, lo, hi, y_wall))
        H.advance(4)
        assert H.sync().status == 0
        whole = {lev: np.full((6, ny << lev, n[0] << lev), np.nan) for lev in range(3)}
        for b, (lev, lo, hi) in enumerate(boxes):
            whole[lev][:, lo[1]:hi[1] + 1, lo[0]:hi[0] + 1] = _valid(H.download(b), lo, hi, 2)
        dts = H.dts(4)
        H.close()
        return whole, dts

    half, dts_h = run(n[1], 0.0, 4, [((0, 0, 0), (43, 15, 0)), ((0, 0, 0), (71, 15, 0))])
    full, dts_f = run(2 * n[1], float(n[1]), 4, [((0, 16, 0), (43, 47, 0)), ((0, 48, 0), (71, 79, 0))])
    tol = 1e-11 if precision == "fp64" else 1e-5
    np.testing.assert_allclose(dts_h, dts_f, rtol=tol)
    for lev in range(3):
        up = full[lev][:, n[1] << lev:]
        assert np.array_equal(np.isnan(up), np.isnan(half[lev]))
        for c in range(6):
            scale = np.nanmax(np.abs(up[c]))
            diff = np.nanmax(np.abs(up[c] - half[lev][c])) / scale
            print(f"{precision} level {lev} component {c}: {diff:.1e}")
            assert diff <= tol, (lev, c, diff)
