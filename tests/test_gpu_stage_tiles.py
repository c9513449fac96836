"""The stage kernel's tile routine at the sizes where its work split can go wrong, against the C oracle.

Tiles are 16^2 (2D) and 8^3 (3D); lines are walked in segments, a ragged tile skips the lines outside the
box, and the second and third stage read ghost cells through the boundary conditions. The plain FP64 form
must give the oracle's bits for every launch shape; the mixed form must stay within its single-precision
reconstruction of it.
"""
import numpy as np
import pytest

import compas_b200 as cb
from compas_b200 import cases
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu

BCS = {"periodic": ((0, 0, 0), (0, 0, 0)), "walls": ((4, 3, 5), (3, 4, 4)), "outflow": ((2, 2, 2), (2, 2, 2)),
       "mixed": ((5, 0, 2), (2, 0, 4))}


def _case(model, n, bc, scheme, precision):
    """The model's flow cropped to n cells, with a random velocity, under the boundary codes of `bc`."""
    rng = np.random.default_rng(sum(n) + len(bc))
    m = max(max(n), 12)
    if model == "five2":
        phys, dim, inputs, geom, U = cases.shock_bubble(nx=m, ny=m, length=1.0, radius=0.2, center=(0.5, 0.5))
    elif model == "five3":
        phys, dim, inputs, geom, U = cases.advected_interface(n=m, dim=3, physics=cb.FIVEEQS)
    elif model == "six2":
        phys, dim, inputs, geom, U = cases.advected_interface(n=m, dim=2, physics=cb.SIXEQS)
    elif model == "six3":
        phys, dim, inputs, geom, U = cases.shock_droplet(n=m)
    else:
        phys, dim, inputs, geom, U = cases.nphase_bubbles(n=m, nphase=3, dim=3 if model == "nphase3" else 2)
    gz = 3 if dim == 3 else 0
    nz = n[2] if dim == 3 else 1
    V = U[:, gz:gz + nz, 3:3 + n[1], 3:3 + n[0]].copy()
    first = 3 if model.startswith("nphase") else 2
    rho = V[:first].sum(0)
    amp = {"five2": 0.1, "five3": 20.0, "six2": 20.0, "six3": 20.0, "nphase": 20.0,
           "nphase3": 50.0}[model]
    u = [amp * rng.standard_normal(rho.shape) for _ in range(dim)]
    work = sum(V[first + d] * u[d] + 0.5 * rho * u[d] ** 2 for d in range(dim))
    for d in range(dim):
        V[first + d] += rho * u[d]
    if phys == cb.SIXEQS:
        V[first + dim] += V[0] / rho * work
        V[first + dim + 1] += V[1] / rho * work
    else:
        V[first + dim] += work
    inputs = dict(inputs, **{"FiniteVolume.Scheme": scheme, "compas_b200.precision": precision})
    p = cb.make_parm(phys, dim, inputs)
    g = cb.make_geom(n=n, dx=geom["dx"], lo_bc=BCS[bc][0], hi_bc=BCS[bc][1])
    out = np.zeros(cb.padded_shape(p, g))
    cb.valid_view(out, p, g)[...] = V
    return p, g, out


def _advance(p, g, U, steps, shape=None, order=0):
    lv = cb.Level(p, g)
    if shape is not None:
        lv.set_kernel(shape, order)
    lv.upload(U)
    lv.advance(steps)
    info = lv.sync(check=False)
    out, dts = lv.download(), lv.dts(steps)
    lv.close()
    assert info.status == 0 and info.steps == steps
    return cb.valid_view(out, p, g), dts


SIZES2 = [(16, 16, 1), (17, 15, 1), (3, 33, 1), (47, 6, 1), (4, 4, 1)]
SIZES3 = [(8, 8, 8), (9, 7, 10), (17, 4, 5), (6, 16, 3)]


@pytest.mark.parametrize("scheme", ["WENO5", "WENO5B"])
@pytest.mark.parametrize("model,n,bc", [("five2", n, b) for n, b in zip(SIZES2, ["periodic", "walls", "outflow", "mixed", "walls"])] +
                         [("nphase", n, b) for n, b in zip(SIZES2, ["walls", "mixed", "walls", "outflow", "periodic"])] +
                         [("six2", n, b) for n, b in zip(SIZES2, ["walls", "periodic", "periodic", "walls", "outflow"])] +
                         [("five3", n, b) for n, b in zip(SIZES3, ["periodic", "walls", "mixed", "walls"])] +
                         [("six3", n, b) for n, b in zip(SIZES3, ["outflow", "walls", "mixed", "periodic"])])
def test_every_shape_gives_the_oracles_bits(model, n, bc, scheme):
    if model == "nphase" and scheme == "WENO5B":
        pytest.skip("the C oracle runs the N-phase model with WENO5")
    p, g, U = _case(model, n, bc, scheme, "fp64")
    ref = U.copy()
    _, dts_ref = Oracle("port", p, g).advance(ref, 2)
    ref = cb.valid_view(ref, p, g)
    assert np.all(np.isfinite(ref))
    for shape in range(3):
        got, dts = _advance(p, g, U, 2, shape, order=shape % 2)
        np.testing.assert_array_equal(dts, dts_ref)
        np.testing.assert_array_equal(got, ref, err_msg=f"shape {shape}")
    # the drop-in right-hand side takes its shape from the box size
    import torch

    Uf = U.copy()
    o = Oracle("port", p, g)
    o.fill_ghosts(Uf)
    dU_ref, cmax_ref = o.compute_dudt(Uf)
    dev = torch.from_numpy(Uf).cuda()
    dU, cm = torch.zeros_like(dev), torch.zeros(1, dtype=torch.float64, device="cuda")
    cb.compute_dUdt_FV(p, g, dev, dU, cmax=cm)
    assert float(cm.item()) == cmax_ref
    np.testing.assert_array_equal(cb.valid_view(dU.cpu().numpy(), p, g), cb.valid_view(dU_ref, p, g))
    # the mixed form of the two-phase models: masses within 1e-5 of the total mass field and the volume fraction
    # within 1e-5 of 1, the mixed form's stated bound (FP32 face values, 2^-24 each, over two steps). The N-phase
    # consistent limiter switches on slope sums that FP32 face values change, so random data has no such bound
    if model == "nphase":
        return
    pm, gm, _ = _case(model, n, bc, scheme, "mixed")
    mix, _ = _advance(pm, gm, U, 2)
    total = np.linalg.norm(ref[:2].sum(0))
    for c in range(2):
        assert np.linalg.norm(mix[c] - ref[c]) <= 1e-5 * total, c
    assert np.linalg.norm(mix[-1] - ref[-1]) <= 1e-5 * np.sqrt(ref[-1].size)


@pytest.mark.parametrize("scheme", ["WENO5", "WENO5B"])
@pytest.mark.parametrize("model,n,bc", [("five2", n, "mixed") for n in SIZES2] + [("nphase", n, "walls") for n in SIZES2] +
                         [("six2", n, "walls") for n in SIZES2] + [("five3", n, "mixed") for n in SIZES3] +
                         [("nphase3", n, "walls") for n in SIZES3] + [("six3", n, "outflow") for n in SIZES3])
def test_every_shape_gives_the_same_mixed_bits(model, n, bc, scheme):
    """The mixed form's launch shapes split lines into other segments and carry face values across their ends, but
    every face takes the same operations: the same bits, at the ragged and odd sizes."""
    p, g, U = _case(model, n, bc, scheme, "mixed")
    ref, dts_ref = _advance(p, g, U, 2, 0)
    assert np.all(np.isfinite(ref))
    for shape in (1, 2):
        got, dts = _advance(p, g, U, 2, shape, order=shape % 2)
        np.testing.assert_array_equal(dts, dts_ref)
        np.testing.assert_array_equal(got, ref, err_msg=f"shape {shape}")


@pytest.mark.parametrize("kind", ["ulps", "ulps_jump", "zero_runs", "wide"])
@pytest.mark.parametrize("scheme", ["WENO5", "WENO5B"])
def test_weno_quotients_are_the_divisions(kind, scheme):
    """Right-hand sides of fields whose smoothness indicators are hard to divide: differences of a few units in
    the last place (ratios of small whole numbers, next to a rounding boundary), whole stencils and halves of
    stencils without any difference, and indicators 60 decades apart. Bit for bit the oracle's, whose
    quotients are IEEE divisions."""
    import torch

    rng = np.random.default_rng({"ulps": 1, "ulps_jump": 2, "zero_runs": 3, "wide": 4}[kind])
    phys, dim, inputs, geom, _ = cases.shock_bubble(nx=64, ny=48, length=64 / 48)
    p = cb.make_parm(phys, dim, dict(inputs, **{"FiniteVolume.Scheme": scheme}))
    g = cb.make_geom(n=(64, 48, 1), dx=geom["dx"], lo_bc=(2, 4, 0), hi_bc=(2, 4, 0))
    U = np.zeros(cb.padded_shape(p, g))
    V = cb.valid_view(U, p, g)
    base = np.array([0.75, 0.25, 0.5, -0.25, 2.75, 0.75])[:, None, None, None] * np.ones_like(V)
    k = rng.integers(0, 9, V.shape).astype(float)
    if kind == "ulps":
        V[...] = base * (1.0 + k * 2.0 ** -52)
    elif kind == "ulps_jump":
        jump = np.where(np.arange(64)[None, None, None, :] % 11 < 5, 1.0, 3.0)
        V[...] = base * (1.0 + k * 2.0 ** -52)
        V[:2] *= jump
        V[4] *= jump[0] * 2.0
    elif kind == "zero_runs":
        V[...] = base * (1.0 + 1e-3 * np.floor(np.arange(64) / 4)[None, None, None, :] * (rng.random((6, 1, 48, 1)) < 0.5))
    else:
        V[...] = base * (1.0 + 10.0 ** rng.uniform(-15, -1, V.shape) * rng.choice([-1.0, 1.0], V.shape))
    V[5] = np.minimum(V[5], 1.0 - 1e-6)
    o = Oracle("port", p, g)
    o.fill_ghosts(U)
    dU_ref, cmax_ref = o.compute_dudt(U)
    dev = torch.from_numpy(U).cuda()
    dU, cm = torch.zeros_like(dev), torch.zeros(1, dtype=torch.float64, device="cuda")
    cb.compute_dUdt_FV(p, g, dev, dU, cmax=cm)
    assert float(cm.item()) == cmax_ref
    np.testing.assert_array_equal(cb.valid_view(dU.cpu().numpy(), p, g), cb.valid_view(dU_ref, p, g))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [(17, 9, 10), (49, 41, 50)])
def test_first_wave_speed_of_a_limited_3d_flow(n, precision):
    """The t = 0 wave-speed pass of the 3D N-phase model, whose flux pass reads the halo planes (the consistent
    limiter about the cells on either side of a face) and which keeps one direction's planes at a time: a box of
    few tiles (the large-CTA shape) and one that fills the GPU, as a level, in a batch and as a hierarchy's boxes.
    The first step's size is that of the largest face speed of compute_dUdt_FV, and in FP64 the C oracle's, every
    time; a warp that converted the next direction's planes early would change a neighbour's limited state."""
    import torch

    from compas_b200 import amr

    p, g, U = _case("nphase3", n, "periodic", "WENO5", precision)
    dev = torch.from_numpy(U.copy()).cuda()
    cb.FillPatch(p, g, dev)
    dU, cm = torch.zeros_like(dev), torch.zeros(1, dtype=torch.float64, device="cuda")
    cb.compute_dUdt_FV(p, g, dev, dU, cmax=cm)
    cm = float(cm.item())
    if precision == "fp64":
        Uf = U.copy()
        o = Oracle("port", p, g)
        o.fill_ghosts(Uf)
        assert cm == o.compute_dudt(Uf)[1]
    dt = min(p.cfl * g.dx[d] / cm for d in range(3))
    boxes = amr.hierarchy(n, 3, [], 28)
    A = cb.Amr(p, g, boxes)
    batch = cb.Batch(cb.FIVEEQS_NPHASE, 3, id_limiter=5, precision=1 if precision == "mixed" else 0, nphase=3)
    lv = cb.Level(p, g)
    lv.set_kernel(0, 0)
    for _ in range(20):
        lv.upload(U)
        lv.advance(1, use_graph=False)
        lv.sync()
        assert lv.dts(1)[0] == dt
        for b, (_, lo, hi) in enumerate(boxes):
            V = np.zeros((U.shape[0],) + tuple(hi[d] - lo[d] + 7 for d in (2, 1, 0)))
            V[:, 3:-3, 3:-3, 3:-3] = cb.valid_view(U, p, g)[:, lo[2]:hi[2] + 1, lo[1]:hi[1] + 1, lo[0]:hi[0] + 1]
            A.upload(b, V)
        cid = batch.add(p, g, U, max_steps=1)
        batch.advance(1)
        assert [i.t for i in batch.poll() if i.id == cid] == [dt]
        batch.remove(cid)
    A.advance(1)
    assert A.dts(1)[0] == dt
    for h in (A, batch, lv):
        h.close()


@pytest.mark.parametrize("scheme", ["WENO5", "MUSCL"])
def test_wave_speed_of_every_part_of_a_tile_counts(scheme):
    """One fast cell at places over a 16^2 tile, whose faces fall to different warps of the CTA, the partial last
    one of the 144-, 272- and 136-thread shapes among them: the second step's size, which the largest face speed
    of the first step's stages sets, is the same for every launch shape, and with WENO5 in FP64 the C oracle's."""
    rng = np.random.default_rng(5)
    phys, dim, inputs, geom, _ = cases.shock_bubble(nx=16, ny=16, length=1.0)
    for i, j in [(0, 0), (7, 0), (8, 5), (7, 8), (8, 15), (15, 15), (3, 8), (15, 2)]:
        V = np.empty((6, 1, 16, 16))
        rho, u = 1.0 + 0.1 * rng.random((1, 16, 16)), 0.1 * rng.standard_normal((2, 1, 16, 16))
        u[:, 0, j, i] += 2.0
        V[0], V[1], V[5] = 0.75 * rho, 0.25 * rho, 0.5
        V[2:4] = rho * u
        V[4] = 2.5 + 0.5 * rho * (u * u).sum(0)
        for precision in ("fp64", "mixed"):
            p = cb.make_parm(phys, dim, dict(inputs, **{"FiniteVolume.Scheme": scheme, "compas_b200.precision": precision}))
            g = cb.make_geom(n=(16, 16, 1), dx=geom["dx"], lo_bc=(2, 2, 0), hi_bc=(2, 2, 0))
            U = np.zeros(cb.padded_shape(p, g))
            cb.valid_view(U, p, g)[...] = V
            dts = [_advance(p, g, U, 2, shape)[1] for shape in range(3)]
            np.testing.assert_array_equal(dts[1], dts[0])
            np.testing.assert_array_equal(dts[2], dts[0])
            if precision == "fp64" and scheme == "WENO5":  # the C oracle has no MUSCL
                np.testing.assert_array_equal(dts[0], Oracle("port", p, g).advance(U.copy(), 2)[1])


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("riemann", ["LLF", "HLL", "HLLC"])
@pytest.mark.parametrize("model", ["five2", "six2", "five3", "six3", "nphase"])
def test_first_step_size_is_the_right_hand_sides_wave_speed(model, riemann, precision):
    """The t = 0 pass forms the face speeds without the fluxes: bit for bit those of the Riemann solver in use, for
    supersonic drifts (where a unit in the last place of |u| shows in c + |u|, in one of some dozen drifts)."""
    import torch

    rng = np.random.default_rng(11)
    n = (12, 9, 1) if model in ("five2", "six2", "nphase") else (9, 8, 5)
    p, g, U0 = _case(model, n, "periodic", "WENO5", precision)
    p.id_riemann = {"LLF": 0, "HLL": 1, "HLLC": 2}[riemann]
    lv = cb.Level(p, g)
    lv.set_kernel(0, 0)
    for _ in range(60):
        U = U0.copy()
        V = cb.valid_view(U, p, g)
        first = 3 if model == "nphase" else 2
        rho = V[:first].sum(0)
        drift = (6.0 if model == "five2" else 6000.0) * (1.0 + 0.3 * rng.random(3))
        work = sum(drift[d] * (V[first + d] + 0.5 * rho * drift[d]) for d in range(p.dim))
        for d in range(p.dim):
            V[first + d] += rho * drift[d]
        if p.physics == cb.SIXEQS:
            V[first + p.dim] += V[0] / rho * work
            V[first + p.dim + 1] += V[1] / rho * work
        else:
            V[first + p.dim] += work
        dev = torch.from_numpy(U).cuda()
        cb.FillPatch(p, g, dev)
        cm = torch.zeros(1, dtype=torch.float64, device="cuda")
        cb.compute_dUdt_FV(p, g, dev, torch.zeros_like(dev), cmax=cm)
        lv.upload(U)
        lv.advance(1, use_graph=False)
        assert lv.dts(1)[0] == min(p.cfl * g.dx[d] / float(cm.item()) for d in range(p.dim))
    lv.close()
