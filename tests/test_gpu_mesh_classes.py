"""The element kernels' specialisations and tilings at the sizes where they can
go wrong: one-value words an element (straight meshes, layered models) against
the general kernels bit for bit, partial blocks and tiles, shots that fill a
warp or not, a model whose class changes under captured step graphs, and 3D
tiles against the oracle.
"""
from dataclasses import replace

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

MATERIALS = {"psv": [(1, 2200.0, 2500.0, 1445.0), (1, 2400.0, 3000.0, 1700.0)],
             "acoustic": [(0, 1020.0, 1500.0, 0.0), (0, 1100.0, 1700.0, 0.0)]}
MATERIALS["sh"] = MATERIALS["poro"] = MATERIALS["psv"]


def grid(kind, nx, nz, relief):
    """An nx x nz mesh of 50 m elements in two layers, its nodes moved by `relief` m."""
    from specfempp_b200 import meshgen
    rows = (np.arange(nz) >= nz // 2).astype(np.int32)
    sides = () if kind == "poro" else ("bottom", "right", "left")
    m = meshgen.structured_mesh(nx, nz, 0.0, 50.0 * nx, 0.0, 50.0 * nz, rows, MATERIALS[kind], absorbing=sides,
                                free_surface=("top",))
    if kind == "poro":
        p = np.array([meshgen.POROUS_SANDSTONE] * 2)
        p[:, 10] = 1e-3
        p[1, 2] = 0.2
        m.mat_poro = p
        m.mat_rho = (1 - p[:, 2]) * p[:, 0] + p[:, 2] * p[:, 1]
    if relief:
        x, z = m.coorg[:, 0] / (50.0 * nx), m.coorg[:, 1] / (50.0 * nz)
        m.coorg = m.coorg + np.stack([np.zeros_like(x), relief * np.sin(5 * x + 1) * z], 1)
    return m


def simulate(mesh, kind, nstep, variant, epb=0, points=None, nshots=1, types=None):
    from specfempp_b200 import meshgen, sfg
    w, h = mesh.coorg.max(0)
    pts = points or {}
    sim = sfg.Simulation2D(mesh, dt=3e-4, nstep=nstep, nshots=nshots, elastic_wave="sh" if kind == "sh" else "psv",
                           kernel_variant=variant, elements_per_block=epb, **pts)
    sim.set_sources([meshgen.RickerSource(0.4 * w + 3 * s % 17, 0.55 * h, 40.0 + s, 1e10, angle=30.0 + s, shot=s)
                     for s in range(nshots)])
    sim.set_receivers([0.3 * w, 0.52 * w], [0.4 * h, 0.6 * h],
                      types=types or (("displacement", "pressure") if kind == "acoustic" else ("displacement", "velocity")))
    sim.initialize()
    sim.run(nstep)
    return sim


@pytest.mark.parametrize("nx,nz", [(3, 2), (33, 1), (16, 10), (13, 37)])
@pytest.mark.parametrize("kind,relief,varied", [
    (kind, relief, varied) for kind in ("psv", "sh", "acoustic", "poro") for relief in (0.0, 9.0)
    for varied in (False, True) if not (kind == "poro" and varied)])     # poroelastic: material constants only
def test_row_form_keeps_the_bits(sfg_lib, kind, nx, nz, relief, varied):
    """Row form (both block sizes) against the colour passes: every
    specialisation, blocks that the mesh fills partly."""
    mesh = grid(kind, nx, nz, relief)
    points = None
    if varied:
        f = 1.0 + 0.1 * np.random.default_rng(1).uniform(-1, 1, (mesh.nspec, 25)).astype(np.float32)
        base = [a[mesh.kmato][:, None].astype(np.float32) for a in (mesh.mat_rho, mesh.mat_vp, mesh.mat_vs)]
        points = dict(zip(("point_rho", "point_vp", "point_vs"), (b * f for b in base)))
    ref = simulate(mesh, kind, 60, 1, 16, points)
    a, med = ref.seismograms(), "acoustic" if kind == "acoustic" else "elastic"
    u = ref.field(med)
    assert np.abs(a).max() > 0
    for epb in (16, 32):
        sim = simulate(mesh, kind, 60, 6, epb, points)
        assert sim.info().kernel_variant == 6
        assert np.array_equal(sim.seismograms(), a)
        assert np.array_equal(sim.field(med), u)


@pytest.mark.parametrize("kind,shots", [("psv", 1), ("sh", 1), ("acoustic", 1), ("poro", 1), ("psv", 6), ("sh", 6)])
def test_one_tilted_element_among_rectangles(sfg_lib, kind, shots):
    """A mesh of rectangles whose corner node is moved by 2% of an element:
    the element there is no rectangle, so the mesh takes the general kernels
    (row form, or thread form of batched shots), and the bits are the colour
    passes' and not those of the straight mesh."""
    mesh = grid(kind, 17, 9, 0.0)
    flat = simulate(mesh, kind, 400, 1, 16, nshots=shots)
    corner = np.argmin(mesh.coorg.sum(1))
    mesh.coorg = mesh.coorg.copy()
    mesh.coorg[corner] += 1.0
    ref, sim = (simulate(mesh, kind, 400, v, 16, nshots=shots) for v in (1, 6 if shots == 1 else 4))
    med = "acoustic" if kind == "acoustic" else "elastic"
    assert sim.info().kernel_variant == (6 if shots == 1 else 4)
    assert np.array_equal(sim.seismograms(), ref.seismograms())
    assert np.array_equal(sim.field(med), ref.field(med))
    assert not np.array_equal(ref.field(med), flat.field(med))


def test_model_class_change_under_captured_graphs(sfg_lib):
    """A layered model replaced by one that varies inside the elements, and
    back: each run equals a fresh handle's, bit for bit."""
    from specfempp_b200 import adjoint
    mesh = grid("psv", 21, 14, 0.0)
    const = [a[mesh.kmato][:, None] * np.ones((1, 25)) for a in (mesh.mat_rho, mesh.mat_vp, mesh.mat_vs)]
    bump = 1.0 + 0.05 * np.random.default_rng(2).uniform(-1, 1, (mesh.nspec, 25))
    models = []
    for f in (1.0, bump):
        rho, vp, vs = (c * f for c in const)
        kappa, mu = adjoint.moduli(rho, vp, vs)
        models.append([x.astype(np.float32) for x in (rho, kappa, mu)])
    sim = simulate(mesh, "psv", 80, 6, 32)

    def run(s, model):
        s.set_model(*model)
        s.reset()
        s.run(80)
        return s.seismograms(), s.field("elastic")

    for model in (models[1], models[0], models[1]):
        got = run(sim, model)
        want = run(simulate(mesh, "psv", 80, 1, 16), model)
        assert all(np.array_equal(x, y) for x, y in zip(got, want))
    row = np.zeros((1, 2, 2, 2), np.float32)      # the streamed step's graph follows the model too
    sim.reset()
    sim.step_io(None, row)
    sim.set_model(*models[0])
    sim.reset()
    for _ in range(80):
        sim.step_io(None, row)
    assert np.array_equal(sim.seismograms(), run(simulate(mesh, "psv", 80, 3, 8), models[0])[0])


def test_model_change_waits_for_the_run_in_flight(sfg_lib):
    """sfg_run returns before the device is done; a model set at once does not
    touch that run's steps."""
    from specfempp_b200 import adjoint
    mesh = grid("psv", 60, 50, 0.0)
    rho, vp, vs = (a[mesh.kmato][:, None] * np.ones((1, 25)) for a in (mesh.mat_rho, mesh.mat_vp, mesh.mat_vs))
    other = [m.astype(np.float32) for m in (1.2 * rho, *adjoint.moduli(1.2 * rho, 0.9 * vp, 0.9 * vs))]
    ref = simulate(mesh, "psv", 3000, 6, 32)
    want = ref.seismograms(), ref.field("elastic")
    sim = simulate(mesh, "psv", 3000, 6, 32)
    sim.reset()
    sim.run(3000)
    sim.set_model(*other)
    assert np.abs(want[0]).max() > 0
    assert np.array_equal(sim.seismograms(), want[0]) and np.array_equal(sim.field("elastic"), want[1])


@pytest.mark.parametrize("kind", ["psv", "sh"])
@pytest.mark.parametrize("nshots", [2, 3, 6, 16, 20, 33])
@pytest.mark.parametrize("relief,varied", [(0.0, False), (7.0, True), (0.0, True)])
def test_batched_thread_form_keeps_the_bits(sfg_lib, kind, nshots, relief, varied):
    """One thread per element and shot (batched variant 4): shots that fill a
    part of a warp's lanes, one more than 32, elements that fill a block
    partly, against the colour passes."""
    mesh = grid(kind, 19, 11, relief)
    points = None
    if varied:
        f = 1.0 + 0.1 * np.random.default_rng(3).uniform(-1, 1, (mesh.nspec, 25)).astype(np.float32)
        base = [a[mesh.kmato][:, None].astype(np.float32) for a in (mesh.mat_rho, mesh.mat_vp, mesh.mat_vs)]
        points = dict(zip(("point_rho", "point_vp", "point_vs"), (b * f for b in base)))
    ref = simulate(mesh, kind, 50, 1, 0, points, nshots)
    sim = simulate(mesh, kind, 50, 4, 0, points, nshots)
    assert sim.info().kernel_variant == 4
    assert np.abs(ref.seismograms()).max() > 0
    assert np.array_equal(sim.seismograms(), ref.seismograms())
    assert np.array_equal(sim.field("elastic"), ref.field("elastic"))


@pytest.mark.parametrize("relief,varied", [(0.0, False), (0.0, True), (8.0, True)])
def test_reverse_row_form_keeps_the_bits(sfg_lib, relief, varied):
    """The reverse row kernel's specialisations against the point form, with
    Stacey edges and a partial last block."""
    from specfempp_b200 import adjoint
    mesh = grid("psv", 19, 13, relief)
    f = 1.0 + (0.05 * np.random.default_rng(4).uniform(-1, 1, (mesh.nspec, 25)) if varied else 0.0)
    rho, vp, vs = (a[mesh.kmato][:, None] * np.ones((1, 25)) * f for a in (mesh.mat_rho, mesh.mat_vp, mesh.mat_vs))
    kappa, mu = adjoint.moduli(rho, vp, vs)
    weights = np.random.default_rng(5).standard_normal((90, 2, 2)).astype(np.float32)
    out = []
    for v in (3, 6):
        sim = simulate(mesh, "psv", 90, v, 16, types=("displacement",))
        sim.set_model(*(x.astype(np.float32) for x in (rho, kappa, mu)))
        sim.forward_checkpointed(90, 40)
        out.append(sim.adjoint_gradient(weights))
    for x, y in zip(*out):
        assert np.abs(x).max() > 0 and np.array_equal(x, y)


def test_3d_one_deformed_element_among_boxes(sfg_lib, oracle_lib):
    """A mesh of boxes whose corner node is moved by 10%: the whole mesh takes
    the general metric, within 1e-5 of the oracle FP32 (the straight mesh's
    field is not)."""
    from oracle import runner3d
    from specfempp_b200 import meshgen, sfg3d
    fields = []
    for moved in (False, True):
        mesh = meshgen.homogeneous_hex_mesh(5, 3, 2, (0, 300.0, 0, 180.0, -120.0, 0), 2300.0, 3000.0, 1700.0,
                                            absorbing=(1, 0, 1, 1, 1, 0))
        if moved:
            mesh.nodes = mesh.nodes.copy()
            mesh.nodes.reshape(-1, 3)[0] += (6.0, -4.0, 5.0)
        src = [runner3d.Source3D(35.0, 30.0, -90.0, f0=45.0, factor=1e10, comp=(0.2, 1.0, -0.6, 0, 0, 0))]
        rec = np.array([[70.0, 60.0, -60.0]])
        sim = sfg3d.Simulation3D(mesh, dt=3e-4, nstep=150)
        sim.set_sources(src)
        sim.set_receivers(rec)
        sim.initialize()
        sim.run(150)
        fields.append(sim.field())
    ref = runner3d.run(runner3d.Case3D(mesh, src, rec, 3e-4, 150, ["displacement"]), "f32", nthreads=4,
                       want_final=True)["final"]
    assert rel_l2(fields[1], ref) <= 1e-5
    assert rel_l2(fields[0], ref) > 1e-3


@pytest.mark.parametrize("shape", [(1, 1, 1), (4, 2, 1), (5, 3, 2), (3, 5, 4), (9, 4, 3)])
@pytest.mark.parametrize("relief", [0.0, 12.0])
def test_3d_tiles_against_the_oracle(sfg_lib, oracle_lib, shape, relief):
    """Boxes and deformed hexahedra; tiles that the mesh fills partly, one or
    several tiles and marches.  Fields within 1e-5 of the oracle FP32, and the
    same bits for every number of layers a block marches and for a run in
    pieces."""
    from oracle import runner3d
    from specfempp_b200 import meshgen, sfg3d
    nx, ny, nz = shape
    mesh = meshgen.homogeneous_hex_mesh(nx, ny, nz, (0, 60.0 * nx, 0, 50.0 * ny, -55.0 * nz, 0), 2300.0, 3000.0, 1700.0,
                                        absorbing=(1, 0, 1, 1, 1, 0))
    rng = np.random.default_rng(6)
    f = 1.0 + 0.05 * rng.uniform(-1, 1, mesh.vp.shape)
    mesh.rho, mesh.vp, mesh.vs = mesh.rho * f, mesh.vp * f, mesh.vs * f
    if relief:
        mesh.nodes = mesh.nodes + rng.uniform(-relief, relief, mesh.nodes.shape) * 0.4
    W, D, H = 60.0 * nx, 50.0 * ny, 55.0 * nz
    src = [runner3d.Source3D(0.45 * W, 0.55 * D, -0.45 * H, f0=45.0, factor=1e12, kind="moment_tensor",
                             comp=(1.0, -0.5, 0.8, 0.3, 0.2, -0.4)),
           runner3d.Source3D(0.6 * W, 0.4 * D, -0.6 * H, f0=40.0, factor=1e10, comp=(0.2, 1.0, -0.6, 0, 0, 0))]
    rec = np.array([[0.3 * W, 0.3 * D, -0.35 * H], [0.7 * W, 0.6 * D, -0.65 * H], [0.52 * W, 0.47 * D, -0.2 * H]])
    types, nstep, dt = ["displacement", "velocity"], 140, 3e-4
    ref = runner3d.run(runner3d.Case3D(mesh, src, rec, dt, nstep, types), "f32", nthreads=4, want_final=True)
    first = None
    for layers in (1, 2, 8, 0):
        sim = sfg3d.Simulation3D(mesh, dt=dt, nstep=nstep, elements_per_block=layers)
        sim.set_sources(src)
        sim.set_receivers(rec, types=types)
        sim.initialize()
        sim.run(nstep if layers else 33)
        if not layers:
            sim.run(nstep - 33)
        got = (sim.seismograms(), sim.field("displacement"), sim.field("velocity"))
        assert sim.check_finite()
        first = first or got
        assert all(np.array_equal(a, b) for a, b in zip(first, got)), layers
    assert np.abs(ref["final"]).max() > 0
    assert rel_l2(first[1], ref["final"]) <= 1e-5
    for t in range(2):
        assert rel_l2(first[0][:, t], ref["seis"][:, t]) <= 1e-5


@pytest.mark.parametrize("kind", ["psv", "sh", "acoustic", "poro"])
def test_timed_point_updates_run_one_after_another(sfg_lib, kind):
    """sfg_time_kernel repeats the point update, which reads the fields that
    the update before it wrote: the state afterwards, and a step from it, are
    the same bits for every form of the step (4, which has no chained
    launches, where the medium has it)."""
    med, which = ("acoustic", 2) if kind == "acoustic" else ("elastic", 1)
    fields = []
    for v in ((3, 6) if kind == "poro" else (4, 3, 6)):
        sim = simulate(grid(kind, 45, 31, 0.0), kind, 60, v, 16)
        assert sim.info().kernel_variant == v
        assert sim.time_kernel(which, 20) > 0
        sim.run(1)
        fields.append((sim.field(med), sim.field(med, "velocity")))
    assert np.abs(fields[0][0]).max() > 0
    for f in fields[1:]:
        assert np.array_equal(f[0], fields[0][0]) and np.array_equal(f[1], fields[0][1])
