"""Batched shots: S independent shots on one mesh in one launch per step.

Each shot's arithmetic is the single-shot kernel's, so a batched run must give
the same bits as running the shots one at a time (seismograms and fields),
including a partial second tile of 32 shots, for the colour-pass,
owner-computes and fused tile kernels; shot 0 is also checked against
the CPU oracle (relative L2 <= 1e-5).
"""
import numpy as np
import pytest

from conftest import rel_l2, workload_case

pytestmark = pytest.mark.gpu


def shots(nshots, seed=3):
    from specfempp_b200 import meshgen
    rng = np.random.default_rng(seed)
    return [meshgen.RickerSource(float(rng.uniform(600, 3400)), float(rng.uniform(600, 2600)),
                                 float(rng.uniform(6.0, 14.0)), 1e10, shot=s) for s in range(nshots)]


def run(w, srcs, nshots, types=("displacement", "velocity"), variant=0):
    from specfempp_b200 import sfg
    sim = sfg.Simulation2D(w.mesh, dt=w.dt, nstep=w.nstep, nshots=nshots, kernel_variant=variant)
    sim.set_sources(srcs)
    sim.set_receivers(w.rec_x, w.rec_z, types=types)
    sim.initialize()
    sim.run(w.nstep)
    return sim


@pytest.mark.parametrize("nshots,variant", [(5, 1), (8, 1), (8, 3), (8, 4), (8, 5), (36, 1), (36, 3), (36, 4), (36, 5), (37, 3)])
def test_batched_equals_single_shots(sfg_lib, nshots, variant):
    from dataclasses import replace
    from specfempp_b200 import meshgen
    w = meshgen.elastic_psv_80x60(nstep=400)
    srcs = shots(nshots)
    batched = run(w, srcs, nshots, variant=variant)
    if variant == 5:
        assert batched.info().kernel_variant == 5
    seis_b = batched.seismograms()
    u_b = batched.field("elastic", "displacement")
    assert seis_b.shape[0] == nshots and u_b.shape[0] == nshots
    for s in sorted({0, 1, nshots // 2, nshots - 1}):
        single = run(w, [replace(srcs[s], shot=0)], 1)
        assert np.array_equal(seis_b[s], single.seismograms()[0]), s
        assert np.array_equal(u_b[s], single.field("elastic", "displacement")), s


def test_batched_shot_matches_oracle(sfg_lib, oracle_lib):
    from dataclasses import replace
    from oracle import runner
    from specfempp_b200 import meshgen
    w = meshgen.elastic_psv_80x60(nstep=700)
    srcs = shots(4, seed=7)
    sim = run(w, srcs, 4, types=("displacement",))
    seis = sim.seismograms()
    for s in (0, 3):
        case = workload_case(w)
        case.sources = [replace(srcs[s], shot=0)]
        ref = runner.run(case, "f32", nthreads=1)["seis"][:, 0]
        assert np.abs(ref).max() > 0
        assert rel_l2(seis[s, :, 0], ref) <= 1e-5, (s, rel_l2(seis[s, :, 0], ref))


def test_batched_handles_of_several_threads(sfg_lib):
    """Threads launch the thread form (variant 4) on handles of different shot
    counts, and so of different shared-memory needs, at the same time: no
    launch is refused (the limit is the function's, shared by all)."""
    import threading
    from specfempp_b200 import meshgen, sfg
    mesh = meshgen.structured_mesh(9, 7, 0.0, 900.0, 0.0, 700.0, np.zeros(7, np.int32),
                                   [(meshgen.ELASTIC, 2300.0, 3000.0, 1730.0)], absorbing=("bottom",))
    x, z = mesh.coorg[:, 0], mesh.coorg[:, 1]
    mesh.coorg = mesh.coorg + np.stack([0 * x, 9.0 * np.sin(x / 100.0) * z / 700.0], 1)
    f = 1.0 + 0.05 * np.random.default_rng(8).uniform(-1, 1, (3, mesh.nspec, 25)).astype(np.float32)
    pts = dict(zip(("point_rho", "point_vp", "point_vs"), (f.T * [2300.0, 3000.0, 1730.0]).T.astype(np.float32)))
    sims = []
    for shots in (2, 33) * 4:     # 57,600 and 3,600 bytes a block
        s = sfg.Simulation2D(mesh, dt=4e-4, nstep=10, nshots=shots, kernel_variant=4, **pts)
        s.set_sources([sfg.Source(x=400.0, z=300.0, f0=20.0, factor=1e10, shot=k) for k in range(shots)])
        s.set_receivers([500.0], [400.0])
        s.initialize()
        sims.append(s)
    errors = []

    def work(s):
        try:
            for _ in range(60):
                s.time_kernel(0, 300)
                s.time_kernel(0, 5, 16)
        except sfg.SfgError as e:
            errors.append(e)
    threads = [threading.Thread(target=work, args=(s,)) for s in sims]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]
