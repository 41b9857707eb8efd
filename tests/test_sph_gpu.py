"""GPU parity of the SPH solver (SPHSimulator over mpm_sph_*) against the
CPU restatement oracle/sph_oracle.c, bit for bit: particle records (position,
velocity, force, density, near density) and posvel."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import assert_bits_equal

pytestmark = pytest.mark.gpu


def run_pair(pkg, oracle_mod, half, n, frames, seed=7, box_changes=None, warp_max=-1):
    sim = pkg.SPHSimulator(None, None, 0.08, maxParticles=200000, seed=seed)
    sim.warpPerParticle = warp_max
    sim.reset(n, half)
    rec = sim.downloadParticles()
    assert len(rec) == n
    real = list(half)
    for f in range(frames):
        if box_changes and f in box_changes:
            real = box_changes[f]
            sim.changeBoxSize(real)
        sim.execute()
        rec, pv = oracle_mod.sph_execute(rec, real, 2)
    got = sim.downloadParticles()
    assert_bits_equal(got, rec, f"records after {frames} frames")
    assert_bits_equal(sim.downloadPosvel(), pv, "posvel")
    sim.close()
    return got


@pytest.mark.parametrize("warp_max", [-1, 0])
def test_default_scene(cuda, pkg, oracle_mod, warp_max):
    """main.ts's SPH defaults: 20,000 particles, half box (1.0, 2.0, 1.0);
    density and forces one warp per particle (the default at this size) and
    one thread per particle."""
    got = run_pair(pkg, oracle_mod, [1.0, 2.0, 1.0], 20000, 30, warp_max=warp_max)
    assert np.isfinite(got).all()
    assert (got[:, 11] > 0).all()  # every particle has neighbours in the grid


def test_warp_per_particle_dense_neighbourhoods(cuda, pkg, oracle_mod):
    """A compressed block (more neighbours than one staging round of 64)
    one warp per particle, and the knob's range."""
    run_pair(pkg, oracle_mod, [0.35, 1.0, 0.35], 20000, 8)
    sim = pkg.SPHSimulator(None, None, 0.08, maxParticles=1000)
    assert sim.warpPerParticle == 32768
    sim.warpPerParticle = 0
    assert sim.warpPerParticle == 0
    with pytest.raises(Exception):
        sim.warpPerParticle = -2
    sim.close()


@pytest.mark.parametrize("n,half", [(10000, [0.7, 2.0, 0.7]), (1, [1.0, 2.0, 1.0]),
                                    (63, [1.0, 2.0, 1.0])])
def test_ragged_counts(cuda, pkg, oracle_mod, n, half):
    run_pair(pkg, oracle_mod, half, n, 10)


def test_change_box_size(cuda, pkg, oracle_mod):
    run_pair(pkg, oracle_mod, [1.0, 2.0, 1.0], 20000, 24,
             box_changes={8: [0.8, 2.0, 1.0], 16: [1.2, 1.5, 0.9]})


def test_particles_outside_the_grid(cuda, pkg, oracle_mod):
    """Out-of-domain particles (flat id outside the grid, or aliasing into
    it) follow the documented rule in both implementations."""
    recs = pkg.sph_scene_dambreak([1.0, 2.0, 1.0], 5000, 3)
    extra = np.zeros((6, 16), np.float32)
    extra[:, 0:3] = [[0.0, -3.0, 0.0], [5.0, 0.0, 0.0], [-2.2, 0.1, 0.1],
                     [0.0, 2.3, 0.0], [np.nan, 0.0, 0.0], [1e30, -1e30, 0.0]]
    recs = np.concatenate([recs, extra])
    sim = pkg.SPHSimulator(None, None, 0.08, maxParticles=10000)
    sim.upload(recs, [1.0, 2.0, 1.0])
    ref = recs.copy()
    for _ in range(5):
        sim.execute()
        ref, pv = oracle_mod.sph_execute(ref, [1.0, 2.0, 1.0], 2)
    assert_bits_equal(sim.downloadParticles(), ref, "records")
    sim.close()


@pytest.mark.parametrize("n,spacing,warp_max", [
    (12000, 0.035, -1), (12001, 0.035, -1),      # 16 / 8 lanes per particle
    (22000, 0.035, -1), (22001, 0.035, -1),      # 8 lanes / a thread for the forces
    (130000, 0.035, -1), (130001, 0.035, -1),    # 8 lanes / a thread for the densities
    (5000, 0.02, -1), (20000, 0.02, -1),         # more neighbours (180) than a list holds
    (20000, 0.02, 0), (130001, 0.02, -1),
])
def test_density_and_force_variants(cuda, pkg, oracle_mod, n, spacing, warp_max):
    """Either side of each change of kernel, and lists that overflow in each:
    a moving block at rest spacing or compressed, some particles at one place
    (distance 0) and some at rest relative to each other, two substeps."""
    rng = np.random.default_rng(n)
    a = int(np.ceil(n ** (1.0 / 3.0)))
    i = np.arange(n)
    rec = np.zeros((n, 16), np.float32)
    rec[:, 0:3] = (np.stack([i % a, (i // a) % a, i // (a * a)], axis=1) - 0.5 * a) * spacing
    rec[:, 0:3] += 0.2 * spacing * rng.random((n, 3))
    rec[:, 4:7] = rng.normal(0.0, 0.3, (n, 3))
    rec[1:20, 0:3] = rec[0, 0:3]
    rec[100:200, 4:7] = 0.0
    half = [2.0, 2.0, 2.0]
    sim = pkg.SPHSimulator(None, None, 0.08, maxParticles=n)
    sim.warpPerParticle = warp_max
    sim.upload(rec, half)
    sim.execute()
    want, pv = oracle_mod.sph_execute(rec, half, 2)
    assert_bits_equal(sim.downloadParticles(), want, "records")
    assert_bits_equal(sim.downloadPosvel(), pv, "posvel")
    sim.close()


@pytest.mark.parametrize("n", [3000, 25000])
def test_capacity_without_neighbour_lists(cuda, pkg, oracle_mod, n):
    """A capacity too large for neighbour lists: the forces walk the rows."""
    recs = pkg.sph_scene_dambreak([1.0, 2.0, 1.0], n, 3)
    sim = pkg.SPHSimulator(None, None, 0.08, maxParticles=(1 << 23) + 1)
    sim.upload(recs, [1.0, 2.0, 1.0])
    sim.execute()
    want, _ = oracle_mod.sph_execute(recs, [1.0, 2.0, 1.0], 2)
    assert_bits_equal(sim.downloadParticles(), want, "records")
    sim.close()


def test_quotients_outside_the_fast_range(cuda, pkg, oracle_mod):
    """Neighbours whose force terms leave the range of the shared-reciprocal
    quotients (tiny and huge velocities, infinities, NaN, near-coincident
    particles) get the divisions' results."""
    recs = pkg.sph_scene_dambreak([1.0, 2.0, 1.0], 4000, 5)
    rng = np.random.default_rng(4)
    recs[:, 4:7] = rng.normal(0.0, 1.0, (len(recs), 3)) * 10.0 ** rng.integers(-38, 39, (len(recs), 1))
    recs[7, 4], recs[99, 5], recs[500, 6] = np.inf, -np.inf, np.nan
    recs[1000:1010, 0:3] = recs[1000, 0:3] + np.float32(1e-30)
    recs[2000:2010, 0] = np.nextafter(recs[2000, 0], np.float32(9), dtype=np.float32)
    recs[2000:2010, 1:3] = recs[2000, 1:3]
    sim = pkg.SPHSimulator(None, None, 0.08, maxParticles=4000)
    for warp_max in (-1, 0):
        sim.warpPerParticle = warp_max
        sim.upload(recs, [1.0, 2.0, 1.0])
        sim.execute(substeps=1)
        want, _ = oracle_mod.sph_execute(recs, [1.0, 2.0, 1.0], 1)
        got = sim.downloadParticles()
        nan = np.isnan(want)
        assert np.array_equal(nan, np.isnan(got))
        assert_bits_equal(np.where(nan, 0, got), np.where(nan, 0, want), "records")
    sim.close()


def test_posvel_feeds_the_renderer(cuda, pkg):
    import math
    sim = pkg.SPHSimulator(None, None, 0.08)
    sim.reset(20000, [1.0, 2.0, 1.0])
    for _ in range(5):
        sim.execute()
    r = pkg.FluidRenderer(128, 96, radius=0.04, fov=45 * math.pi / 180)
    u = pkg.camera_uniforms(128, 96, 3.0, [0.0, -1.5, 0.0], 45 * math.pi / 180, 0.08)
    r.execute(sim.posvelDevicePtr(), sim.numParticles, u)
    assert (r.download("depth") != 0).any()
    r.close()
    sim.close()


def test_graph_replay_equals_launches(cuda, pkg):
    """Frames replayed as CUDA graphs give the same records as launching every
    kernel, box changes between frames included."""
    outs = []
    for graph in (True, False):
        sim = pkg.SPHSimulator(None, None, 0.08, maxParticles=50000, seed=3)
        sim.setGraph(graph)
        sim.reset(12000, [1.0, 2.0, 1.0])
        for f in range(12):
            if f == 5:
                sim.changeBoxSize([0.8, 2.0, 1.0])
            sim.execute()
        outs.append(sim.downloadParticles())
        sim.close()
    assert_bits_equal(outs[0], outs[1], "graph vs launches")


@pytest.mark.parametrize("name", ["sph_dambreak", "sph_walls"])
def test_sph_solver_reproduces_wgsl_golden(cuda, pkg, name):
    """The CUDA SPH solver against the reference's SPH shaders run by the
    WGSL interpreter (tests/golden/make_golden_sph.py), one substep at a time
    with the fixture's real box: every record and posvel bit for bit."""
    import os
    here = os.path.dirname(os.path.abspath(__file__))
    f = dict(np.load(os.path.join(here, "golden", f"{name}.npz")))
    recs = f["records"]
    sim = pkg.SPHSimulator(None, None, 0.08, maxParticles=len(recs))
    sim.upload(recs, [float(x) for x in f["real_halves"][0]])
    for s in range(int(f["substeps"])):
        sim.changeBoxSize([float(x) for x in f["real_halves"][s]])
        sim.execute(substeps=1)
        assert_bits_equal(sim.downloadParticles(), f[f"s{s}_particles"], f"{name} substep {s}")
        assert_bits_equal(sim.downloadPosvel(), f[f"s{s}_posvel"], f"{name} substep {s} posvel")
    sim.close()


def test_frames_on_a_side_stream_after_an_upload(cuda, pkg, oracle_mod):
    """A frame on a stream of the caller's own finds the upload done: the
    records of particles outside the grid, which the frame's first kernel
    writes, are not overwritten by what the upload clears."""
    recs = pkg.sph_scene_dambreak([1.0, 2.0, 1.0], 30000, 3)
    recs[::7, 1] = -3.0
    recs[::7, 4:7] = 0.25
    sim = pkg.SPHSimulator(None, None, 0.08, maxParticles=len(recs))
    stream = cuda.cuda.Stream()
    want, pv = oracle_mod.sph_execute(recs, [1.0, 2.0, 1.0], 2)
    for _ in range(10):
        sim.upload(recs, [1.0, 2.0, 1.0])
        sim.execute(stream)
        assert_bits_equal(sim.downloadParticles(), want, "records")
        assert_bits_equal(sim.downloadPosvel(), pv, "posvel")
    sim.close()


@pytest.mark.parametrize("capacity", [5000, (1 << 23) + 1])  # with neighbour lists, without
@pytest.mark.parametrize("n", [1, 31, 33, 127, 129, 5000])
def test_a_thread_per_particle(cuda, pkg, oracle_mod, n, capacity):
    """The one-thread kernels at counts around their warps and blocks: a fall
    of ten frames, some particles outside the grid or aliasing into it."""
    recs = pkg.sph_scene_dambreak([0.5, 2.0, 0.5], n, 3)
    odd = np.array([[0.0, -3.0, 0.0], [5.0, 0.0, 0.0], [-2.2, 0.1, 0.1], [0.0, 2.3, 0.0],
                    [np.nan, 0.0, 0.0], [1e30, -1e30, 0.0]], np.float32)
    m = min(len(odd), n // 5)
    recs[:m, 0:3] = odd[:m]
    sim = pkg.SPHSimulator(None, None, 0.08, maxParticles=capacity)
    sim.warpPerParticle = 0
    sim.upload(recs, [0.5, 2.0, 0.5])
    for _ in range(10):
        sim.execute()
        recs, pv = oracle_mod.sph_execute(recs, [0.5, 2.0, 0.5], 2)
    assert_bits_equal(sim.downloadParticles(), recs, "records")
    sim.close()
