"""The library's host side over a CUDA runtime that runs no kernels
(fake_cudart.cpp): what it launches, what it waits for, and what it does when
memory is short.  On CPU."""
from __future__ import annotations

import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SIDE_STREAM = 0x1000  # a stream of the caller's own, as a handle


@pytest.fixture(scope="session")
def fake_lib(pkg, tmp_path_factory):
    """Path of the library with the fake runtime."""
    nvcc = shutil.which(pkg.build.nvcc())
    objects = [os.path.join(pkg.build.BUILD, src.replace(".cu", ".o")) for src in pkg.build.SOURCES]
    if not (nvcc and shutil.which("g++")):
        pytest.skip("no host toolchain")
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    out = str(tmp_path_factory.mktemp("fake") / "libmpm_fake.so")
    subprocess.check_call(["g++", "-shared", "-fPIC", "-std=c++17", "-O1", "-I" + cuda, "-Wl,-Bsymbolic",
                           "-Wl,-z,defs", "-o", out, os.path.join(HERE, "fake_cudart.cpp"), *objects])
    return out


@pytest.fixture
def fake(pkg, fake_lib, monkeypatch):
    """The package over that library; fake.fake_*: the runtime's own functions."""
    monkeypatch.setattr(pkg._lib, "_lib", None)
    monkeypatch.setattr(pkg.build, "build", lambda *a, **k: fake_lib)
    lib = pkg._lib.load()
    lib.fake_reset.argtypes = lib.fake_room.argtypes = [ctypes.c_size_t]
    lib.fake_used.restype = ctypes.c_size_t
    lib.fake_launched.restype = ctypes.c_char_p
    lib.fake_reset(-1)
    return lib


def test_sph_upload_is_done_when_it_returns(fake, pkg):
    """A frame on the caller's own stream does not wait for the null stream, so
    the upload's copies and memsets have to be done when it returns."""
    sim = pkg.SPHSimulator(None, None, 0.08, maxParticles=100)
    recs = np.zeros((100, 16), np.float32)
    for graph in (False, True):
        sim.setGraph(graph)
        sim.upload(recs, [1.0, 2.0, 1.0])
        sim.execute(SIDE_STREAM)
        sim.reset(100, [1.0, 2.0, 1.0])
        sim.execute(SIDE_STREAM)
    assert b"k_sph_force" in fake.fake_launched()
    assert fake.fake_unordered() == 0
    sim.close()


def test_sph_without_room_for_neighbour_lists(fake, pkg):
    """2^23 particles, the most with neighbour lists: 4.3 GB of them beside 1.5
    GB.  Where they do not fit the simulator works without; where the rest does
    not fit either, creating it fails and leaves nothing behind."""
    cap = 1 << 23
    sim = pkg.SPHSimulator(None, None, 0.08, maxParticles=cap)
    assert fake.fake_used() > 512 * cap
    sim.close()
    assert fake.fake_used() == 0
    fake.fake_reset(2 << 30)
    sim = pkg.SPHSimulator(None, None, 0.08, maxParticles=cap)
    assert fake.fake_used() < 2 << 30
    sim.upload(np.zeros((1000, 16), np.float32), [1.0, 2.0, 1.0])
    sim.execute()
    assert b"k_sph_force" in fake.fake_launched()
    sim.close()
    fake.fake_reset(1 << 30)
    with pytest.raises(pkg.MPMError):
        pkg.SPHSimulator(None, None, 0.08, maxParticles=cap)
    assert fake.fake_used() == 0


@pytest.mark.parametrize("n,warp_max,density,force", [
    (12000, -1, 16, 16), (12001, -1, 8, 8), (22000, -1, 8, 8), (22001, -1, 8, 1),
    (130000, -1, 8, 1), (130001, -1, 1, 1),
    (1, 0, 1, 1), (12000, 0, 1, 1), (100000, 0, 1, 1),          # 0: always a thread
    (500, 500, 16, 16), (501, 500, 1, 1),                       # the caller's own limit
    (30000, 32767, 8, 8), (30000, 32768, 8, 1), (30000, 29999, 1, 1), (140000, 200000, 8, 8),
])
def test_sph_lanes_per_particle(fake, pkg, n, warp_max, density, force):
    """Which kernels run: the fastest at a particle count, or the ones that the
    caller's limit asks for, of the densities and of the forces."""
    sim = pkg.SPHSimulator(None, None, 0.08, maxParticles=n)
    sim.setGraph(False)
    sim.upload(np.zeros((n, 16), np.float32), [1.0, 2.0, 1.0])
    sim.warpPerParticle = warp_max
    sim.execute(substeps=1)
    ran = fake.fake_launched().decode()
    for what, lanes in (("density", density), ("force", force)):
        name = f"k_sph_{what}_thread" if lanes == 1 else f"k_sph_{what}ILi{lanes}E"
        assert [k for k in ran.split() if f"k_sph_{what}" in k] == [k for k in ran.split() if name in k] != []
    sim.warpPerParticle = -1
    assert sim.warpPerParticle == 32768
    sim.close()


@pytest.mark.parametrize("box,chunk_sums,one_launch", [
    ((32, 32, 32), False, True),     # 514 bins
    ((124, 44, 48), False, True),    # 4,094
    ((64, 64, 64), False, False),    # 4,098
    ((80, 80, 80), False, False),    # 8,002: 32 chunks
    ((84, 80, 80), True, False),     # 8,402: 33 chunks
    ((128, 128, 128), True, False),  # 32,770: 129 chunks
])
def test_scan_launches(fake, pkg, box, chunk_sums, one_launch):
    """The counting sort's launches by the scene's bins, as measured."""
    sim = pkg.MLSMPMSimulator(None, None, maxParticles=100, maxGrid=box)
    sim.setGraph(False)
    sim.upload(np.full((100, 20), 5.0, np.float32), [float(b) for b in box])
    sim.execute()
    fake.fake_reset(-1)
    sim.execute()
    ran = fake.fake_launched().decode()
    assert ("k_chunk_sums" in ran) == chunk_sums
    assert ("k_scan_scatter" in ran) == one_launch
    sim.close()


def _scenes(pkg):
    return [pkg.scene_desc(40, [16.0, 12.0, 20.0]), pkg.scene_desc(24, [14.0, 14.0, 14.0])]


def _use_simulator(pkg):
    sim = pkg.MLSMPMSimulator(None, None, maxParticles=64, maxGrid=(16, 16, 16))
    recs = np.full((64, 20), 5.0, np.float32)
    for graph in (True, False):
        sim.setGraph(graph)
        sim.upload(recs, [16.0, 16.0, 16.0])
        sim.execute(SIDE_STREAM)
        sim.changeBoxSize([16.0, 16.0, 15.0])
        sim.execute(SIDE_STREAM)
    sim.close()


def _use_batch(pkg):
    recs = np.full((64, 20), 5.0, np.float32)
    batch = pkg.MLSMPMBatch(_scenes(pkg), recs)
    batch.step(2, SIDE_STREAM)
    batch.setScene(0, pkg.scene_desc(40, [16.0, 12.0, 20.0], stiffness=2.0))
    batch.step(2, SIDE_STREAM)
    batch.upload(recs)
    batch.step(2, SIDE_STREAM)
    rt = pkg._lib.load()
    stream, graph = ctypes.c_void_p(SIDE_STREAM), ctypes.c_void_p()
    rt.cudaStreamBeginCapture(stream, 0)
    batch.step(2, SIDE_STREAM)
    rt.cudaStreamEndCapture(stream, ctypes.byref(graph))
    for stiffness in (3.0, 4.0):
        rt.cudaGraphLaunch(graph, stream)
        batch.setScene(1, pkg.scene_desc(24, [14.0, 14.0, 14.0], stiffness=stiffness))
    rt.cudaGraphLaunch(graph, stream)
    batch.close()


def _use_adjoint(pkg, tape):
    recs = np.full((64, 20), 5.0, np.float32)
    adj = pkg.MLSMPMAdjoint(_scenes(pkg), 4, 2, tape=tape)
    for _ in range(2):
        adj.forward(recs, 4, SIDE_STREAM)
        adj.setObservations({4: np.zeros((64, 3), np.float32)})
        adj.observationLoss(SIDE_STREAM)
        adj.backwardObserved(SIDE_STREAM)
        adj.setScene(0, pkg.scene_desc(40, [16.0, 12.0, 20.0], stiffness=2.0))
    adj.forward(recs, 4, SIDE_STREAM)
    adj.backward({4: recs}, SIDE_STREAM)
    adj.close()


def _use_renderer(pkg):
    posvel = np.zeros((8, 8), np.float32)
    u = pkg.camera_uniforms(64, 48, 40.0, [10.0, 4.0, 12.0], 0.8, 1.2)
    r = pkg.FluidRenderer(64, 48, 0.6, 0.8)
    for spheres in (True, False):
        r.execute(posvel.ctypes.data, 8, u, SIDE_STREAM, sphereRenderFl=spheres)
    r.setEnvmap(np.ones((6, 4, 4, 4), np.float32))
    r.execute(posvel.ctypes.data, 8, u, SIDE_STREAM)
    r.close()


def _use_sph(pkg):
    sim = pkg.SPHSimulator(None, None, 0.08, maxParticles=1000)
    sim.upload(np.zeros((1000, 16), np.float32), [1.0, 2.0, 1.0])
    sim.execute(SIDE_STREAM)
    sim.close()


@pytest.mark.parametrize("use", [
    _use_simulator, _use_batch, lambda pkg: _use_adjoint(pkg, "fp64"), lambda pkg: _use_adjoint(pkg, "fixed"),
    _use_renderer], ids=["simulator", "batch", "adjoint fp64", "adjoint fixed", "renderer"])
def test_streams_and_uploads_in_order(fake, pkg, use):
    """Work on the caller's own stream finds what was uploaded before it, and
    an upload waits for the work in flight."""
    use(pkg)
    assert fake.fake_launched()
    assert fake.fake_unordered() == 0


def test_autotune_chooses_by_the_longer_timing(fake, pkg):
    """What is the fastest over one window of substeps need not be over five:
    every part of the choice is by the longer timing."""
    sim = pkg.MLSMPMSimulator(None, None, maxParticles=64, maxGrid=(16, 16, 16))
    sim.upload(np.full((64, 20), 5.0, np.float32), [16.0, 16.0, 16.0])
    timed = []

    @ctypes.CFUNCTYPE(ctypes.c_float, ctypes.c_int)
    def elapsed(windows):
        t = sim.tuning()
        ms = 10.0 + (t["task_threads"] != 256) + (t["task_size"] != 512) + (t["bin_pairing"] != 0)
        short, long = t["lane_table_min"] == 32, t["lane_table_min"] == 512
        timed.append(windows)
        return windows * ms - (0.5 if windows == 1 and short else 0.0) - (2.5 if windows > 1 and long else 0.0)

    fake.fake_elapsed(elapsed)
    assert sim.autotune(8) == 512
    assert sim.tuning() == {"bin_pairing": 0, "task_threads": 256, "task_size": 512, "lane_table_min": 512}
    assert set(timed) == {1, 5}
    sim.close()


@pytest.mark.parametrize("use", [
    _use_simulator, _use_batch, lambda pkg: _use_adjoint(pkg, "fp64"), lambda pkg: _use_adjoint(pkg, "fixed"),
    _use_renderer, _use_sph], ids=["simulator", "batch", "adjoint fp64", "adjoint fixed", "renderer", "sph"])
def test_a_failed_call_leaves_no_error_behind(fake, pkg, use):
    """Where memory runs out anywhere on the way, the call that fails says so,
    and the next ones, with memory again, do not fail for it."""
    failed = 0
    room = 1 << 10
    while room < 1 << 30:
        fake.fake_room(room)
        try:
            use(pkg)
        except pkg.MPMError:
            failed += 1
            fake.fake_room(1 << 40)
            use(pkg)
        room *= 2
    assert failed > 3
