"""What the engine asks of the CUDA runtime, with a runtime of two devices in
host memory in its place (fake_cudart.cpp; kernels do not run)."""
import ctypes
import shutil
import subprocess

import numpy as np
import pytest

from courant_b200 import boards, build, scenes, serve
from courant_b200.api import Courant, CourantError, DebyeModel


class Fake:
    def __init__(self, path):
        self.lib = Courant(path)
        self.so = ctypes.CDLL(str(path))
        self.so.fake_count.restype = ctypes.c_long
        self.so.fake_fail_copy.argtypes = [ctypes.c_long]
        self.so.fake_elapsed.argtypes = [ctypes.c_float, ctypes.c_float]

    def count(self, what):
        return self.so.fake_count(what.encode())

    current = property(lambda self: self.so.fake_current(), lambda self, d: self.so.fake_set_current(d))


@pytest.fixture(scope="module")
def fake_path(tmp_path_factory):
    if build.needs_build():
        build.build()
    objs = [build.PKG / "_build" / (p.stem + (".cu.o" if p.suffix == ".cu" else ".o")) for p in build.sources()]
    if not all(o.exists() for o in objs):
        pytest.skip("the library's objects are not here")
    out = tmp_path_factory.mktemp("fake") / "libcourant_fake.so"
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-Wall", "-Wextra", f"-I{build.CUDA_LIB.parent / 'include'}",
                    str(build.PKG.parent / "tests" / "fake_cudart.cpp"), *map(str, objs), "-o", str(out), "-Wl,-Bsymbolic",
                    "-lpthread"], check=True)
    return out


@pytest.fixture(scope="module")
def fake(fake_path):
    return Fake(fake_path)


READS = {"field": lambda s: s.field(4), "spectrum": lambda s: s.portV(0), "checkpoint": lambda s: s.checkpoint(),
         "release": lambda s: s.releaseDevice(), "state": lambda s: s.c.ex.cem_state_array(s.h, 2, 0, 0)}


@pytest.mark.parametrize("read", READS)
def test_state_is_read_from_a_thread_on_another_device(fake, read):
    fake.current = 0
    s = scenes.lossy_scene(fake.lib)[0]
    s.prepareDevice(1)
    s.step(10)
    fake.current = 0
    before = fake.count("k_move")
    READS[read](s)
    assert fake.count("k_move") > before and fake.current == 0
    s.step(1)   # still in order
    s.destroy()


@pytest.mark.parametrize("read", ["field", "spectrum", "checkpoint", "release"])
def test_a_read_that_fails_is_an_error(fake, read):
    """A copy from the device that fails, and any read of the failed device after it: no zeros in place of the state."""
    fake.current = 0
    s = scenes.lossy_scene(fake.lib)[0]
    s.step(10)
    fake.so.fake_fail_copy(0)
    try:
        for _ in range(2):
            with pytest.raises(CourantError):
                READS[read](s)
    finally:
        fake.so.fake_fail_copy(-1)
    for later in (s.checkpoint, lambda: s.field(1), lambda: s.sourceSpectrum()):
        with pytest.raises(CourantError):
            later()
    s.destroy()


def test_mode_port_waves_of_a_failed_read_are_an_error(fake):
    fake.current = 0
    s, meta = scenes.modeport_scene(fake.lib)
    s.step(10)
    fake.so.fake_fail_copy(0)
    try:
        with pytest.raises(CourantError):
            s.modePortWaves(meta["modeports"][0])
    finally:
        fake.so.fake_fail_copy(-1)
    s.destroy()


@pytest.mark.parametrize("read", ["field", "spectrum", "checkpoint", "release"])
@pytest.mark.parametrize("scene", [scenes.parity_scene, scenes.lossy_scene], ids=["plain", "lossy"])
def test_moving_state_allocates_nothing_on_the_device(fake, scene, read):
    """Callers may have given all device memory away by the time they read results or go back to a saved state."""
    fake.current = 0
    s = scene(fake.lib)[0]
    s.step(10)
    made = fake.count("malloc")
    saved = READS[read](s)
    assert fake.count("malloc") == made
    if read == "checkpoint":
        s.restore(saved)
        s.step(1)
        assert fake.count("malloc") == made
    s.destroy()


@pytest.mark.parametrize("scene", [scenes.parity_scene, scenes.lossy_scene], ids=["plain", "lossy"])
def test_small_tables_go_up_together(fake, scene):
    """Dozens of tables of a few kilobytes: one copy, and one more for each array too large to share it."""
    fake.current = 0
    s = scene(fake.lib)[0]
    before = fake.count("up")
    s.prepareDevice()
    assert fake.count("up") - before <= 8
    s.destroy()


def probed_box(c):
    """A small closed box full of probes: the samples outweigh the fields."""
    s = c.createSim(1e-4 * np.arange(31), 1e-4 * np.arange(29), 1e-4 * np.arange(25))
    s.setFrequencies(np.linspace(1e9, 20e9, 50))
    for q in range(60):
        s.addIProbe(0, 2 + q % 26, 2, 26, 2, 22)
    s.finalize(0.9)
    return s, {}


@pytest.mark.parametrize("make", [scenes.parity_scene, scenes.lossy_scene, scenes.modeport_scene, probed_box,
                                  lambda c: boards.seeded_board(c, seed=4, cells=8e4, ports="lumped", nf=8),
                                  lambda c: boards.seeded_board(c, seed=6, cells=3e5, ports="mode", nf=8)],
                         ids=["plain", "lossy", "mode ports", "probes", "board", "larger board"])
def test_device_bytes_are_all_counted(fake, make):
    """sizes() tells what is allocated, before and after results were read, and a server's estimate covers it."""
    fake.current = 0
    s = make(fake.lib)[0]
    estimate, before = serve.footprint(s), fake.count("live")
    s.prepareDevice()
    assert s.sizes()["device_bytes"] == fake.count("live") - before
    s.step(40)
    s.checkpoint(), s.sourceSpectrum(), s.energy()
    held = fake.count("live") - before
    assert s.sizes()["device_bytes"] == held
    assert held <= estimate <= 1.3 * held + (6 << 20)
    s.destroy()
    assert fake.count("live") == before


def debye_box(c, n, poles):
    """CPML round a box whose lower half is Debye material."""
    s = c.createSim(*(1e-4 * np.arange(q + 1) for q in n))
    for f in (0, 1, 2, 3, 5):
        s.setBoundary(f, 1, 6)
    fp = np.geomspace(1e9, 40e9, poles)
    s.setDebyePoles(fp)
    s.materialBoxDebye(-1, 1, -1, 1, 0, 1e-4 * (n[2] // 2), DebyeModel(3.5, fp, np.full(poles, 0.05), 0.0))
    p = s.addLumpedPort(2, n[0] // 2, n[1] // 2, 0, 4, 1, 50.0)
    s.setGaussian(p, 1.0, 8e-12, 3e-12)
    s.setFrequencies([5e9])
    s.finalize(0.9)
    return s


@pytest.mark.parametrize("n,poles,apart", [((120, 104, 84), 12, True), ((80, 72, 60), 12, False), ((140, 132, 112), 7, True),
                                           ((140, 132, 112), 6, False), ((120, 104, 84), 8, False)])
def test_lean_blocks_of_grids_with_many_poles_run_by_themselves(fake, n, poles, apart):
    fake.current = 0
    s = debye_box(fake.lib, n, poles)
    before = {k: fake.count(k) for k in ("k_whole_e", "k_update_e_fast")}
    s.step(3)
    assert fake.count("k_whole_e") - before["k_whole_e"] == 3
    assert fake.count("k_update_e_fast") - before["k_update_e_fast"] == (3 if apart else 0)
    s.destroy()


def closed_box(c, n, copper=False):
    s = c.createSim(*(1e-4 * np.arange(q + 1) for q in n))
    if copper:
        s.setConductorLoss(5.8e7, 1e9, 40e9)
        s.pecBox(1e-3, 1.4e-3, 1e-3, 1.5e-3, 0.9e-3, 1.2e-3)
    p = s.addLumpedPort(2, n[0] // 2, n[1] // 2, 0, n[2] // 4, 1, 50.0)
    s.setGaussian(p, 1.0, 8e-12, 3e-12)
    s.setFrequencies([5e9])
    s.finalize(0.9)
    return s


@pytest.mark.parametrize("n,copper,lean", [((60, 50, 40), False, True), ((120, 120, 90), False, True), ((60, 50, 40), True, False),
                                           ((110, 110, 90), True, True), ((300, 8, 8), False, False)])
def test_grids_of_lean_blocks_run_in_the_lean_kernels(fake, n, copper, lean):
    fake.current = 0
    s = closed_box(fake.lib, n, copper)
    before = {k: fake.count(k) for k in ("k_whole_h", "k_whole_e", "k_update_h_fast", "k_update_e_fast")}
    s.step(3)
    made = {k: fake.count(k) - v for k, v in before.items()}
    whole, fast = (0, 3) if lean else (3, 0)
    assert made == {"k_whole_h": whole, "k_whole_e": whole, "k_update_h_fast": fast, "k_update_e_fast": fast}
    s.destroy()


def open_box(c, n):
    s = c.createSim(*(1e-4 * np.arange(q + 1) for q in n))
    for f in (0, 1, 2, 3, 5):
        s.setBoundary(f, 1, 6)
    s.setFrequencies([5e9])
    s.finalize(0.9)
    return s


@pytest.mark.parametrize("n,streams", [((140, 132, 112), 2), ((40, 36, 30), 1)], ids=["two streams", "one stream"])
def test_the_tuner_times_each_choice_on_its_own_graph(fake, tmp_path, monkeypatch, n, streams):
    """Every choice times faster than the one before, so each is kept: a graph of its own must have been captured for
    it (as it is, z tails, two thin-segment thresholds, streams, two graph lengths), none for a stream that is not used.
    Of the steps left, with 7 choices 1376, the first run ends with the sample ring after 352: 5 graphs of 64 and one of
    the 32 steps that were left over before as well; with 6 choices 1472, after 448, 7 graphs of 64."""
    monkeypatch.setenv("CEM_B200_TUNE_CACHE", str(tmp_path / "shapes.txt"))
    fake.current = 0
    s = open_box(fake.lib, n)
    s.prepareDevice()
    s.tune(True)
    fake.so.fake_elapsed(1.0, 0.5)
    before = fake.count("capture")
    try:
        s.step(2048)
    finally:
        fake.so.fake_elapsed(1.0, 1.0)
    st = s.tuneState()
    assert st["tuned"] and fake.count("capture") - before == (8 if streams == 2 else 6)
    assert st["side_stream"] == (streams == 1)
    s.destroy()


def test_tables_of_launches_in_flight_are_not_freed(fake, tmp_path, monkeypatch):
    """A tuned shape from the cache file replaces the place tables of a simulation that has steps in flight."""
    cache = tmp_path / "shapes.txt"
    monkeypatch.setenv("CEM_B200_TUNE_CACHE", str(cache))
    fake.current = 0
    a, b = open_box(fake.lib, (60, 200, 180)), open_box(fake.lib, (60, 200, 180))
    a.tune(True)
    fake.so.fake_elapsed(1.0, 0.5)
    a.step(2048)
    fake.so.fake_elapsed(1.0, 1.0)
    assert len(cache.read_text().splitlines()) == 1 and a.tuneState()["z_tails"] != b.tuneState()["z_tails"]
    a.synchronize()
    b.step(40)
    b.tune(True)
    before = fake.count("free"), fake.count("free in flight")
    b.step(2048)
    assert b.tuneState()["from_cache"] and fake.count("free") > before[0]
    assert fake.count("free in flight") == before[1]
    a.destroy()
    b.destroy()


def test_shapes_tuned_for_earlier_kernels_are_measured_again(fake_path, tmp_path, monkeypatch):
    """A cache file from before the merged launches: its lines are of the same grid, but of other kernels."""
    cache = tmp_path / "shapes.txt"
    monkeypatch.setenv("CEM_B200_TUNE_CACHE", str(cache))
    old = "40x36x30/p0/sibc0/pml6.6.6.6.0.6 8 0 64 0.05 1\n"
    cache.write_text(old)
    for name, from_cache in (("first", False), ("second", True)):   # copies of their own: the file is read once a process
        own = tmp_path / f"lib{name}.so"
        shutil.copy(fake_path, own)
        f = Fake(own)
        s = open_box(f.lib, (40, 36, 30))
        s.tune(True)
        s.step(2048)
        st = s.tuneState()
        assert st["tuned"] and st["from_cache"] == from_cache
        s.destroy()
    lines = cache.read_text().splitlines()
    assert lines[0] + "\n" == old and len(lines) == 2


def test_batch_statistics_are_what_was_launched(fake, tmp_path, monkeypatch):
    """Runs without a graph, with graphs of 32 steps, and with one of the steps left over as well."""
    monkeypatch.setenv("CEM_B200_TUNE_CACHE", str(tmp_path / "shapes.txt"))
    fake.current = 0
    sims = [scenes.parity_scene(fake.lib)[0], scenes.lossy_scene(fake.lib)[0], open_box(fake.lib, (140, 132, 112))]
    b = fake.lib.createBatch()
    for s in sims:
        b.add(s, 5000)
    for n in (7, 1, 42, 42, 300, 1100, 64):
        before = fake.count("launch") + fake.count("graph")
        b.run(n)
        made = fake.count("launch") + fake.count("graph") - before
        st = b.stats()
        assert (st["launches"], st["chunk"], st["steps"]) == (made, 32, n)
    b.remove(sims[2])
    sims[2].tune(True)
    fake.so.fake_elapsed(1.0, 0.5)
    sims[2].step(2048)
    fake.so.fake_elapsed(1.0, 1.0)
    b.add(sims[2], 10)
    sims[2].step(3)   # in flight when the run begins
    b.run(10)
    assert b.stats()["chunk"] == sims[2].tuneState()["graph_steps"] == 64
    b.destroy()
    for s in sims:
        s.destroy()


def test_a_short_call_launches_no_more_than_its_run(fake):
    """One step: the run's begin, H, E and its sample rows; the step count and source values are the run's own."""
    fake.current = 0
    s = scenes.parity_scene(fake.lib)[0]
    s.step(5)
    before = fake.count("launch")
    s.step(1)
    assert fake.count("launch") - before == 4
    s.destroy()


def test_a_graph_is_captured_when_it_will_be_replayed(fake):
    """Not for the first 32 steps (a capture costs the host more than their launches); for the next, or for 64 at once."""
    fake.current = 0
    a, b = scenes.parity_scene(fake.lib)[0], scenes.parity_scene(fake.lib)[0]
    made = fake.count("capture")
    a.step(32)
    assert fake.count("capture") == made
    a.step(32)
    b.step(64)
    assert fake.count("capture") == made + 2
    a.destroy()
    b.destroy()


LAUNCHES = {"plain": lambda c: scenes.parity_scene(c)[0], "lossy": lambda c: scenes.lossy_scene(c)[0],
            "closed": lambda c: closed_box(c, (60, 50, 40)), "closed copper": lambda c: closed_box(c, (60, 50, 40), True),
            "larger closed copper": lambda c: closed_box(c, (110, 110, 90), True), "large": lambda c: open_box(c, (140, 132, 112)),
            "many poles": lambda c: debye_box(c, (120, 104, 84), 12), "large, poles": lambda c: debye_box(c, (140, 132, 112), 4)}


@pytest.mark.parametrize("name", LAUNCHES)
def test_launches_per_step_are_what_is_launched(fake, name):
    fake.current = 0
    s = LAUNCHES[name](fake.lib)
    s.step(1)
    before = fake.count("launch")
    s.step(5)   # and the run's begin and its sample rows
    assert fake.count("launch") - before == 5 * s.sizes()["launches_per_step"] + 2
    s.destroy()


@pytest.mark.parametrize("n,lean", [((3000, 6, 6), True), ((2999, 6, 6), False), ((3000, 60, 40), True), ((3000, 24, 20), False)])
def test_thousands_of_short_planes_run_in_the_lean_kernels(fake, n, lean):
    """One block of a few threads per plane and component, thousands of times (and not with planes of more than one block,
    unless they are four)."""
    fake.current = 0
    s = closed_box(fake.lib, n)
    before = fake.count("k_whole_h"), fake.count("k_update_h_fast")
    s.step(3)
    assert (fake.count("k_whole_h") - before[0], fake.count("k_update_h_fast") - before[1]) == ((0, 3) if lean else (3, 0))
    s.destroy()
