"""Runs of whole steps (cem_step) against the phases they are made of (cem_mt_*).

A run samples probes and ports inside its update launches and turns the
samples into probe rows afterwards; which launch carries what depends on the
scene (CPML or none, surface impedance, probes). Both ways must give the same
bits, for run lengths at the edges: single steps, the steps around a replayed
graph (32), and past the sample ring (1024 rows)."""
import numpy as np
import pytest

from courant_b200 import scenes

pytestmark = pytest.mark.gpu


def closed_box(c, copper: bool, probes: bool = True):
    """A PEC cavity (no CPML, so no general blocks), optionally around a copper block."""
    s = c.createSim(1e-4 * np.arange(20), 1e-4 * np.arange(18), 0.8e-4 * np.arange(15))
    s.materialBox(-1, 1, -1, 1, 0, 4e-4, 3.0, 0.05)
    if copper:
        s.setConductorLoss(5.8e7, 1e9, 40e9)
        s.pecBox(8e-4, 1.2e-3, 7e-4, 1.1e-3, 0, 4e-4)
    p = s.addLumpedPort(2, 4, 4, 0, 4, 1, 50.0)
    s.setGaussian(p, 1.0, 12e-12, 5e-12)
    s.setFrequencies([5e9, 20e9, 60e9])
    if probes:
        s.addVProbe(2, 6, 5, 0, 5, -1)
        s.addIProbe(2, 6, 2, 7, 2, 6)
    s.finalize(0.95)
    return s


SCENES = {"closed": lambda c: closed_box(c, False), "closed, port only": lambda c: closed_box(c, False, False),
          "closed copper": lambda c: closed_box(c, True), "lossy": lambda c: scenes.lossy_scene(c)[0]}


def phases(s, n):
    ex, h = s.c.ex, s.h
    for _ in range(n):
        ex.cem_mt_pre(h)
        ex.cem_mt_H(h, 0, s.nx + 1)
        ex.cem_mt_mid(h)
        ex.cem_mt_E(h, 0, s.nx)
        ex.cem_mt_post(h)


@pytest.mark.parametrize("name", SCENES)
@pytest.mark.parametrize("chunks", [(1, 1, 1), (31, 2, 32, 65)], ids=["single", "graph"])
def test_runs_equal_their_phases(lib, name, chunks):
    a, b = SCENES[name](lib), SCENES[name](lib)
    for n in chunks:
        a.step(n)
    phases(b, sum(chunks))
    assert a.steps == b.steps == sum(chunks)
    assert np.array_equal(a.checkpoint(), b.checkpoint())
    assert np.array_equal(a.sourceSpectrum(), b.sourceSpectrum())


def test_run_past_the_sample_ring(lib):
    a, b = SCENES["closed copper"](lib), SCENES["closed copper"](lib)
    a.step(2500)
    for n in (1000, 24, 1, 1475):
        b.step(n)
    assert np.array_equal(a.checkpoint(), b.checkpoint())
    assert np.array_equal(a.portV(0), b.portV(0)) and np.array_equal(a.iprobe(0), b.iprobe(0))


def test_repeated_short_runs(lib):
    """A run's rest replays a graph once the run before left as much; other rests in between, single steps among them."""
    a, b = SCENES["lossy"](lib), SCENES["lossy"](lib)
    chunks = (10, 10, 10, 42, 10, 3, 3, 10, 10, 1, 1, 31, 31)
    for n in chunks:
        a.step(n)
    for _ in range(sum(chunks)):
        b.step(1)
    assert np.array_equal(a.checkpoint(), b.checkpoint())
    assert np.array_equal(a.portI(1), b.portI(1))
