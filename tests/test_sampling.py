"""Probe and port edges sampled by blocks of the update launches: the numbers
of entries around a block's (128 of a family), in every kind of launch that
carries them, give the bits of the phases; and many entries cost a step little."""
import numpy as np
import pytest

from courant_b200.api import DebyeModel

pytestmark = pytest.mark.gpu

BIG = (172, 130, 96)   # above 2 M cells: a kernel per class of blocks


def box(c, n, edges, loops, cpml=False, copper=False):
    """A box with a voltage probe of `edges` edges and current loops round it."""
    s = c.createSim(*(1e-4 * np.arange(q + 1) for q in n))
    if cpml:
        for f in (0, 1, 2, 3, 5):
            s.setBoundary(f, 1, 6)
    if copper:
        s.setConductorLoss(5.8e7, 1e9, 40e9)
        s.pecBox(1.2e-3, 1.6e-3, 1e-3, 1.5e-3, 0.9e-3, 1.2e-3)
    p = s.addLumpedPort(2, 8, 8, 0, 4, 1, 50.0)
    s.setGaussian(p, 1.0, 8e-12, 3e-12)
    s.setFrequencies([5e9, 20e9])
    while edges > 0:   # parts of a line, from row to row
        m = min(edges, n[1] - 16)
        s.addVProbe(1, 8 + (edges % 5), 7 + edges % 7, 8, 8 + m, 1)
        edges -= m
    for q in range(loops):
        s.addIProbe(0, 9 + q % (n[0] - 18), 8, n[1] - 8, 8, n[2] - 8)
    s.finalize(0.9)
    return s


def debye_box(c, n, poles, copper):
    """CPML round a box whose lower half is Debye material, with or without a block of copper in it."""
    s = c.createSim(*(1e-4 * np.arange(q + 1) for q in n))
    for f in (0, 1, 2, 3, 5):
        s.setBoundary(f, 1, 6)
    fp = np.geomspace(1e9, 40e9, poles)
    s.setDebyePoles(fp)
    s.materialBoxDebye(-1, 1, -1, 1, 0, 1e-4 * (n[2] // 2), DebyeModel(3.5, fp, np.full(poles, 0.05), 0.0))
    if copper:
        s.setConductorLoss(5.8e7, 1e9, 40e9)
        s.pecBox(2e-3, 2.4e-3, 2e-3, 2.5e-3, 0.9e-3, 1.2e-3)
    p = s.addLumpedPort(2, n[0] // 2, n[1] // 2, 0, 4, 1, 50.0)
    s.setGaussian(p, 1.0, 8e-12, 3e-12)
    s.setFrequencies([5e9])
    s.addVProbe(2, n[0] // 2 + 3, n[1] // 2, 0, 6, 1)
    s.addIProbe(2, 5, n[0] // 2 - 3, n[0] // 2 + 3, n[1] // 2 - 3, n[1] // 2 + 3)
    s.finalize(0.9)
    return s


def phases(s, n):
    ex, h = s.c.ex, s.h
    for _ in range(n):
        ex.cem_mt_pre(h)
        ex.cem_mt_H(h, 0, s.nx + 1)
        ex.cem_mt_mid(h)
        ex.cem_mt_E(h, 0, s.nx)
        ex.cem_mt_post(h)


CASES = [(dict(n=(40, 36, 28), edges=e, loops=k), 45) for e, k in ((0, 0), (123, 0), (124, 1), (125, 2), (380, 9), (2100, 40))]
CASES += [(dict(n=(40, 36, 28), edges=300, loops=12, cpml=p, copper=q), 45) for p, q in ((True, False), (True, True), (False, True))]
CASES += [(dict(n=BIG, edges=e, loops=6, cpml=p, copper=q), 12)
          for e, p, q in ((300, False, False), (300, True, False), (300, True, True), (300, False, True), (0, True, False))]


@pytest.mark.parametrize("kw,steps", CASES, ids=lambda v: "-".join(str(x) for x in v.values()) if isinstance(v, dict) else None)
def test_runs_sample_what_the_phases_do(lib, kw, steps):
    a, b = box(lib, **kw), box(lib, **kw)
    for n in (steps - 9, 1, 8):
        a.step(n)
    phases(b, steps)
    assert np.array_equal(a.checkpoint(), b.checkpoint())   # fields and all spectra
    assert np.abs(a.portV(0)).max() > 0
    a.destroy()
    b.destroy()


@pytest.mark.parametrize("n,poles,copper", [((120, 104, 84), 9, True), ((140, 132, 112), 7, False), ((140, 132, 112), 16, True),
                                            ((140, 132, 112), 4, True), ((140, 132, 112), 1, False)])
def test_e_of_large_grids_with_poles_gives_the_bits_of_the_phases(lib, n, poles, copper):
    """All blocks of E in one launch, and with many poles the lean rectangles in a launch beside the others."""
    a, b = debye_box(lib, n, poles, copper), debye_box(lib, n, poles, copper)
    for k in (33, 1, 6):
        a.step(k)
    phases(b, 40)
    assert np.array_equal(a.checkpoint(), b.checkpoint())
    a.destroy()
    b.destroy()


def test_many_probes_cost_a_step_little(lib):
    """Six thousand entries are read side by side: less than as much again as the step without them."""
    t = []
    for loops in (1, 64):
        s = box(lib, (61, 47, 35), 0, loops)
        s.stepTimed(96)
        t.append(min(s.stepTimed(320) for _ in range(5)))
        s.destroy()
    assert t[1] < 2 * t[0]


@pytest.mark.parametrize("faces", [(), (0, 1), (0, 1, 5)], ids=["closed", "x", "x and z"])
def test_thousands_of_short_planes_give_the_bits_of_the_phases(lib, faces):
    def make():
        s = lib.createSim(*(1e-4 * np.arange(q + 1) for q in (3001, 7, 9)))
        for f in faces:
            s.setBoundary(f, 1, 4 if f < 2 else 2)
        p = s.addLumpedPort(2, 1500, 3, 0, 4, 1, 50.0)
        s.setGaussian(p, 1.0, 8e-12, 3e-12)
        s.setFrequencies([5e9])
        for q in range(60):
            s.addVProbe(0, 3, 4, 1400 + q, 1480 + q, 1)
        s.addIProbe(0, 1520, 1, 5, 1, 6)
        s.finalize(0.9)
        return s

    a, b = make(), make()
    for n in (64, 1, 7):
        a.step(n)
    phases(b, 72)
    assert np.array_equal(a.checkpoint(), b.checkpoint())
    assert np.abs(a.portV(0)).max() > 0
