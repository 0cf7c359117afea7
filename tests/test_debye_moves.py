"""Debye currents between host and device: up to 2^20 edges they move packed,
of more their boxes move whole; either way cut by the chunks of a move (2^20
words), in rows of every length, with air between two blocks of material."""
import numpy as np
import pytest

from courant_b200 import scenes  # noqa: F401  (the package's path)
from courant_b200.api import DebyeModel

pytestmark = pytest.mark.gpu


def blocks(c, n, poles, split):
    """Debye material in two blocks along x and z with air between them (split), or in one that ends inside the grid."""
    x, y, z = (1e-4 * np.arange(q + 1) for q in n)
    s = c.createSim(x, y, z)
    fp = np.geomspace(1e9, 40e9, poles)
    s.setDebyePoles(fp)
    m = DebyeModel(3.5, fp, np.full(poles, 0.05), 0.0)
    a, b = (n[0] // 2 - 2, n[2] * 3 // 4) if split else (n[0] - 1, n[2] - 1)
    s.materialBoxDebye(-1, x[a], -1, 1, z[1], z[max(b, 2)], m)
    if split:
        s.materialBoxDebye(x[n[0] - a], 1, y[2], 1, z[n[2] - b], 1, m)
    p = s.addLumpedPort(2, n[0] // 2, n[1] // 2, 0, 2, 1, 50.0)
    s.setGaussian(p, 1.0, 12e-12, 5e-12)
    s.setFrequencies([5e9, 20e9])
    s.finalize(0.9)
    return s


@pytest.mark.parametrize("n,poles,split", [((5, 4, 6), 1, False), ((23, 17, 13), 5, True), ((61, 45, 37), 3, True),
                                           ((112, 90, 61), 2, False), ((120, 101, 78), 1, True)])
def test_currents_go_up_and_come_down_unchanged(lib, n, poles, split):
    s = blocks(lib, n, poles, split)
    want = s.checkpoint()
    rng = np.random.default_rng(5)
    want[8:] = rng.standard_normal(want.size - 8).astype(np.float32)
    s.restore(want)
    s.prepareDevice()
    got = s.checkpoint()
    at = 8 + 6 * s.N
    assert (s.sizes()["ndisp"] > 1 << 20) == (n[0] > 100)
    assert np.array_equal(got[8:at + s.stateLen(2)], want[8:at + s.stateLen(2)])
    s.destroy()


@pytest.mark.parametrize("n", [(61, 45, 37), (120, 101, 78)], ids=["packed", "whole boxes"])
def test_a_run_goes_on_from_its_checkpoint(lib, n):
    """Nothing but the edges' own currents is set: the same steps from a saved state give the same state."""
    a, b = blocks(lib, n, 2, True), blocks(lib, n, 2, True)
    a.step(90)
    saved = a.checkpoint()
    b.step(7)
    b.restore(saved)
    a.step(40)
    b.step(40)
    assert np.array_equal(a.checkpoint(), b.checkpoint())
    a.destroy()
    b.destroy()
