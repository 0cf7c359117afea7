"""The cem_mt_* phases while a caller holds a field pointer: E goes up and down
between any two of them, and the port voltages are still the mean of those
before and after the E update."""
import numpy as np
import pytest

from courant_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("comp", [0, 2, 5])
def test_phases_with_a_live_field_give_the_same_spectra(lib, comp):
    a, b = scenes.lossy_scene(lib)[0], scenes.lossy_scene(lib)[0]
    a.step(60)
    b.step(60)
    a.fieldView(comp)
    ex, m = a.c.ex, a.nx // 2
    for _ in range(6):
        ex.cem_mt_pre(a.h)
        ex.cem_mt_H(a.h, 0, m)
        ex.cem_mt_H(a.h, m, a.nx + 1)
        ex.cem_mt_mid(a.h)
        ex.cem_mt_E(a.h, 0, m)
        ex.cem_mt_E(a.h, m, a.nx)
        ex.cem_mt_post(a.h)
    a.step(5)
    b.step(11)
    assert np.array_equal(a.checkpoint(), b.checkpoint())
    for p in range(2):
        assert np.array_equal(a.portV(p), b.portV(p)) and np.array_equal(a.portI(p), b.portI(p))
