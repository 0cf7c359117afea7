"""State between host and device: a checkpoint of FP32 values goes up (host
copies -> device arrays) and comes down again unchanged, whatever arrays the
scene has and wherever the moves are cut (a chunk is 2^20 words)."""
import numpy as np
import pytest

from courant_b200 import scenes

pytestmark = pytest.mark.gpu


def plain_box(c, n):
    s = c.createSim(*(1e-4 * np.arange(q + 1) for q in n))
    s.setFrequencies([5e9, 20e9])
    s.finalize(0.9)
    return s


SCENES = {"smallest": lambda c: plain_box(c, (2, 2, 2)), "ragged": lambda c: plain_box(c, (7, 13, 5)),
          "one chunk and a little": lambda c: plain_box(c, (55, 66, 46)),
          "three chunks": lambda c: plain_box(c, (101, 73, 57)),
          "CPML, copper, Debye": lambda c: scenes.lossy_scene(c)[0],
          "CPML on all faces": lambda c: scenes.parity_scene(c)[0]}


@pytest.mark.parametrize("name", SCENES)
def test_a_checkpoint_goes_up_and_comes_down_unchanged(lib, name):
    s = SCENES[name](lib)
    want = s.checkpoint()
    rng = np.random.default_rng(11)
    want[8:] = rng.standard_normal(want.size - 8).astype(np.float32)
    s.restore(want)
    s.prepareDevice()
    got = s.checkpoint()
    # not state of their own: E before the last update (reads back as E now), the phasors of the step
    psi = sum(s.stateLen(e, c, w) for e in range(2) for c in range(3) for w in range(2))
    old = 8 + 6 * s.N + psi + s.stateLen(2)
    keep = np.ones(want.size, bool)
    keep[old:old + s.stateLen(3)] = False
    keep[want.size - 4 * s.nf:] = False
    assert np.array_equal(got[keep], want[keep])
