"""Large grids with all launches on one stream (a choice of the tuner, taken from
its cache file here) give the bits of two streams: the blocks that carry a run's
samples, its begin and the surface impedance then come after the lean ones, or
before them where the lean blocks of E run apart."""
import shutil

import numpy as np
import pytest

from courant_b200 import build
from courant_b200.api import Courant, DebyeModel

pytestmark = pytest.mark.gpu


def box(c, n, poles=0, copper=False):
    s = c.createSim(*(1e-4 * np.arange(q + 1) for q in n))
    for f in (0, 1, 2, 3, 5):
        s.setBoundary(f, 1, 6)
    if poles:
        fp = np.geomspace(1e9, 40e9, poles)
        s.setDebyePoles(fp)
        s.materialBoxDebye(-1, 1, -1, 1, 0, 1e-4 * (n[2] // 2), DebyeModel(3.5, fp, np.full(poles, 0.05), 0.0))
    if copper:
        s.setConductorLoss(5.8e7, 1e9, 40e9)
        s.pecBox(2e-3, 2.4e-3, 2e-3, 2.5e-3, 0.9e-3, 1.2e-3)
    p = s.addLumpedPort(2, n[0] // 2, n[1] // 2, 0, 4, 1, 50.0)
    s.setGaussian(p, 1.0, 8e-12, 3e-12)
    s.setFrequencies([5e9, 20e9])
    s.addVProbe(2, n[0] // 2 + 3, n[1] // 2, 0, 6, 1)
    s.addIProbe(2, 5, n[0] // 2 - 3, n[0] // 2 + 3, n[1] // 2 - 3, n[1] // 2 + 3)
    s.finalize(0.9)
    return s


@pytest.mark.parametrize("kw", [dict(n=(172, 130, 96), copper=True), dict(n=(120, 104, 84), poles=9)], ids=lambda kw: "-".join(str(v) for v in kw.values()))
def test_one_stream_gives_the_bits_of_two(lib, tmp_path, monkeypatch, kw):
    n = kw["n"]
    cache = tmp_path / "shapes.txt"
    cache.write_text(f"{n[0]}x{n[1]}x{n[2]}/p{kw.get('poles', 0)}/sibc{int(kw.get('copper', False))}/pml6.6.6.6.0.6/l2 16 0 32 0.05 1\n")
    monkeypatch.setenv("CEM_B200_TUNE_CACHE", str(cache))
    own = tmp_path / "libone.so"   # a copy of its own: the file is read once per process and library
    shutil.copy(build.LIB, own)
    a, b = box(lib, **kw), box(Courant(own), **kw)
    b.tune(True)
    for s in (a, b):
        s.step(2100)
    st = b.tuneState()
    assert st["from_cache"] and not st["side_stream"]
    assert np.array_equal(a.checkpoint(), b.checkpoint())
    a.destroy()
    b.destroy()
