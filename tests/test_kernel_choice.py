"""The kernel choice (cemx_use_fused) in mid-run. A fused step writes the other
one of two field buffers; what is stepped with the separate kernels afterwards,
replayed graphs included, must go on from there."""
import numpy as np
import pytest

from courant_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 10, 32, 75])
def test_separate_kernels_go_on_from_a_fused_step(lib, n):
    a, b = scenes.lossy_scene(lib)[0], scenes.lossy_scene(lib)[0]
    a.step(n)
    a.step(n)            # a run of this length has its graph now
    for _ in range(2):   # to the second buffer, and back to the first
        a.useFused(True)
        a.step(1)
        a.useFused(False)
        a.step(n)
        a.step(n)
    for _ in range(6 * n + 2):
        b.step(1)
    assert a.steps == b.steps
    assert np.array_equal(a.checkpoint(), b.checkpoint())
    assert np.array_equal(a.portV(0), b.portV(0)) and a.energy() == b.energy()


def test_replayed_graphs_give_the_bits_of_launches(lib, monkeypatch):
    """Graphs of 32 steps and of the 12 left over, a graph of 7 steps replayed, and no graph at all
    (CEM_B200_GRAPHS=0), past a flush of the sample ring (1024 steps)."""
    monkeypatch.setenv("CEM_B200_GRAPHS", "0")
    plain = scenes.lossy_scene(lib)[0]
    plain.prepareDevice()
    monkeypatch.delenv("CEM_B200_GRAPHS")
    a, b = scenes.lossy_scene(lib)[0], scenes.lossy_scene(lib)[0]
    plain.step(1100)
    a.step(1100)
    for n in [7] * 157 + [1]:
        b.step(n)
    want = plain.checkpoint()
    assert np.array_equal(a.checkpoint(), want) and np.array_equal(b.checkpoint(), want)


def test_state_is_read_from_a_thread_without_a_device(lib):
    """A thread that has made no CUDA call reads fields, spectra and a checkpoint of another thread's simulation."""
    import threading

    s = scenes.lossy_scene(lib)[0]
    s.step(50)
    got = []
    t = threading.Thread(target=lambda: got.extend([s.portV(0), s.field(2), s.checkpoint()]))
    t.start()
    t.join()
    want = scenes.lossy_scene(lib)[0]
    want.step(50)
    assert len(got) == 3
    assert np.array_equal(got[0], want.portV(0)) and np.array_equal(got[1], want.field(2)) and np.array_equal(got[2], want.checkpoint())
