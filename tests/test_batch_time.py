"""What a batch run reports as its time on the device."""
import pytest

from courant_b200 import boards

pytestmark = pytest.mark.gpu


def test_earlier_steps_of_a_member_are_not_in_the_time(lib):
    """Steps queued before the run (they take some thousand times as long as its one step) are over when its time begins."""
    s, _ = boards.seeded_board(lib, seed=5, cells=2e5, ports="lumped", nf=4, steps=100)
    b = lib.createBatch()
    b.add(s, 10**6)
    b.run(64)
    alone = s.stepTimed(4000)
    s.step(4000)
    b.run(1)
    assert b.stats()["ms"] < 0.5 * alone
    b.destroy()
    s.destroy()
