"""Heartbeats when the rank that hosts the store has ended before the others ask it who is late."""
import pytest

from zorse_b200.utils.health import DictStore, Heartbeat


@pytest.mark.parametrize("reads_left", range(6))
def test_a_store_that_is_gone_names_nobody(reads_left):
    class Store(DictStore):
        left = 100

        def get(self, k):
            self.left -= 1
            if self.left < 0:
                raise RuntimeError("Connection was likely closed")
            return super().get(k)

    store = Store()
    hbs = [Heartbeat(store, r, 4, clock=lambda: 0.0) for r in range(4)]
    for r in (0, 1, 2, 3):
        hbs[r].beat_enter(2)
    for r in (0, 1, 3):                       # rank 2 never enters step 3
        hbs[r].beat_enter(3)
    assert hbs[3].not_entered(3) == [2]
    store.left = reads_left                   # goes away before or while rank 3 asks: it takes five reads
    assert hbs[3].not_entered(3) == ([2] if reads_left >= 5 else [])
