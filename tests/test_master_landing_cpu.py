"""How many landing buffers a stage with parked parameters keeps on the device."""
import pytest

from zorse_b200.engine.zero import MasterLanding


@pytest.mark.parametrize("n,units,want", [
    (40_200_000, 14, 5),              # OPT 125M: its embedding
    ((1 << 27), 26, 5),               # the fourth and fifth take a GiB together
    ((1 << 27) + 1, 26, 3),
    (315_000_000, 42, 3),             # a block of OPT 13B: as before there were five
    (40_200_000, 4, 4), (315_000_000, 2, 2), (1024, 1, 1)])
def test_the_number_follows_from_the_size_and_number_of_units(n, units, want):
    assert MasterLanding.count(n, units) == want


def test_a_smaller_number_can_be_set(monkeypatch):
    for buffers in (1, 2):
        monkeypatch.setattr(MasterLanding, "BUFFERS", buffers)
        assert MasterLanding.count(40_200_000, 14) == buffers and MasterLanding.count(315_000_000, 42) == buffers
