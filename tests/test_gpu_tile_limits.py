"""Which runtime tiles a grid takes does not depend on how many exchanges its
transforms make: at three radices (240 = 16 3 5) the largest z tile that fits is
the one whose layout has a second transform buffer, though two of the radices run
as one stage."""
import pytest

pytestmark = pytest.mark.gpu


def test_tiles_of_three_radices(qvti):
    with qvti.Simulation(16, 16, 240, 4, 10.0, 10.0, 10.0, 1e-3, 20.0) as sim:
        sim.set_tiles([0, 0, 0, 0, 0, 4])
        with pytest.raises(qvti.QvtiError):
            sim.set_tiles([0, 0, 0, 0, 0, 8])
        assert sim.tiles()[0][5] == 4
