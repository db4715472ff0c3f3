"""Tile widths without a tuning entry follow one step by size at most: no width
that comes and goes again as the state grows."""
import pytest

from quict_b200.simulation.autotune import default_knobs


@pytest.mark.parametrize("esize", [16, 8])
def test_widths_are_monotone(esize):
    widths = [default_knobs(esize, n).tile_bits for n in range(8, 37)]
    assert widths == sorted(widths)
    assert all(default_knobs(esize, n).low_bits == 5 and default_knobs(esize, n).merge_bits == 2 for n in range(8, 37))
