"""The waits of the whole-GPU kernel: a CTA that misses a word ends the whole solve as
TIMEOUT, never as another end with some rows wrong, and the context stays usable."""
import pytest

pytestmark = pytest.mark.gpu

PASSES = 6  # of the probe: two exchanges before them, two in each


@pytest.mark.parametrize("exchange", range(0, 3 + 2 * PASSES))
def test_a_lost_word_is_a_timeout(gb, handle, exchange):
    st, ms = gb.probe_grid_timeout(0, exchange)
    assert st == (gb.MAX_ITER if exchange in (0, 2 + 2 * PASSES) else gb.TIMEOUT)
    assert exchange == 0 or 20 <= ms < 1000, ms  # one wait of 20 ms for the word, one for the CTA that gave up


def test_probe_arguments(gb, handle):
    with pytest.raises(gb.GbdpcgError):
        gb.probe_grid_timeout(0, 3 + 2 * PASSES)
