"""The plain search's and CRS-DE's square root (GPU): correctly rounded on every float of the
range that squared traveltimes in seconds have."""
import pytest

import semb

pytestmark = pytest.mark.gpu


def test_square_root_is_correctly_rounded_on_its_whole_range():
    tested, wrong = semb.selftest_sqrt()
    assert tested == 2 * (75 * 2**23 + 1)
    assert wrong == 0
