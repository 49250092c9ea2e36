"""Rendering groups around the count from which several threads print them (no
device): the output is one thread's, in order, on either side."""

import pytest

from tests.test_render_groups_host import test_groups_in_order as in_order


@pytest.mark.parametrize("fmt", ["ndjson", "csv", "count"])
@pytest.mark.parametrize("n", [4095, 4096, 4097])
def test_around_the_line(n, fmt):
    in_order(n, fmt)
