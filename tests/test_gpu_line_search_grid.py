"""Steps with a known answer where one scenario's links make up to two blocks per
SM (152 x 256 links each), just below, in between and from there on."""

import pytest

import test_gpu_line_search as known

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spare", [38_900, 38_920, 60_000, 77_550, 77_820])
@pytest.mark.parametrize("rule", ["reference", "exact"])
def test_known_steps(built_lib, spare, rule):
    known.test_known_steps(built_lib, spare, rule)
