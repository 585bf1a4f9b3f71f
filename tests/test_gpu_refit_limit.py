"""The top-level refit on both sides of the count up to which one block does it
(2,048 instances): closest hits after a move as in a fresh build."""
import pytest

import test_gpu_refit_block as block

pytestmark = pytest.mark.gpu

room = block.room


@pytest.mark.parametrize("n", [2047, 2048, 2049, 3000])
def test_refit_at_the_limit_equals_fresh_build(room, n):
    block.test_refit_equals_fresh_build(room, n)
