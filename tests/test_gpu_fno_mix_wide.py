"""The mixing's gradients with more channels than a grid has rows of blocks (65535
of four inputs or 32 outputs); reference and tolerance of the ordinary sizes."""

import pytest

from test_gpu_fno_mix import test_mixing_and_gradients as check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C,O", [(65535 * 4 + 5, 1), (1, 65535 * 32 + 5)])
def test_many_channels(cuda, C, O):
    check(cuda, C, O, 1, 1, 1)
