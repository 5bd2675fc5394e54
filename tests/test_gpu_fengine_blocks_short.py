"""Spectrum-block F-engines at the shortest transforms, where a row has N / 8 threads."""
import pytest

from test_gpu_fengine_blocks import test_blocks_match_rows as blocks_match_rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nch", [32, 64])
@pytest.mark.parametrize("ntaps,ne,nsp", [(4, 37, 250), (8, 37, 250), (8, 3, 9), (5, 11, 70),
                                           (16, 37, 250), (16, 5, 11)])
def test_short_blocks_match_rows(mdt, cuda, nch, ntaps, ne, nsp):
    blocks_match_rows(mdt, cuda, nch, ntaps, ne, nsp)
