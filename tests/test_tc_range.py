"""Which geometries the tensor-core form takes, and what set_form says of the others."""
import numpy as np
import pytest

from slipcam_b200 import framecor

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('size,limit', [(80, 37), (96, 44), (128, 48), (144, 49), (160, 54)])
def test_largest_search(size, limit):
    for search in (limit, limit + 1):
        window = size - 2 * search
        if window < 3:
            continue
        cor = framecor.Correlator(400, 400, np.array([120]), np.array([120]), window=window, search=search)
        assert cor.info()[2] == size
        if search == limit:
            cor.set_form('tc')
        else:
            with pytest.raises(ValueError, match=f'searches up to {limit} px at FFT size {size}, not {search}'):
                cor.set_form('tc')


def test_largest_transform():
    cor = framecor.Correlator(400, 400, np.array([120]), np.array([120]), window=64, search=64)
    with pytest.raises(ValueError, match='FFT sizes up to 160, not 192'):
        cor.set_form('tc')
