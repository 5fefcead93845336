"""The summed-area tables at the edges of their tiles, and the box sums of the largest windows in 32 bits."""
import numpy as np
import pytest
import torch

from slipcam_b200 import framecor

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('shape', [(1, 1), (11, 31), (12, 127), (13, 128), (191, 129), (192, 130), (193, 33), (385, 259)])
@pytest.mark.parametrize('offset', [0, 1])
def test_tables_at_tile_edges(shape, offset):
    """rows in steps of 128 pixels, columns in chunks of 192 rows: whole numbers, equal to the cumulative sums"""
    rng = np.random.default_rng(shape[0] * 1000 + shape[1])
    f = rng.integers(0, 256, (2,) + shape, dtype=np.uint8)
    buf = torch.zeros(f.size + 4, dtype=torch.uint8, device='cuda')   # frames on and off a word boundary
    t = buf[offset:offset + f.size].view(f.shape)
    t.copy_(torch.as_tensor(f))
    s, s2 = framecor.sat(t)
    for got, p in ((s, 1), (s2, 2)):
        want = np.zeros((2, shape[0] + 1, shape[1] + 1), np.int64)
        want[:, 1:, 1:] = (f.astype(np.int64) ** p).cumsum(1).cumsum(2)
        assert np.array_equal(got.cpu().numpy().astype(np.int64) & 0xffffffff if p == 1 else got.cpu().numpy(), want)


@pytest.mark.parametrize('window', [253, 254])
def test_box_sums_near_two_to_the_32(window):
    """squares of 254 x 254 pixels of 254 and 255 sum to 4.2e9; the frame against itself peaks at 1 (the
    FP32 form's surfaces are within 1e-5, the bound here ten times that)"""
    rng = np.random.default_rng(window)
    f = torch.as_tensor(rng.integers(254, 256, (300, 301), dtype=np.uint8), device='cuda')
    down, across = np.array([20], np.int32), np.array([23], np.int32)
    cor = framecor.Correlator(300, 301, down, across, window=window, search=1)
    cor.set_reference(f)
    out = cor.correlate(f[None])
    assert abs(float(out['peak'].reshape(-1)[0]) - 1.0) < 1e-4
