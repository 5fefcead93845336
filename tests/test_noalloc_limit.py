"""The largest frame of the no-allocation entry point, and what it says of a larger one."""
import numpy as np
import pytest

from slipcam_b200 import _lib, framecor

pytestmark = pytest.mark.gpu
torch = pytest.importorskip('torch')


@pytest.mark.parametrize('shape,fits', [((1080, 1920), True), ((1200, 2000), False)])
def test_largest_frame(shape, fits):
    """16 bytes per pixel are set aside; the message says so, and not that the tables need them"""
    h, w = shape
    cor = framecor.Correlator(h, w, np.array([200, 500]), np.array([300, 900]), window=32, search=8)
    frame = torch.randint(0, 256, (1, h, w), dtype=torch.uint8, device='cuda')
    cor.set_reference(frame[0])
    out = [torch.empty((1, 2, 2) + k, dtype=torch.float32, device='cuda') for k in ((2,), (), (), (3,))]
    rc = _lib.lib().b200_correlate_device_noalloc(cor._h, frame.data_ptr(), 1, w, None, _lib.GROSS_NONE,
                                                  *[o.data_ptr() for o in out], torch.cuda.current_stream().cuda_stream)
    if fits:
        _lib.raise_for(rc, cor._h)
        assert (out[1] > 0.999).all()
    else:
        with pytest.raises(ValueError, match='too large for the no-allocation entry point, which sets aside'):
            _lib.raise_for(rc, cor._h)
