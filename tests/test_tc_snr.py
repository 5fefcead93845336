"""
The SNR of the tensor-core form (csrc/corr_tc.cuh) against the surfaces of the same call: the squares of the FP32
values around the peak, summed in FP64.
"""
import numpy as np
import pytest
import torch

from slipcam_b200 import _lib, framecor

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('stat', [3, 21, 41, 97])
@pytest.mark.parametrize('scene', ['plain', 'faint', 'steps'])
def test_snr_of_the_surface(scene, stat):
    """
    plain: correlated frames; faint: a smooth frame under a chequered reference, whose values are all near 1e-4;
    steps: boxes of one odd pixel or a few. The reference is a float
    frame, so that the peaks are not refined and the SNR is the kernel's own. Bounds: the rounding of the FP32
    result, and 1e-13 of the sum for FP64's.
    """
    H, W_, W, R = 240, 368, 64, 48
    M = 2 * R + 1
    rng = np.random.default_rng(4)
    y, x = np.mgrid[:H, :W_]
    smooth = 128 + 100 * np.sin(x / 31.0) * np.cos(y / 37.0)
    ref, frame = 128.0 + 90.0 * ((x + y) % 2 * 2 - 1), smooth
    if scene == 'plain':
        ref = rng.integers(0, 256, (H, W_)).astype(np.float64)
        frame = np.clip(np.roll(ref, (2, -3), (0, 1)) + rng.normal(0, 40, (H, W_)), 0, 255)
    elif scene == 'steps':
        frame = np.full((H, W_), 200.0)
        frame[::50, ::50] = 201.0
    frames = torch.as_tensor(np.rint(frame).astype(np.uint8)[None], device='cuda')
    down, across = np.array([50, 100]), np.array([50, 120, 200])
    cor = framecor.Correlator(H, W_, down, across, window=W, search=R, stat_size=stat)
    cor.set_form('tc')
    r = torch.as_tensor(ref, dtype=torch.float32, device='cuda').contiguous()
    _lib.raise_for(_lib.lib().b200_set_reference_f32_device(cor._h, r.data_ptr(), W_, torch.cuda.current_stream().cuda_stream),
                   cor._h)
    cor._ready = True
    out = cor.correlate(frames, surfaces=True)
    cor.check()
    s = out['surface'].cpu().numpy().astype(np.float64).reshape(-1, M, M)
    got = out['snr'].cpu().numpy().astype(np.float64).reshape(-1)
    checked = 0
    for a, snr in zip(s, got):
        u, v = divmod(int(a.argmax()), M)
        if not a[u, v] > 0:
            assert np.isnan(snr) or snr == 0
            continue
        n = min(stat, M)
        p = a[max(u - n // 2, 0):u - n // 2 + n, max(v - n // 2, 0):v - n // 2 + n]
        total, f0 = (p * p).sum(), a[u, v] ** 2
        mean = (total - f0) / (p.size - 1)
        if mean <= 0:
            continue
        want = f0 / mean
        assert abs(snr / want - 1) < 2.0 ** -24 * 1.01 + 1e-13 * total / (total - f0)
        checked += 1
    assert checked
