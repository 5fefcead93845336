"""
The tensor-core kernel (csrc/corr_tc.cuh) at every transform size it has and at the edges of its tiles:
surfaces of one and of several 16-column tiles, chips shorter than the transform (zero padding), rows on
and off 16-byte boundaries, pairs outside the frame between valid ones, fewer pairs than SMs. Against the
FP32 form on the same frames, with the bounds of test_parity.test_tc_surfaces_close_to_fft32 (FP16 operand
rounding: 2e-3 on a surface) and the exact refinement's for the offsets and peaks.
"""

import numpy as np
import pytest
import torch

from slipcam_b200 import framecor, synth

pytestmark = pytest.mark.gpu

# window, search: transform sizes 16, 32, 48, 64, 80, 96, 128, 144, 160; L equal to and below the size,
# M one above and one below a multiple of 16 or 8
SIZES = [(8, 4), (7, 3), (20, 6), (33, 7), (34, 15), (48, 16), (47, 8), (48, 24), (64, 32), (40, 40), (66, 38), (64, 40),
         (64, 48), (72, 44), (57, 47)]


@pytest.mark.parametrize('width', [400, 397])
@pytest.mark.parametrize('window,search', SIZES)
def test_tc_size(window, search, width):
    h = 260
    motion = np.array([[0.0, 0.0], [1.7, -2.4], [-1.3, 2.1]])
    frames = torch.as_tensor(synth.video(h, width, 3, motion, np.zeros(3), sigma=2.0, noise=1.0, seed=3)).cuda()
    down, across = framecor.window_grid(h, width, window, search, 31)
    # a search centre per window; the last row and column of windows look outside the frame
    rng = np.random.default_rng(window * 1000 + search)
    gross = rng.integers(-2, 3, (2, len(down), len(across), 2)).astype(np.int32)
    gross[:, -1, :, 0] = h
    gross[:, :, -1, 1] = -width
    gross = torch.as_tensor(gross).cuda()
    out = {}
    for form in ('fft32', 'tc'):
        cor = framecor.Correlator(h, width, down, across, window=window, search=search)
        cor.set_form(form)
        cor.set_reference(frames[0])
        out[form] = cor.correlate(frames[1:], gross=gross, surfaces=True)
        cor.check()
    a, b = out['fft32'], out['tc']
    valid = torch.isfinite(a['offsets'][..., 0])
    assert torch.equal(valid, torch.isfinite(b['offsets'][..., 0]))
    assert not valid[:, -1].any() and not valid[:, :, -1].any()
    assert (a['surface'] - b['surface']).abs().max().item() < 2e-3
    if valid.any():
        assert (a['offsets'][valid] - b['offsets'][valid]).abs().max().item() < 1e-3
        assert (a['peak'][valid] - b['peak'][valid]).abs().max().item() < 1e-5


@pytest.mark.parametrize('pairs', [0, 1, 2, 3, 149])
def test_tc_pairs_per_cta(pairs):
    """No valid pair, one, and CTAs with several pairs in flight beside CTAs with one: outputs as FP32's"""
    h, w, window, search = 240, 1280, 64, 48
    frames = torch.as_tensor(synth.video(h, w, 2, np.array([[0.0, 0.0], [0.6, -1.4]]), np.zeros(2), sigma=2.0, noise=1.0,
                                         seed=5)).cuda()
    count = max(pairs, 1)
    across = 48 + np.arange(count) * ((w - 160) // max(count, 2))
    gross = None if pairs else torch.full((1, 2), h, dtype=torch.int32, device='cuda')
    out = {}
    for form in ('fft32', 'tc'):
        cor = framecor.Correlator(h, w, [80], across, window=window, search=search)
        cor.set_form(form)
        cor.set_reference(frames[0])
        out[form] = cor.correlate(frames[1:], gross=gross)
        cor.check()
    a, b = out['fft32'], out['tc']
    valid = torch.isfinite(a['offsets'][..., 0])
    assert torch.equal(valid, torch.isfinite(b['offsets'][..., 0])) and int(valid.sum()) == pairs
    if pairs:
        assert (a['offsets'] - b['offsets']).abs().max().item() < 1e-3
        assert (a['peak'] - b['peak']).abs().max().item() < 1e-5


def test_tc_many_invalid_between_valid():
    """Runs of more than 32 pairs outside the frame (a lane each in the kernel's look ahead) between valid ones"""
    h, w, window, search = 360, 1280, 48, 16
    frames = torch.as_tensor(synth.video(h, w, 13, np.zeros((13, 2)), np.zeros(13), sigma=2.0, noise=1.0, seed=6)).cuda()
    down, across = framecor.window_grid(h, w, window, search, 16)
    gross = torch.full((12, 2), 2 * h, dtype=torch.int32, device='cuda')
    gross[5] = 0
    cor = framecor.Correlator(h, w, down, across, window=window, search=search)
    cor.set_form('tc')
    cor.set_reference(frames[0])
    out = cor.correlate(frames[1:], gross=gross)
    cor.check()
    valid = torch.isfinite(out['offsets'][..., 0])
    assert valid[5].all() and not valid[[0, 1, 2, 3, 4, 6, 7, 8, 9, 10, 11]].any()
    one = cor.correlate(frames[6:7])
    for key in ('offsets', 'peak', 'snr', 'cov'):
        assert torch.equal(out[key][5], one[key][0])
