"""
The differentiable correlation where a part of the frame is constant (a black border, a masked or saturated
area) larger than the window: its boxes have no variance, so the surface is 0 there, whatever texture
lies beside them, and neither offsets nor gradients take anything from them.
"""
import numpy as np
import pytest
import torch

import diff_f64 as ref
from slipcam_b200 import synth
from slipcam_b200.diff import DiffCorrelator

pytestmark = pytest.mark.gpu


# the edge of the constant area moves over the column sums' runs of three and the segments of rows
@pytest.mark.parametrize('level', [0.0, 180.0])
@pytest.mark.parametrize('edge', [9, 10, 11, 12])
@pytest.mark.parametrize('side', ['right', 'left', 'below', 'above'])
@pytest.mark.parametrize('W,R', [(3, 8), (16, 8), (32, 8), (48, 20)])
def test_flat_area(W, R, side, edge, level):
    """
    Against FP64. The surface: 0 at the constant boxes; elsewhere within 2e-5 of the surface of a box as
    textured as the search window's most textured one, more by the ratio of their deviations (the FFT's error
    is the chip's). Gradients (of the boxes with 0.3 of that deviation, any cotangent at the constant
    ones) within 1e-4 of their norm, offsets of peaks at such boxes within 1e-3 px.
    """
    rng = np.random.default_rng(1000 * W + edge)
    L, M = W + 2 * R, 2 * R + 1
    H = L + 16
    mover = synth.Mover(synth.texture(H + 16, H + 16, 1.5, rng))
    frames = np.stack([mover.shifted(0.4 * k, -0.3 * k)[:H, :H] for k in range(2)]).astype(np.float32)
    r0f = mover.shifted(0.0, 0.0)[:H, :H].astype(np.float32)
    down, across = np.array([R + 5]), np.array([R + 4])
    mask = np.zeros((H, H), bool)   # the constant area: all but `edge` rows or columns of the chip
    at = 5 + edge
    if side == 'right':
        mask[:, at:] = True
    elif side == 'left':
        mask[:, H - at:] = False
        mask[:, :H - at] = True
    elif side == 'below':
        mask[at:] = True
    else:
        mask[:H - at] = True
    frames[:, mask] = level
    shift = rng.uniform(0.1, 0.9, (2, 1, 1, 2)).astype(np.float32)
    win, norms = ref.reference_windows(r0f, down, across, W)
    f64 = torch.tensor(frames, dtype=torch.float64, requires_grad=True)
    s64 = torch.tensor(shift, dtype=torch.float64, requires_grad=True)
    chips = ref.chips(f64, s64, down, across, W, R)
    # deviations of the boxes about the constant level: exactly 0 where the box is constant
    with torch.no_grad():
        x = (chips.detach() - level).reshape(-1, 1, L, L)
        x[x.abs() < 1e-9] = 0.0
        ones = torch.ones((1, 1, W, W), dtype=torch.float64)
        s1, s2 = (torch.nn.functional.conv2d(t, ones) for t in (x, x * x))
        dev = (s2 - s1 * s1 / W ** 2).clamp(min=0).sqrt().view(2, 1, 1, M, M)
        inside = torch.nn.functional.conv2d((x != 0).double(), ones).view(dev.shape)
    flat = inside == 0
    assert flat.any()
    top = dev.max()
    good = dev > 0.3 * top
    rho64 = ref.surfaces(chips, win, norms, W)
    G = torch.as_tensor(rng.standard_normal((2, 1, 1, M, M)))
    g64 = torch.autograd.grad((rho64 * torch.where(good, G, torch.zeros_like(G))).sum(), (f64, s64))

    dc = DiffCorrelator(H, H, down, across, window=W, search=R)
    dc.set_reference(torch.as_tensor(r0f, device='cuda'))
    f = torch.tensor(frames, device='cuda', requires_grad=True)
    s = torch.tensor(shift, device='cuda', requires_grad=True)
    rho = dc.surface(f, s)
    got = rho.detach().cpu().double()
    assert (got[flat] == 0).all()
    some = ~flat & (dev > 1e-3 * top)   # (fewer digits than the bound has to spare below that)
    assert ((got - rho64.detach())[some].abs() * dev[some] / top).max() < 2e-5
    g = torch.autograd.grad((rho * torch.where(good | flat, G, torch.zeros_like(G)).to(rho)).sum(), (f, s))
    for a, b in zip(g, g64):
        assert float((a.cpu().double() - b).norm() / b.norm()) < 1e-4

    # the offsets, where the largest value stands at a textured box and clear of those at the others
    want = torch.where(some, rho64.detach(), torch.zeros_like(dev)).flatten(-2)
    best = want.max(-1)
    clear = torch.gather(good.flatten(-2), -1, best.indices[..., None])[..., 0] & (best.values > 0.1)
    weak = torch.where(good, torch.full_like(dev, -1.0), got).flatten(-2).max(-1).values
    clear &= weak < best.values - 1e-3
    out = dc.offsets(f, s).detach().cpu().double()
    o64 = ref.offsets(torch.where(some, rho64.detach(), torch.zeros_like(dev)), s64.detach(), R)
    # and curved there: an error of 2e-5 / 0.3 in the values moves a peak of second difference 0.2 by less than 1e-3
    for q in range(2):
        u, v = divmod(int(best.indices[q, 0, 0]), M)
        c = rho64.detach()[q, 0, 0]
        clear[q] &= (0 < u < M - 1 and 0 < v < M - 1 and bool(c[u - 1, v] - 2 * c[u, v] + c[u + 1, v] < -0.2)
                     and bool(c[u, v - 1] - 2 * c[u, v] + c[u, v + 1] < -0.2))
    peaks = torch.sort(want, -1).values
    clear &= peaks[..., -1] - peaks[..., -2] > 1e-3
    assert torch.equal(torch.isnan(out), torch.isnan(o64))
    assert float((out - o64)[clear].abs().max() if clear.any() else 0.0) < 1e-3
