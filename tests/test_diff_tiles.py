"""The differentiable kernels at the edges of their strips (16 chip rows), scans (32 grid columns) and column tiles,
against the float64 restatement and its autograd gradients."""
import numpy as np
import pytest
import torch

import diff_f64 as ref
from slipcam_b200 import synth
from slipcam_b200.diff import DiffCorrelator

pytestmark = pytest.mark.gpu


# (window, search): L = 10, 15, 16, 17, 32, 33; a grid of 55 columns whose column sums take two tiles; one of 61
@pytest.mark.parametrize('W,R', [(8, 1), (9, 3), (8, 4), (11, 3), (16, 8), (17, 8), (9, 27), (40, 30)])
def test_surface_adjoint_at_tile_edges(W, R):
    """FP32 kernels against FP64: the surface within 2e-5 (its own 1e-5 of the FFT, and the chips' rounding),
    the gradients within 1e-4 of their norm, the bounds that hold for these kernels at other sizes"""
    rng = np.random.default_rng(100 * W + R)
    H = W + 2 * R + 14
    mover = synth.Mover(synth.texture(H + 16, H + 16, 1.5, rng))
    frames = np.stack([mover.shifted(0.4 * k, -0.3 * k)[:H, :H] for k in range(2)]).astype(np.float32)
    r0f = mover.shifted(0.0, 0.0)[:H, :H].astype(np.float32)
    down, across = np.array([R, R + 11]), np.array([R + 1, R + 13])   # the interpolation leaves the frame at the edges
    shift = rng.uniform(0.1, 0.9, (2, 2, 2, 2)).astype(np.float32)
    M = 2 * R + 1
    G = torch.as_tensor(rng.standard_normal((2, 2, 2, M, M)))
    f64 = torch.tensor(frames, dtype=torch.float64, requires_grad=True)
    s64 = torch.tensor(shift, dtype=torch.float64, requires_grad=True)
    win, norms = ref.reference_windows(r0f, down, across, W)
    rho64 = ref.surfaces(ref.chips(f64, s64, down, across, W, R), win, norms, W)
    g64 = torch.autograd.grad((rho64 * G).sum(), (f64, s64))
    dc = DiffCorrelator(H, H, down, across, window=W, search=R)
    dc.set_reference(torch.as_tensor(r0f, device='cuda'))
    f = torch.tensor(frames, device='cuda', requires_grad=True)
    s = torch.tensor(shift, device='cuda', requires_grad=True)
    rho = dc.surface(f, s)
    g = torch.autograd.grad((rho * G.to(rho)).sum(), (f, s))
    assert float((rho.detach().cpu().double() - rho64.detach()).abs().max()) < 2e-5
    for a, b in zip(g, g64):
        assert float((a.cpu().double() - b).norm() / b.norm()) < 1e-4
