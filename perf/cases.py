"""
The measured workloads of the b200 backend: what a program that uses it calls, from a single small
frame to the batches of the 720p and 1080p videos, each through the public entry points.

listed() gives the workloads, draw() more of the same ranges; prepare() makes what the program has in
hand before the call (frames made from the seed, the correlator with its reference set), run() is one
call with its whole outputs, work() the bytes and operations it cannot do without, and exact() the
outputs in 64 bits from plain torch and numpy.
"""

import math

import numpy as np
import torch

from slipcam_b200 import framecor, scans, stabilize
from slipcam_b200.diff import DiffCorrelator

DEV = 'cuda'


def listed():
    """The workloads. Sizes: the repository's own (bench.py, tests, synth.py) and generic odd ones."""
    def cor(name, height, width, window, search, skip, frames, gross='frame', host=False):
        return dict(name=name, kind='correlate', height=height, width=width, window=window, search=search,
                    skip=skip, frames=frames, gross=gross, host=host)
    return [
        # a live view: one small frame at a time, where launches and latency count
        cor('small_w32_one_frame', 360, 640, 32, 16, 16, 1, 'none'),
        # the everyday batch of a 720p video: camera motion per frame, a fault step; frames on the GPU
        cor('hd_w64_batch', 720, 1280, 64, 48, 16, 16),
        # the same from numpy frames in pageable memory, as the reference's callers pass them
        cor('hd_w64_host', 720, 1280, 64, 48, 16, 16, host=True),
        # a second pass around an offset map: every window has a search centre of its own
        cor('hd_w64_window_gross', 720, 1280, 64, 48, 16, 8, 'window'),
        # a cropped region: odd frame size (rows not on word boundaries), odd grid, no offsets
        cor('ragged_w48', 477, 853, 48, 21, 13, 5, 'none'),
        # a dense 1080p stream with large motion (transform size 192)
        cor('fullhd_w64_s64', 1080, 1920, 64, 64, 8, 4),
        # large windows of a low-contrast scene (transform size 256)
        cor('hd_w128_s64', 720, 1280, 128, 64, 16, 4, 'window'),
        # the check of a reference frame's texture: correlator, reference and surfaces in one call
        dict(name='periodicity_hd', kind='periodicity', height=720, width=1280, window=64, search=48, skip=16),
        # the camera's motion through a video, stabilize's defaults
        dict(name='coarse_track_hd', kind='coarse', height=720, width=1280, window=96, step=96, search=32, frames=64),
        # the frames of that video resampled onto the reference, text blanked
        dict(name='stabilize_hd', kind='stabilize', height=720, width=1280, frames=32),
        # the first look at a video: frame differences and the burned-in text
        dict(name='scans_hd', kind='scans', height=720, width=1280, frames=150),
        # a training step through the sub-pixel offsets: forward and backward to frames and shifts
        dict(name='diff_offsets', kind='diff', height=256, width=256, window=64, search=8, skip=32, frames=41),
    ]


def _log(rng, lo, hi):
    """a whole number spread over the logarithm of [lo, hi]"""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more workload of the same ranges."""
    what = rng.choice(['w32', 'w64', 'w64', 'w64', 'w64', 'stream', 'w128', 'periodicity', 'coarse', 'stabilize',
                       'scans', 'diff'])
    if what in ('w32', 'w64', 'stream', 'w128'):
        if what == 'w32':
            height, window, search, skip, frames = rng.randint(240, 720), rng.randint(24, 32), rng.randint(8, 24), rng.randint(10, 24), _log(rng, 1, 16)
        elif what == 'w64':
            height, window, search, skip, frames = rng.randint(360, 720), rng.randint(40, 72), rng.randint(16, 44), rng.randint(13, 32), _log(rng, 1, 16)
        elif what == 'stream':
            height, window, search, skip, frames = rng.randint(540, 1080), rng.randint(56, 66), rng.randint(52, 63), rng.randint(9, 24), rng.randint(1, 4)
        else:
            height, window, search, skip, frames = rng.randint(480, 720), rng.randint(100, 128), rng.randint(50, 64), rng.randint(16, 40), rng.randint(1, 4)
        width = height * 16 // 9 + rng.randint(-3, 3)
        return dict(kind='correlate', height=height, width=width, window=window, search=search, skip=skip, frames=frames,
                    gross=rng.choice(['none', 'frame', 'frame', 'window']), host=rng.random() < 0.25)
    height = rng.randint(360, 720)
    width = height * 16 // 9 + rng.randint(-3, 3)
    if what == 'periodicity':
        return dict(kind='periodicity', height=height, width=width, window=rng.randint(32, 64), search=rng.randint(16, 48),
                    skip=rng.randint(16, 32))
    if what == 'coarse':
        return dict(kind='coarse', height=height, width=width, window=2 * rng.randint(32, 48), step=rng.randint(72, 96),
                    search=rng.randint(16, 32), frames=rng.randint(8, 64))
    if what == 'stabilize':
        return dict(kind='stabilize', height=height, width=width, frames=rng.randint(2, 32))
    if what == 'scans':
        return dict(kind='scans', height=height, width=width, frames=rng.randint(30, 150))
    return dict(kind='diff', height=rng.randint(192, 256), width=rng.randint(192, 256), window=rng.randint(32, 64),
                search=rng.randint(6, 10), skip=rng.randint(24, 40), frames=rng.randint(2, 41))


# ---- inputs: the texture and motions of the videos (slipcam_b200/synth.py's distributions), on the GPU

def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _texture_spectrum(h, w, gen, sigma=2.0):
    """the spectrum of smoothed Gaussian noise rescaled to mean 128 and deviation 40, clipped to 0-255"""
    ky = torch.fft.fftfreq(h, dtype=torch.float64, device=DEV)[:, None]
    kx = torch.fft.fftfreq(w, dtype=torch.float64, device=DEV)[None, :]
    noise = torch.randn(h, w, generator=gen, dtype=torch.float64, device=DEV)
    t = torch.fft.ifft2(torch.fft.fft2(noise) * torch.exp(-2 * math.pi ** 2 * sigma ** 2 * (ky * ky + kx * kx))).real
    t = ((t - t.mean()) / t.std() * 40 + 128).clamp(0, 255)
    return torch.fft.fft2(t), ky, kx


def _moved(spec, ky, kx, dy, dx):
    return torch.fft.ifft2(spec * torch.exp(-2j * math.pi * (ky * dy + kx * dx))).real


def _video(h, w, n, gen, step_px, noise=2.0):
    """a reference frame and n frames (uint8) of a camera walking 0.5 px a frame past a fault at 30
    degrees whose far side has slipped by up to step_px; and the camera's motion (n, 2), numpy"""
    spec, ky, kx = _texture_spectrum(h, w, gen)
    y, x = torch.meshgrid(torch.arange(h, device=DEV), torch.arange(w, device=DEV), indexing='ij')
    far = (-(x - w / 2) * math.sin(math.pi / 6) + (y - h / 2) * math.cos(math.pi / 6)) > 0
    theta = torch.rand(n, generator=gen, dtype=torch.float64, device=DEV).cpu().numpy() * 2 * math.pi
    motion = np.cumsum(0.5 * np.stack([np.sin(theta), np.cos(theta)], 1), 0)
    frames = torch.empty((n + 1, h, w), dtype=torch.uint8, device=DEV)
    for k in range(n + 1):
        dy, dx = (0.0, 0.0) if k == 0 else motion[k - 1]
        img = _moved(spec, ky, kx, dy, dx)
        if k:
            img = torch.where(far, _moved(spec, ky, kx, dy, dx + step_px * k / n), img)
        img = img + noise * torch.randn(h, w, generator=gen, dtype=torch.float64, device=DEV)
        frames[k] = img.round().clamp(0, 255).to(torch.uint8)
    return frames[0].contiguous(), frames[1:].contiguous(), motion


def _camera(h, w, n, seed):
    """n uint8 frames of a camera moving over a textured scene with burned-in text, the reference in
    the middle; the frames, the similarity transforms (n, 4) and the text mask, numpy"""
    gen = _generator(seed)
    pad = 96
    spec, _, _ = _texture_spectrum(h + 2 * pad, w + 2 * pad, gen)
    scene = torch.fft.ifft2(spec).real.float()[None, None]
    ref = n // 2
    steps = torch.randn(n, 4, generator=gen, dtype=torch.float64, device=DEV).cpu().numpy() * (1.0, 1.0, 3e-4, 3e-4)
    params = np.zeros((n, 4))
    for k in range(ref + 1, n):
        params[k] = params[k - 1] + steps[k]
    for k in range(ref - 1, -1, -1):
        params[k] = params[k + 1] + steps[k]
    yy, xx = torch.meshgrid(torch.arange(h, device=DEV, dtype=torch.float64) - h / 2,
                            torch.arange(w, device=DEV, dtype=torch.float64) - w / 2, indexing='ij')
    boxes = [(w // 8, 8, w // 2, 24), (w // 10, h - 40, w // 3, h - 20)]
    text = np.zeros((h, w), bool)
    frames = torch.empty((n, h, w), dtype=torch.uint8, device=DEV)
    for k in range(n):
        p, q, a, s = params[k]
        det = (1 + s) ** 2 + a ** 2   # the scene point seen at each pixel: the transform's inverse
        zx, zy = xx - p, yy - q
        gx = ((1 + s) * zx + a * zy) / det + w / 2 + pad
        gy = (-a * zx + (1 + s) * zy) / det + h / 2 + pad
        g = torch.stack([gx / (w + 2 * pad - 1) * 2 - 1, gy / (h + 2 * pad - 1) * 2 - 1], -1)[None].float()
        img = torch.nn.functional.grid_sample(scene, g, mode='bicubic', padding_mode='border', align_corners=True)[0, 0]
        img = img + torch.randn(h, w, generator=gen, device=DEV)
        for x0, y0, x1, y1 in boxes:   # a bright outline around dark strokes, the same in every frame
            img[y0:y1, x0:x1] = 30.0
            img[y0:y0 + 2, x0:x1] = img[y1 - 2:y1, x0:x1] = 240.0
            img[y0:y1, x0:x0 + 2] = img[y0:y1, x1 - 2:x1] = 240.0
            img[y0 + 4:y1 - 4:4, x0 + 4:x1 - 4] = 220.0
            text[y0:y1, x0:x1] = True
        frames[k] = img.round().clamp(0, 255).to(torch.uint8)
    return frames, params, text, ref


def _correlate_inputs(case, seed):
    """the reference, the frames (CUDA, uint8), the grid and the gross offsets (numpy or None)"""
    gen = _generator(seed)
    h, w, n = case['height'], case['width'], case['frames']
    ref, frames, motion = _video(h, w, n, gen, 0.6 * case['search'])
    down, across = framecor.window_grid(h, w, case['window'], case['search'], case['skip'])
    gross = None
    if case['gross'] == 'frame':
        gross = np.rint(motion).astype(np.int32)
    elif case['gross'] == 'window':   # an earlier map: the camera's motion give or take a few pixels
        jitter = torch.randint(-6, 7, (n, len(down), len(across), 2), generator=gen, device=DEV).cpu().numpy()
        gross = (np.rint(motion)[:, None, None, :] + jitter).astype(np.int32)
    return ref, frames, down, across, gross


def _diff_inputs(case, seed):
    gen = _generator(seed)
    h, w, n = case['height'], case['width'], case['frames']
    spec, ky, kx = _texture_spectrum(h, w, gen)
    shifts = (torch.rand(n, 2, generator=gen, dtype=torch.float64, device=DEV) * 6 - 3).cpu().numpy()
    ref = torch.fft.ifft2(spec).real.float()
    frames = torch.stack([_moved(spec, ky, kx, *s) for s in shifts])
    frames = (frames + torch.randn(n, h, w, generator=gen, dtype=torch.float64, device=DEV)).float()
    down, across = framecor.window_grid(h, w, case['window'], case['search'], case['skip'], margin=4)
    shape = (n, len(down), len(across), 2)
    shift = torch.rand(shape, generator=gen, dtype=torch.float64, device=DEV).float() * 2 - 1
    target = torch.as_tensor(shifts, device=DEV).float()[:, None, None, :].expand(shape).contiguous()
    return ref, frames, shift, target, down, across


def prepare(case, seed):
    """What the program has before the call: its frames, and the correlator with its reference set."""
    kind = case['kind']
    if kind == 'correlate':
        ref, frames, down, across, gross = _correlate_inputs(case, seed)
        cor = framecor.Correlator(case['height'], case['width'], down, across, window=case['window'],
                                  search=case['search'], backend='b200')
        if case['host']:
            ref, frames = ref.cpu().numpy(), frames.cpu().numpy()
        elif gross is not None:
            gross = torch.as_tensor(gross).to(DEV)
        cor.set_reference(ref)
        return dict(kind=kind, cor=cor, frames=frames, gross=gross)
    if kind == 'periodicity':
        ref, _, _ = _video(case['height'], case['width'], 1, _generator(seed), 0.0)
        down, across = framecor.window_grid(case['height'], case['width'], case['window'], case['search'], case['skip'])
        return dict(kind=kind, ref=ref, down=down, across=across, window=case['window'], search=case['search'])
    if kind == 'coarse':
        frames, _, text, ref = _camera(case['height'], case['width'], case['frames'], seed)
        return dict(kind=kind, frames=frames, text=text, ref=ref, window=case['window'], step=case['step'],
                    search=case['search'])
    if kind == 'stabilize':
        frames, params, text, _ = _camera(case['height'], case['width'], case['frames'], seed)
        return dict(kind=kind, frames=frames, params=params, text=text)
    if kind == 'scans':
        frames, _, _, _ = _camera(case['height'], case['width'], case['frames'], seed)
        return dict(kind=kind, frames=frames)
    ref, frames, shift, target, down, across = _diff_inputs(case, seed)
    dc = DiffCorrelator(case['height'], case['width'], down, across, window=case['window'], search=case['search'])
    dc.set_reference(ref)
    return dict(kind=kind, dc=dc, frames=frames.requires_grad_(), shift=shift.requires_grad_(), target=target)


def run(state):
    """One call of the program, its outputs whole."""
    kind = state['kind']
    if kind == 'correlate':
        return state['cor'].correlate(state['frames'], gross=state['gross'])
    if kind == 'periodicity':
        return framecor.periodicity(state['ref'], state['down'], state['across'], state['window'], state['search'])
    if kind == 'coarse':
        params, used, count = stabilize.coarse_track(state['frames'], state['ref'], state['text'], window=state['window'],
                                                     step=state['step'], search=state['search'])
        return dict(params=params, used=used, count=count)
    if kind == 'stabilize':
        frames, union = stabilize.stabilize(state['frames'], state['params'], state['text'])
        return dict(frames=frames, union=union)
    if kind == 'scans':
        return dict(differences=scans.frame_differences(state['frames']), mask=scans.text_mask(state['frames'], 0))
    offsets = state['dc'].offsets(state['frames'], state['shift'])
    loss = (offsets - state['target']).square().mean()
    grad_frames, grad_shift = torch.autograd.grad(loss, (state['frames'], state['shift']))
    return dict(offsets=offsets, loss=loss, grad_frames=grad_frames, grad_shift=grad_shift)


def _grid_size(case, margin=0):
    down, across = framecor.window_grid(case['height'], case['width'], case['window'], case['search'], case['skip'], margin)
    return len(down) * len(across)


def work(case):
    """Bytes: each input read once, each output written once. Flops of a correlation: a real 2-D
    transform of its search window, the product with the reference's spectrum, and the inverse."""
    kind = case['kind']
    pixels = case['height'] * case['width']

    def fft(L):
        return 2 * 2.5 * L * L * math.log2(L * L) + 6 * L * (L // 2 + 1)
    if kind == 'correlate':
        nwin, n, L = _grid_size(case), case['frames'], case['window'] + 2 * case['search']
        gross = {'none': 0, 'frame': 8 * n, 'window': 8 * n * nwin}[case['gross']]
        return dict(bytes=n * pixels + nwin * case['window'] ** 2 + 28 * n * nwin + gross, flops=n * nwin * fft(L))
    if kind == 'periodicity':
        nwin, L = _grid_size(case), case['window'] + 2 * case['search']
        return dict(bytes=pixels + 8 * nwin, flops=1.5 * nwin * fft(L))
    if kind == 'coarse':
        half = case['window'] // 2
        yc, xc = stabilize.template_grid(case['height'], case['width'], case['window'], case['step'], case['search'])
        L = 2 * half + 2 * case['search']
        return dict(bytes=case['frames'] * (pixels + 40), flops=case['frames'] * len(yc) * len(xc) * fft(L))
    if kind == 'stabilize':   # blanking and a bilinear tap per pixel
        return dict(bytes=2 * case['frames'] * pixels + 2 * pixels, flops=30 * case['frames'] * pixels)
    if kind == 'scans':
        return dict(bytes=case['frames'] * pixels + pixels, flops=6 * case['frames'] * pixels)
    pairs, L = case['frames'] * _grid_size(case, 4), case['window'] + 2 * case['search']
    return dict(bytes=8 * case['frames'] * pixels + 40 * pairs, flops=3 * pairs * fft(L) + 72 * pairs * L * L)


# ---- the outputs in 64 bits

def _surfaces(chips, windows):
    """the normalized correlation (B, M, M) of zero-mean windows (B, W, W) over chips (B, L, L), float64"""
    L, W = chips.shape[-1], windows.shape[-1]
    M = L - W + 1
    r0 = windows - windows.mean((-2, -1), keepdim=True)
    x = chips - chips.mean((-2, -1), keepdim=True)
    c = torch.fft.irfft2(torch.fft.rfft2(x) * torch.fft.rfft2(r0, s=(L, L)).conj(), s=(L, L))[..., :M, :M]

    def box(a):
        s = torch.nn.functional.pad(a.cumsum(-1).cumsum(-2), (1, 0, 1, 0))
        return s[..., W:, W:] - s[..., :M, W:] - s[..., W:, :M] + s[..., :M, :M]
    var = box(x * x) - box(x) ** 2 / (W * W)
    norm = r0.square().sum((-2, -1)).sqrt()[..., None, None]
    ok = (var > 1e-6) & (norm > 0)
    return torch.where(ok, c / (norm * torch.where(ok, var, torch.ones_like(var)).sqrt()), torch.zeros_like(c))


def _cut(frame, y, x, size):
    """the size x size boxes of the frame at (y, x), vectors of rows and columns"""
    i = torch.arange(size, device=frame.device)
    return frame[(y[:, None] + i)[:, :, None], (x[:, None] + i)[:, None, :]]


def _subpixel(f):
    """(du, dv) of the 3 x 3 values f (B, 3, 3): the quadratic fit, else a parabola per axis"""
    c1 = (f[:, 2].sum(-1) - f[:, 0].sum(-1)) / 6
    c2 = (f[:, :, 2].sum(-1) - f[:, :, 0].sum(-1)) / 6
    c3 = (f[:, 0].sum(-1) + f[:, 2].sum(-1) - 2 * f[:, 1].sum(-1)) / 6
    c5 = (f[:, :, 0].sum(-1) + f[:, :, 2].sum(-1) - 2 * f[:, :, 1].sum(-1)) / 6
    c4 = (f[:, 2, 2] - f[:, 2, 0] - f[:, 0, 2] + f[:, 0, 0]) / 4
    det = 4 * c3 * c5 - c4 * c4
    safe = torch.where(det > 0, det, torch.ones_like(det))
    du, dv = (c4 * c2 - 2 * c5 * c1) / safe, (c4 * c1 - 2 * c3 * c2) / safe
    fitted = (c3 < 0) & (det > 0) & (du.abs() <= 1) & (dv.abs() <= 1)

    def parabola(m, c, p):
        den = m - 2 * c + p
        return torch.where(den < 0, 0.5 * (m - p) / torch.where(den < 0, den, -torch.ones_like(den)), torch.zeros_like(den))
    return (torch.where(fitted, du, parabola(f[:, 0, 1], f[:, 1, 1], f[:, 2, 1])),
            torch.where(fitted, dv, parabola(f[:, 1, 0], f[:, 1, 1], f[:, 1, 2])))


def _around(s, u, v):
    """the 3 x 3 values around (u, v) of the surfaces s, the centre moved inside them"""
    M = s.shape[-1]
    d = torch.arange(-1, 2, device=s.device)
    b = torch.arange(len(s), device=s.device)
    uc, vc = u.clamp(1, M - 2), v.clamp(1, M - 2)
    return s[b[:, None, None], (uc[:, None] + d)[:, :, None], (vc[:, None] + d)[:, None, :]]


def _peaks(s, R, gross, tsize, stat=21):
    """offsets, peak, snr and cov of the surfaces s (B, M, M)"""
    B, M = len(s), s.shape[-1]
    f0, at = s.flatten(1).max(1)
    at = (s.flatten(1) == f0[:, None]).to(torch.uint8).argmax(1)
    u, v = at // M, at % M
    inside = (u > 0) & (u < M - 1) & (v > 0) & (v < M - 1)
    f = _around(s, u, v)
    du, dv = _subpixel(f)
    zero = torch.zeros_like(du)
    offsets = torch.stack([gross[:, 0] + u - R + torch.where(inside, du, zero),
                           gross[:, 1] + v - R + torch.where(inside, dv, zero)], -1)
    n = min(stat, M)
    i0, j0 = (u - n // 2).clamp(min=0), (v - n // 2).clamp(min=0)
    i1, j1 = (u - n // 2 + n).clamp(max=M), (v - n // 2 + n).clamp(max=M)
    rows = torch.arange(M, device=s.device)
    my = ((rows >= i0[:, None]) & (rows < i1[:, None])).double()
    mx = ((rows >= j0[:, None]) & (rows < j1[:, None])).double()
    total = torch.einsum('bij,bi,bj->b', s * s, my, mx)
    count = (i1 - i0) * (j1 - j0)
    mean = (total - f0 * f0) / (count - 1).clamp(min=1)
    snr = torch.where(mean > 0, f0 * f0 / torch.where(mean > 0, mean, torch.ones_like(mean)), zero)
    T = float(tsize)
    dxx = -(f[:, 2, 1] + f[:, 0, 1] - 2 * f0) * T
    dyy = -(f[:, 1, 2] + f[:, 1, 0] - 2 * f0) * T
    dxy = (f[:, 2, 2] + f[:, 0, 0] - f[:, 2, 0] - f[:, 0, 2]) * 0.25 * T
    n2 = (1 - f0).clamp(min=0)
    n4 = n2 * n2 * 0.5 * T
    n2 = 2 * n2
    w = dxy * dxy - dxx * dyy
    has = inside & (w.abs() >= 1e-2)
    w2 = torch.where(has, w * w, torch.ones_like(w))
    cov = torch.stack([(-n2 * w * dyy + n4 * (dyy * dyy + dxy * dxy)) / w2,
                       (-n2 * w * dxx + n4 * (dxx * dxx + dxy * dxy)) / w2,
                       (n2 * w * dxy - n4 * (dxx + dyy) * dxy) / w2], -1)
    flat = torch.tensor([99.0, 99.0, 0.0], dtype=torch.float64, device=s.device)
    cov = torch.where(has[:, None], cov, flat)
    ok = f0 > 0
    nan = torch.full_like(offsets, float('nan'))
    return (torch.where(ok[:, None], offsets, nan), torch.where(ok, f0, zero), torch.where(ok, snr, zero),
            torch.where(ok[:, None], cov, flat))


def _exact_correlate(case, seed):
    ref, frames, down, across, gross = _correlate_inputs(case, seed)
    h, w, n, W, R = case['height'], case['width'], case['frames'], case['window'], case['search']
    L, ny, nx = W + 2 * R, len(down), len(across)
    nwin = ny * nx
    y = torch.as_tensor(np.repeat(down, nx), device=DEV)
    x = torch.as_tensor(np.tile(across, ny), device=DEV)
    g = np.zeros((n, ny, nx, 2), np.int64) if gross is None else np.broadcast_to(
        gross[:, None, None, :] if gross.ndim == 2 else gross, (n, ny, nx, 2))
    g = torch.as_tensor(np.ascontiguousarray(g).reshape(n, nwin, 2), device=DEV).long()
    out = dict(offsets=torch.full((n, nwin, 2), float('nan'), dtype=torch.float64, device=DEV),
               peak=torch.zeros((n, nwin), dtype=torch.float64, device=DEV),
               snr=torch.zeros((n, nwin), dtype=torch.float64, device=DEV),
               cov=torch.tensor([99.0, 99.0, 0.0], dtype=torch.float64, device=DEV).repeat(n, nwin, 1))
    refd = ref.double()
    some = max(1, (1 << 25) // (L * L))
    for k in range(n):
        fk = frames[k].double()
        sy, sx = y + g[k, :, 0] - R, x + g[k, :, 1] - R
        fits = ((sy >= 0) & (sx >= 0) & (sy + L <= h) & (sx + L <= w)).nonzero()[:, 0]
        for a in range(0, len(fits), some):
            i = fits[a:a + some]
            s = _surfaces(_cut(fk, sy[i], sx[i], L), _cut(refd, y[i], x[i], W))
            for key, val in zip(('offsets', 'peak', 'snr', 'cov'), _peaks(s, R, g[k, i], W * W)):
                out[key][k, i] = val
    shape = (n, ny, nx)
    return dict(offsets=out['offsets'].view(*shape, 2), peak=out['peak'].view(shape), snr=out['snr'].view(shape),
                cov=out['cov'].view(*shape, 3))


def _exact_periodicity(case, seed, exclude=5):
    state = prepare(case, seed)
    W, R, down, across = case['window'], case['search'], state['down'], state['across']
    ref = state['ref'].double()
    y = torch.as_tensor(np.repeat(down, len(across)), device=DEV)
    x = torch.as_tensor(np.tile(across, len(down)), device=DEV)
    out, some = [], max(1, (1 << 25) // (W + 2 * R) ** 2)
    for a in range(0, len(y), some):
        s = _surfaces(_cut(ref, y[a:a + some] - R, x[a:a + some] - R, W + 2 * R), _cut(ref, y[a:a + some], x[a:a + some], W))
        local = torch.nn.functional.max_pool2d(s[:, None], 5, 1, 2)[:, 0]
        peak = s == local
        peak[:, R - exclude:R + exclude + 1, R - exclude:R + exclude + 1] = False
        best = torch.where(peak, s, torch.full_like(s, -2.0)).flatten(1).max(1).values
        out.append(torch.where(best > -2, best, torch.zeros_like(best)))
    return torch.cat(out).view(len(down), len(across)).cpu().numpy()


def _exact_fit(dx, dy, x, y):
    """the robust similarity fit of the offsets: three rounds of least squares"""
    use = np.isfinite(dx) & np.isfinite(dy)
    m = np.full(4, np.nan)
    for _ in range(3):
        if use.sum() < 4:
            return np.full(4, np.nan)
        o, z = np.ones(use.sum()), np.zeros(use.sum())
        G = np.vstack([np.column_stack([o, z, -y[use], x[use]]), np.column_stack([z, o, x[use], y[use]])])
        m = np.linalg.lstsq(G, np.concatenate([dx[use], dy[use]]), rcond=None)[0]
        rx, ry = dx[use] - (m[0] - m[2] * y[use] + m[3] * x[use]), dy[use] - (m[1] + m[2] * x[use] + m[3] * y[use])
        r = np.concatenate([rx, ry])
        limit = max(3 * 1.4826 * np.median(np.abs(r - np.median(r))), 0.3)
        use[np.flatnonzero(use)] = (np.abs(rx) < limit) & (np.abs(ry) < limit)
    return m


def _exact_coarse(case, seed, min_peak=0.5):
    frames, _, text, ref = _camera(case['height'], case['width'], case['frames'], seed)
    n, h, w = frames.shape
    W, R = case['window'], case['search']
    half, L, M = W // 2, W + 2 * R, 2 * R + 1
    yc, xc = np.arange(R + half, h - R - half, case['step']), np.arange(R + half, w - R - half, case['step'])
    cy, cx = (v.ravel() for v in np.meshgrid(yc, xc, indexing='ij'))
    img = frames[ref].double()
    wins = _cut(img, torch.as_tensor(cy - half, device=DEV), torch.as_tensor(cx - half, device=DEV), W)
    clear = np.array([not text[b - half:b + half, a - half:a + half].any() for b, a in zip(cy, cx)])
    keep = clear & (wins.flatten(1).std(1, correction=0) > 2).cpu().numpy()
    cy, cx, wins = cy[keep], cx[keep], wins[torch.as_tensor(keep, device=DEV)]
    X, Y = cx - w / 2, cy - h / 2
    params = np.full((n, 4), np.nan)
    params[ref] = 0
    for order in (range(ref + 1, n), range(ref - 1, -1, -1)):
        p = np.zeros(4)
        for k in order:
            left = np.rint(X + p[0] - p[2] * Y + p[3] * X + w / 2).astype(int) - half - R
            top = np.rint(Y + p[1] + p[2] * X + p[3] * Y + h / 2).astype(int) - half - R
            i = np.flatnonzero((top >= 0) & (left >= 0) & (top + L <= h) & (left + L <= w))
            dx, dy = np.full(len(cx), np.nan), np.full(len(cx), np.nan)
            if len(i):
                s = _surfaces(_cut(frames[k].double(), torch.as_tensor(top[i], device=DEV),
                                   torch.as_tensor(left[i], device=DEV), L), wins[torch.as_tensor(i, device=DEV)])
                f0, at = s.flatten(1).max(1)
                u, v = at // M, at % M
                f = _around(s, u, v)

                def vertex(a, b, c, ok):
                    den = a - 2 * b + c
                    return torch.where(ok & (den.abs() >= 1e-12), 0.5 * (a - c) / den, torch.zeros_like(den))
                oy = (u + vertex(f[:, 0, 1], f[:, 1, 1], f[:, 2, 1], (u > 0) & (u < M - 1)) - R).cpu().numpy()
                ox = (v + vertex(f[:, 1, 0], f[:, 1, 1], f[:, 1, 2], (v > 0) & (v < M - 1)) - R).cpu().numpy()
                good = (f0 >= min_peak).cpu().numpy()
                i, oy, ox = i[good], oy[good], ox[good]
                dx[i] = left[i] + R + half + ox - w / 2 - X[i]
                dy[i] = top[i] + R + half + oy - h / 2 - Y[i]
            fit = _exact_fit(dx, dy, X, Y)
            p = fit if np.isfinite(fit).all() else p
            params[k] = p
    return dict(params=params, used=None, count=None)


def _exact_scans(case, seed):
    frames, _, _, _ = _camera(case['height'], case['width'], case['frames'], seed)
    diff = [(frames[k + 1].long() - frames[k].long()).abs().sum().item() / frames[0].numel() for k in range(len(frames) - 1)]
    return dict(differences=np.asarray(diff), mask=None)


def _exact_diff(case, seed):
    ref, frames, shift, target, down, across = _diff_inputs(case, seed)
    n, h, w = frames.shape
    W, R = case['window'], case['search']
    ny, nx, L, M = len(down), len(across), W + 2 * R, 2 * R + 1
    x64 = frames.double().requires_grad_()
    t = shift.double().requires_grad_()

    def weights(q):   # Keys' six-point cubic convolution, the taps at -2 .. 3
        k1, k2, k3 = (lambda a: (4 / 3 * a - 7 / 3) * a * a + 1), (lambda a: ((-7 / 12 * a + 3) * a - 59 / 12) * a + 2.5), \
            (lambda a: ((1 / 12 * a - 2 / 3) * a + 1.75) * a - 1.5)
        return torch.stack([k3(q + 2), k2(q + 1), k1(q), k1(1 - q), k2(2 - q), k3(3 - q)], -1)
    y = torch.as_tensor(np.repeat(down, nx), device=DEV)
    x = torch.as_tensor(np.tile(across, ny), device=DEV)
    base = torch.floor(t.detach())
    wy, wx = weights((t - base)[..., 0]).view(n, ny * nx, 6), weights((t - base)[..., 1]).view(n, ny * nx, 6)
    i = torch.arange(L + 5, device=DEV)
    offsets = []
    wins = _cut(ref.double(), y, x, W)
    for k in range(n):
        b = base[k].view(-1, 2).long()
        rows = (y + b[:, 0] - R - 2)[:, None] + i
        cols = (x + b[:, 1] - R - 2)[:, None] + i
        c = x64[k][rows.clamp(0, h - 1)[:, :, None], cols.clamp(0, w - 1)[:, None, :]]
        c = sum(wy[k, :, d, None, None] * c[:, d:d + L] for d in range(6))
        c = sum(wx[k, :, d, None, None] * c[:, :, d:d + L] for d in range(6))
        s = _surfaces(c, wins)
        at = s.detach().flatten(1).argmax(1)
        u, v = at // M, at % M
        inside = ((u > 0) & (u < M - 1) & (v > 0) & (v < M - 1)).double()
        du, dv = _subpixel(_around(s, u, v))
        offsets.append(torch.stack([u - R + du * inside, v - R + dv * inside], -1).view(ny, nx, 2) + t[k])
    offsets = torch.stack(offsets)
    loss = (offsets - target.double()).square().mean()
    gf, gs = torch.autograd.grad(loss, (x64, t))
    return dict(offsets=offsets.detach(), loss=loss.detach(), grad_frames=gf, grad_shift=gs)


def exact(case, seed):
    """run's outputs for prepare(case, seed) in 64 bits; None for whole-number outputs."""
    kind = case['kind']
    if kind == 'stabilize':   # bytes and truth values
        return None
    return dict(correlate=_exact_correlate, periodicity=_exact_periodicity, coarse=_exact_coarse, scans=_exact_scans,
                diff=_exact_diff)[kind](case, seed)
