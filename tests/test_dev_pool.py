"""The handles' memory pool: what it holds without a handle is bounded, and handles made and destroyed by several
threads at once, on streams of their own, give the results of one."""
import gc
import threading

import numpy as np
import pytest
import torch

from slipcam_b200 import framecor

pytestmark = pytest.mark.gpu


def correlate(ref, frames, search):
    down, across = framecor.window_grid(ref.shape[0], ref.shape[1], 32, search, 16)
    cor = framecor.Correlator(ref.shape[0], ref.shape[1], down, across, window=32, search=search)
    cor.set_reference(ref)
    return cor.correlate(frames)


def test_the_pool_is_bounded():
    """a handle with 2.5 GB of tables: at most 1 GiB stays (and 256 MiB for what else the first calls load)"""
    gen = torch.Generator(device='cuda').manual_seed(1)
    f = torch.randint(0, 256, (33, 2160, 3840), dtype=torch.uint8, device='cuda', generator=gen)
    down, across = np.array([100, 1200]), np.array([200, 3000])

    def use(n):
        cor = framecor.Correlator(2160, 3840, down, across, window=32, search=8)
        cor.set_reference(f[0])
        out = cor.correlate(f[1:1 + n])
        torch.cuda.synchronize()
        low = torch.cuda.mem_get_info()[0]
        del cor, out
        gc.collect()
        torch.cuda.synchronize()
        return low, torch.cuda.mem_get_info()[0]

    before = torch.cuda.mem_get_info()[0]
    low, after = use(32)
    assert before - after < (1 << 30) + (256 << 20)
    assert after - low > 1 << 30   # what was above the bound went back


@pytest.mark.parametrize('threads', [1, 4])
def test_handles_of_several_threads(threads):
    gen = torch.Generator(device='cuda').manual_seed(2)
    frames = torch.randint(0, 256, (4, 360, 640), dtype=torch.uint8, device='cuda', generator=gen)
    want = [{k: v.clone() for k, v in correlate(frames[0], frames[1:], s).items()} for s in (8, 16)]
    torch.cuda.synchronize()
    bad = []

    def work():
        stream = torch.cuda.Stream()
        for i in range(6):
            with torch.cuda.stream(stream):
                got = correlate(frames[0], frames[1:], (8, 16)[i % 2])
            stream.synchronize()
            bad.extend(k for k, v in got.items() if not torch.equal(v.nan_to_num(), want[i % 2][k].nan_to_num()))

    pool = [threading.Thread(target=work) for _ in range(threads)]
    for t in pool:
        t.start()
    for t in pool:
        t.join()
    assert not bad
