"""Handles and the device's memory: what is held without them, and handles that go while a stream is captured."""
import gc

import numpy as np
import pytest
import torch

from slipcam_b200 import framecor

pytestmark = pytest.mark.gpu


def make(height, width, window, search, skip):
    down, across = framecor.window_grid(height, width, window, search, skip)
    return framecor.Correlator(height, width, down, across, window=window, search=search)


def test_handle_goes_during_a_relaxed_capture():
    """
    A relaxed capture lets other calls that free memory pass, as cudaFree does: it stays valid when a handle is destroyed
    in it, and the handle's memory (some 300 MB of spectra) is there for the next one.
    """
    def used():
        gc.collect()
        torch.cuda.synchronize()
        return -torch.cuda.mem_get_info()[0]

    x = torch.zeros(8, device='cuda')
    held = []   # after each round; the first loads what captures need
    for _ in range(3):
        cor = make(720, 1280, 64, 48, 16)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, capture_error_mode='relaxed'):
            x.add_(1)
            del cor
            x.add_(1)
        graph.replay()
        del graph
        held.append(used())
    assert x.tolist() == [6.0] * 8
    assert held[2] - held[0] < 64 << 20


@pytest.mark.parametrize('frames', [1, 16])
def test_memory_of_several_handles(frames):
    """Handles of buffers that are each well below the bound, some GB in all: at most 1 GiB stays of them, and none
    of it after release_memory."""
    f = torch.randint(0, 256, (frames + 1, 720, 1280), dtype=torch.uint8, device='cuda')
    down, across = framecor.window_grid(720, 1280, 64, 48, 16)

    def round_():
        cors = [make(720, 1280, 64, 48, 16) for _ in range(5)]
        for cor in cors:
            cor.set_reference(f[0])
            cor.correlate(f[1:])
        torch.cuda.synchronize()
        low = torch.cuda.mem_get_info()[0]
        del cors, cor
        gc.collect()
        return low, torch.cuda.mem_get_info()[0]   # nothing synchronizes in between

    round_()   # loads what the calls need
    framecor.release_memory()
    before = torch.cuda.mem_get_info()[0]
    low, after = round_()
    assert before - low > 2 << 30
    assert before - after <= (1 << 30) + (4 << 20)
    framecor.release_memory()
    assert before - torch.cuda.mem_get_info()[0] <= 4 << 20


def test_release_memory_of_no_device():
    with pytest.raises(RuntimeError, match='could not be released'):
        framecor.release_memory(99)
