"""Which kernels the allocation-free call launches.

It has no error flag that a caller could read, so none of its kernels may hold
a wait that can run out: its filter/inverse kernel is the form that loads its
spectra itself, not the one that waits for bulk copies.
"""
import ctypes
import re

import pytest

from neo_fft3d_b200 import engine
from neo_fft3d_b200.params import FFT3DParams, PlaneDesc, make_params


def _kernels(torch, bits=8, **kw):
    """Names of the kernels of one call on a 160 x 120 plane."""
    fn = engine.lib().fft3d_filter2d_static
    fn.argtypes = [ctypes.POINTER(FFT3DParams), ctypes.POINTER(PlaneDesc), ctypes.c_void_p, ctypes.c_int,
                   ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p]
    fn.restype = ctypes.c_int
    src = torch.zeros((120, 160), dtype=torch.uint8 if bits == 8 else torch.float32, device="cuda")
    dst = torch.empty_like(src)
    pitch = 160 * src.element_size()
    p, d = make_params(sigma=3.0, **kw), PlaneDesc(160, 120, bits, 0, 0, 0, 1)
    call = lambda: fn(ctypes.byref(p), ctypes.byref(d), src.data_ptr(), pitch, dst.data_ptr(), pitch,  # noqa: E731
                      torch.cuda.current_stream().cuda_stream)
    assert call() == 0
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA], acc_events=True) as prof:
        assert call() == 0
        torch.cuda.synchronize()
    return [e.name for e in prof.events() if "fft3d" in e.name or "k_static" in e.name]


@pytest.mark.gpu
@pytest.mark.parametrize("bt", [1, -1])
@pytest.mark.parametrize("bw", [8, 16, 32, 48])
def test_static_filter_waits_for_nothing(gpu, bw, bt):
    import torch
    names = [n for n in _kernels(torch, bt=bt, bw=bw, bh=bw, ow=bw // 2, oh=bw // 2, sharpen=0.4) if "filter_inverse" in n]
    assert len(names) == 1, names
    if "k_filter_inverse_group" in names[0]:  # (a warp per block otherwise, which waits for nothing)
        staged = re.search(r"k_filter_inverse_group<\d+, \d+, -?\d+, (\w+)>", names[0])
        assert staged and staged.group(1) in ("false", "0"), names


@pytest.mark.gpu
def test_static_tables_of_small_blocks_go_up_in_less(gpu):
    """Blocks up to 32 x 32 (the default) send their tables in the smaller set of
    launch parameters, larger blocks in the large one."""
    import torch
    sent = {}
    for bw, bh, ow in ((8, 8, 4), (16, 32, 8), (32, 32, 16), (32, 32, 0), (32, 48, 16), (48, 48, 24)):
        names = [n for n in _kernels(torch, bt=1, bw=bw, bh=bh, ow=ow, oh=ow) if "k_static_tables" in n]
        assert len(names) == 1, names
        sent[bw, bh, ow] = int(re.search(r"k_static_tables<(\d+)>", names[0]).group(1))
    small, large = sent[8, 8, 4], sent[48, 48, 24]
    assert small < large
    assert [sent[k] for k in ((16, 32, 8), (32, 32, 16), (32, 32, 0), (32, 48, 16))] == [small, small, small, large], sent
