"""The filter/inverse kernels over block shapes, windows and run lengths.

One-frame calls and frame groups of every run length take different kernels
(a warp per block, a CTA for a few blocks with its spectra read or staged by
bulk copies, longer walks of a pair through the run's frames); all must give
the CPU restatement's pixels (>= 99.9 % within 1 LSB, none off by more than 3)
and one another's bytes. The planes have odd sizes, few blocks (fewer than a
CTA takes) or many, and 8- and 16-bit samples.
"""
import numpy as np
import pytest

from neo_fft3d_b200 import engine, synth
from neo_fft3d_b200.params import make_params, plane_descs
from oracle import restate

F = 13


def _filter(torch, a, bits, filt, sizes):
    """Plane [F, H, W] in groups of the given sizes (cycled); 0 = one-frame calls."""
    dev = torch.from_numpy(a.view(np.int16) if a.dtype == np.uint16 else a).cuda()
    out = torch.full_like(dev, 1)
    e = engine.PlaneEngine(make_params(**filt), plane_descs([a.shape[1:]], bits, F)[0])
    st = a.shape[2] * a.itemsize
    fb = a.shape[1] * st
    src = lambda n: dev.data_ptr() + n * fb if 0 <= n < F else 0  # noqa: E731
    n0, i = 0, 0
    while n0 < F:
        k = min(sizes[i % len(sizes)], F - n0)
        if k == 0:
            e.filter_device(n0, [src(n0 + d) for d in range(-2, 3)], [st] * 5, out.data_ptr() + n0 * fb, st)
            k = 1
        else:
            e.filter_frames_device(n0, [src(n) for n in range(n0 - 2, n0 + k + 2)], [st] * (k + 4),
                                   [out.data_ptr() + n * fb for n in range(n0, n0 + k)], [st] * k)
        n0 += k
        i += 1
    e.synchronize()
    e.close()
    got = out.cpu().numpy()
    return got.view(np.uint16) if a.dtype == np.uint16 else got


SHAPES = [(32, 32, 16, 16), (48, 48, 16, 16), (16, 16, 5, 7), (24, 24, 8, 8), (8, 8, 4, 4), (12, 12, 6, 6),
          (16, 32, 8, 10), (48, 16, 10, 5)]


@pytest.mark.gpu
@pytest.mark.parametrize("bt", [-1, 0, 1, 2, 3, 4, 5])
@pytest.mark.parametrize("bw,bh,ow,oh", SHAPES, ids=["%dx%d" % s[:2] for s in SHAPES])
def test_runs_match_oracle(gpu, bw, bh, ow, oh, bt):
    import torch
    bits = 16 if (bw + bt) % 3 == 0 else 8
    a = synth.make_clip(117, 83, F, bits=bits, noise_sigma=5.0 * (1 << (bits - 8)), seed=40 + bt, planes=1)[0]
    filt = dict(sigma=2.5, bt=bt, bw=bw, bh=bh, ow=ow, oh=oh)
    if bt != 0:
        filt.update(sharpen=0.4, dehalo=0.3 if bt % 2 else 0.0)
    if bt == 4:
        filt["degrid"] = 0.0
    want = restate.filter_clip([a], bits=bits, **filt)[0]
    ref = _filter(torch, a, bits, filt, [0])
    d = np.abs(ref.astype(int) - want.astype(int))
    assert (d <= 1).mean() >= 0.999 and d.max() <= 3, ((d <= 1).mean(), d.max())
    for sizes in ([13], [2], [3, 1, 5]):
        assert np.array_equal(ref, _filter(torch, a, bits, filt, sizes)), sizes


@pytest.mark.gpu
@pytest.mark.parametrize("w,h", [(24, 19), (33, 32), (65, 40), (640, 480), (801, 505)])
def test_block_counts(gpu, w, h):
    """From a single block step to more blocks than the chip holds CTAs (the
    blocks a CTA takes, its last CTA's remainder, and the change from CTAs to
    warps above 4000 blocks): frame groups equal one-frame calls."""
    import torch
    a = synth.make_clip(w, h, F, noise_sigma=5.0, seed=7, planes=1)[0]
    for bt in (1, 3, 5):
        filt = dict(sigma=2.5, bt=bt, bw=16, bh=16, ow=8, oh=8, sharpen=0.3)
        ref = _filter(torch, a, 8, filt, [0])
        assert np.array_equal(ref, _filter(torch, a, 8, filt, [8]))
        assert np.array_equal(ref, _filter(torch, a, 8, filt, [2, 7]))


@pytest.mark.gpu
@pytest.mark.parametrize("bits", [8, 16])
@pytest.mark.parametrize("w,bw,ow,crop", [(118, 16, 6, {}), (118, 16, 8, {}), (120, 32, 10, {}), (120, 16, 8, {}),
                                          (121, 16, 5, dict(l=3, t=2, r=6, b=4)), (126, 16, 8, dict(l=2, r=4, b=2)),
                                          (130, 16, 8, dict(t=5, b=1))])
def test_overlap_add_widths_and_borders(gpu, w, bw, ow, crop, bits):
    """1, 2 and 4 pixels a thread in the overlap-add, few and many rows, with
    crop borders copied from the source: against the restatement, and the
    whole group against one-frame calls."""
    import torch
    a = synth.make_clip(w, 90, F, bits=bits, noise_sigma=5.0 * (1 << (bits - 8)), seed=51, planes=1)[0]
    filt = dict(sigma=2.5, bt=3, bw=bw, bh=16, ow=ow, oh=5, **crop)
    want = restate.filter_clip([a], bits=bits, **filt)[0]
    ref = _filter(torch, a, bits, filt, [0])
    d = np.abs(ref.astype(int) - want.astype(int))
    assert (d <= 1).mean() >= 0.999 and d.max() <= 3, ((d <= 1).mean(), d.max())
    for sizes in ([13], [4]):
        assert np.array_equal(ref, _filter(torch, a, bits, filt, sizes)), sizes


@pytest.mark.gpu
@pytest.mark.parametrize("w,h", [(176, 144), (640, 480)])
def test_captured_call_replays(gpu, w, h):
    """A one-frame device call captured in a CUDA graph (small planes: one
    launch with arrival counters; larger ones: three launches) gives the frame
    of whatever its source holds at each replay."""
    import torch
    a = synth.make_clip(w, h, 4, noise_sigma=5.0, seed=9, planes=1)[0]
    filt = dict(sigma=2.5, bt=1, bw=32, bh=32, ow=16, oh=16, sharpen=0.3)
    want = [_filter_one(torch, a[k], filt) for k in range(4)]
    e = engine.PlaneEngine(make_params(**filt), plane_descs([a.shape[1:]], 8, 4)[0])
    src = torch.from_numpy(a[0]).cuda()
    out = torch.empty_like(src)
    s = torch.cuda.Stream()
    call = lambda n: e.filter_device(n, [0, 0, src.data_ptr(), 0, 0], [w] * 5, out.data_ptr(), w, s.cuda_stream)  # noqa: E731
    with torch.cuda.stream(s):
        call(0)  # kernels loaded, the plane's reset passed
        s.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            call(1)
        for k in (1, 2, 3, 0, 0):
            src.copy_(torch.from_numpy(a[k]))
            out.fill_(1)
            graph.replay()
            s.synchronize()
            assert np.array_equal(out.cpu().numpy(), want[k]), k
        # a plain call afterwards (which also records the plane's last work outside the capture)
        src.copy_(torch.from_numpy(a[2]))
        call(2)
        s.synchronize()
        assert np.array_equal(out.cpu().numpy(), want[2])
    del graph
    e.close()


def _filter_one(torch, frame, filt):
    e = engine.PlaneEngine(make_params(**filt), plane_descs([frame.shape], 8, 1)[0])
    src = torch.from_numpy(frame).cuda()
    out = torch.full_like(src, 1)
    w = frame.shape[1]
    e.filter_device(0, [0, 0, src.data_ptr(), 0, 0], [w] * 5, out.data_ptr(), w)
    e.synchronize()
    e.close()
    return out.cpu().numpy()
