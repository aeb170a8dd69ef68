"""Device calls whose output plane is a source plane.

A one-frame call may write its frame over the newest frame of its window (bt =
-1, 0, 1, 2: its own source; bt >= 3 at the clip's ends, where the window is one
frame), and over a frame whose spectrum the ring already holds. It must give
the bytes of separate buffers, for small planes (one launch per frame) and
larger ones (three launches), and leave the right spectra in the ring for the
frames that follow.
"""
import numpy as np
import pytest

from neo_fft3d_b200 import engine, synth
from neo_fft3d_b200.params import make_params, plane_descs

F = 9


def _run(torch, a, bits, filt, dst_of, pitch):
    """One frame per call over a clip in device rows of `pitch` bytes. dst_of(n):
    the frame of the source clip that output n is written over, None = a buffer
    of its own."""
    _, h, w = a.shape
    row = w * a.itemsize
    clip = np.zeros((F, h, pitch), np.uint8)
    clip[:, :, :row] = a.view(np.uint8).reshape(F, h, row)
    dev = torch.from_numpy(clip).cuda()
    out = torch.full_like(dev, 1)
    size = h * pitch
    e = engine.PlaneEngine(make_params(**filt), plane_descs([(h, w)], bits, F)[0])
    got = []
    src = lambda m: dev.data_ptr() + m * size if 0 <= m < F else 0  # noqa: E731
    for n in range(F):
        k = dst_of(n)
        dst = out if k is None else dev
        at = n if k is None else k
        e.filter_device(n, [src(n + d) for d in range(-2, 3)], [pitch] * 5, dst.data_ptr() + at * size, pitch)
        e.synchronize()
        got.append(dst[at, :, :row].cpu().numpy().copy())
    e.close()
    return got


# few blocks: one launch per frame; (448, 400) at 16 x 16: more than 450 blocks, three launches
@pytest.mark.gpu
@pytest.mark.parametrize("w,h,bw,ow,crop", [(176, 144, 32, 10, {}), (640, 480, 48, 16, {}), (121, 90, 16, 5, {}),
                                            (176, 144, 32, 16, dict(l=6, t=4, r=10, b=2)), (448, 400, 16, 8, {})])
@pytest.mark.parametrize("bt", [-1, 0, 1, 2, 3, 5])
@pytest.mark.parametrize("bits", [8, 16])
def test_one_frame_in_place(gpu, bits, bt, w, h, bw, ow, crop):
    import torch
    a = synth.make_clip(w, h, F, bits=bits, noise_sigma=5.0 * (1 << (bits - 8)), seed=60 + bt, planes=1)[0]
    filt = dict(sigma=2.5, bt=bt, bw=bw, bh=bw, ow=ow, oh=ow, **crop)
    if bt != 0:
        filt["sharpen"] = 0.4
    pitch = w * a.itemsize + 2  # (rows that end in a gap)
    want = _run(torch, a, bits, filt, lambda n: None, pitch)
    # (Kalman's frame 0 is a plain copy)
    got = _run(torch, a, bits, filt, lambda n: n if bt or n else None, pitch)
    for n in range(F):
        assert np.array_equal(want[n], got[n]), n
    if bt >= 3 and not crop:  # (crop borders come from the output's own source plane)
        # over the newest frame of the window. Its pixels are read by this call
        # alone (the later ones take the spectrum from the ring), up to the
        # clip's last frames, whose window is one frame
        last = (bt - 1) // 2
        over = lambda n: n + last if bt // 2 <= n < F - last else None  # noqa: E731
        got = _run(torch, a, bits, filt, over, pitch)
        for n in range(F):
            assert np.array_equal(want[n], got[n]), (n, "newest")
