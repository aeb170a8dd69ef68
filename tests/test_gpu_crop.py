"""Crop borders of device calls: copied from the source plane to the output."""
import numpy as np
import pytest

from neo_fft3d_b200 import engine, synth
from neo_fft3d_b200.engine import FFT3DError
from neo_fft3d_b200.params import make_params, plane_descs


@pytest.mark.gpu
@pytest.mark.parametrize("w,h", [(160, 128), (640, 480)])  # one launch per frame, three launches
def test_overlapping_rows_are_refused(gpu, w, h):
    """A pitch below the row (rows that overlap) is refused for the planes that
    the borders' copy touches, in one-frame calls and frame groups, and nothing
    is written; without a crop the pitches are the caller's affair."""
    import torch
    a = synth.make_clip(w, h, 6, noise_sigma=5, seed=3, planes=1)[0]
    dev = torch.from_numpy(a).cuda()
    out = torch.full_like(dev, 1)
    torch.cuda.synchronize()
    for crop in (dict(l=6, t=4), dict(b=2), {}):
        e = engine.PlaneEngine(make_params(sigma=2.0, bt=1, bw=32, bh=32, ow=16, oh=16, **crop),
                               plane_descs([(h, w)], 8, 6)[0])
        one = lambda sp, dp: e.filter_device(0, [0, 0, dev.data_ptr(), 0, 0], [sp] * 5, out.data_ptr(), dp)  # noqa: E731
        two = lambda sp, dp: e.filter_frames_device(0, [0, 0, dev.data_ptr(), dev[1].data_ptr(), 0, 0],  # noqa: E731
                                                    [w, w, w, sp, w, w], [out.data_ptr(), out[1].data_ptr()], [w, dp])
        for call in (one, two):
            for sp, dp in ((w - 1, w), (w, w - 1), (0, w), (w, -w)):
                if crop:
                    with pytest.raises(FFT3DError, match=r"plane copy.*\(status -2\)"):
                        call(sp, dp)
                    e.synchronize()
                    assert int((out != 1).sum()) == 0
                elif (sp, dp) == (w - 1, w):
                    call(sp, dp)
            e.reset()
            call(w, w)
            e.synchronize()
            out.fill_(1)
            torch.cuda.synchronize()
        e.close()


def _rows(torch, planes, pitch, offset, fill):
    """The planes [n, h, row bytes] in device memory, rows `pitch` bytes apart
    from `offset` bytes on; the gaps hold `fill`."""
    n, h, row = planes.shape
    flat = torch.full((offset + n * h * pitch,), fill, dtype=torch.uint8, device="cuda")
    flat[offset:].view(n, h, pitch)[:, :, :row] = torch.from_numpy(planes).cuda()
    return flat


@pytest.mark.gpu
@pytest.mark.parametrize("bits", [8, 16, 32])
@pytest.mark.parametrize("w,crop", [(96, dict(l=2, r=3)), (96, dict(t=1)), (100, dict(l=17, t=3, r=1, b=5)),
                                    (121, dict(l=60, r=40, t=11, b=9)), (128, dict(l=16, r=32, t=30, b=30)),
                                    (83, dict(r=1, b=1)), (1500, dict(l=701, r=603, t=2, b=3))])
def test_borders_are_the_source(gpu, w, crop, bits):
    """Every border byte comes from the source, at every row alignment (1 to 16
    bytes, pointer offsets and pitches), the rows' gaps stay as they were, and
    the interior is that of unpadded rows; one frame per call and a group."""
    import torch
    h, n = 75, 4
    size = {8: 1, 16: 2, 32: 4}[bits]
    if bits == 32:
        a = synth.make_clip(w, h, n, noise_sigma=5, seed=5, planes=1)[0].astype(np.float32) / 255.0
    else:
        a = synth.make_clip(w, h, n, bits=bits, noise_sigma=5.0 * (1 << (bits - 8)), seed=5, planes=1)[0]
    row = w * size
    planes = np.ascontiguousarray(a).view(np.uint8).reshape(n, h, row)
    inside = np.zeros((h, row), bool)
    inside[crop.get("t", 0):h - crop.get("b", 0), crop.get("l", 0) * size:row - crop.get("r", 0) * size] = True
    assert inside.any()
    e = engine.PlaneEngine(make_params(sigma=2.0, bt=1, bw=16, bh=16, ow=8, oh=8, **crop),
                           plane_descs([(h, w)], bits, n)[0])
    first = None
    for spitch, soff, dpitch, doff in ((row, 0, row, 0), (-(-row // 16) * 16, 0, -(-row // 16) * 16 + 16, 0),
                                       (row + size, size, row + 2 * size, 0), (row + 8, 8, -(-row // 8) * 8, 0),
                                       (row + 3 * size, 0, row + 4 * size, 4 * size)):
        src = _rows(torch, planes, spitch, soff, 3)
        blank = np.full_like(planes, 7)
        for group in (1, n):
            out = _rows(torch, blank, dpitch, doff, 9)
            torch.cuda.synchronize()
            at = lambda m: src.data_ptr() + soff + m * h * spitch if 0 <= m < n else 0  # noqa: E731
            to = lambda m: out.data_ptr() + doff + m * h * dpitch  # noqa: E731
            e.reset()
            if group == 1:
                for m in range(n):
                    e.filter_device(m, [at(m + d) for d in range(-2, 3)], [spitch] * 5, to(m), dpitch)
            else:
                e.filter_frames_device(0, [at(m) for m in range(-2, n + 2)], [spitch] * (n + 4),
                                       [to(m) for m in range(n)], [dpitch] * n)
            e.synchronize()
            got = out.cpu().numpy()
            assert (got[:doff] == 9).all()
            got = got[doff:].reshape(n, h, dpitch)
            assert (got[:, :, row:] == 9).all()
            got = got[:, :, :row]
            assert np.array_equal(got[:, ~inside], planes[:, ~inside])
            if first is None:
                first = got.copy()
            assert np.array_equal(got, first)
    e.close()
