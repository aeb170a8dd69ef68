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
