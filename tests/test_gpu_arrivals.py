"""The arrival counters of fused overlap-adds (NEO_FFT3D_FUSED_OLA=1) after a
launch that failed: a CTA whose bounded wait ran out never counts its block, so
tiles keep part of their count. The hook that raises the error flag leaves the
counters like that; when the error has been reported, and after a reset, the
next calls must give the right frames (a frame group's run, and the one-launch
frame of a small plane, which shares the counters).
"""
import numpy as np
import pytest

from neo_fft3d_b200 import engine, synth
from neo_fft3d_b200.engine import FFT3DError
from neo_fft3d_b200.params import make_params, plane_descs

F = 12


def _group(e, dev, out, n0, k):
    h, w = dev.shape[1:]
    ptrs = [dev[m].data_ptr() if 0 <= m < F else 0 for m in range(n0 - 2, n0 + k + 2)]
    if k == 1:
        e.filter_device(n0, ptrs, [w] * 5, out[n0].data_ptr(), w)
    else:
        e.filter_frames_device(n0, ptrs, [w] * (k + 4), [out[m].data_ptr() for m in range(n0, n0 + k)], [w] * k)


@pytest.mark.gpu
@pytest.mark.parametrize("how", ["synchronize", "reset"])
@pytest.mark.parametrize("k", [1, 4])
@pytest.mark.parametrize("ow", [0, 10, 16])
def test_counters_after_a_failed_launch(gpu, monkeypatch, ow, k, how):
    import torch
    monkeypatch.setenv("NEO_FFT3D_FUSED_OLA", "1")
    a = synth.make_clip(200, 136, F, noise_sigma=5, seed=33, planes=1)[0]
    dev = torch.from_numpy(a).cuda()
    make = lambda: engine.PlaneEngine(make_params(sigma=2.5, bt=3, ow=ow, oh=ow),  # noqa: E731
                                      plane_descs([a.shape[1:]], 8, F)[0])
    want, got = torch.full_like(dev, 1), torch.full_like(dev, 1)
    torch.cuda.synchronize()
    ref = make()
    _group(ref, dev, want, 4, k)
    ref.synchronize()
    e = make()
    _group(e, dev, got, 0, 4)
    e.synchronize()
    engine.lib().fft3d_plane_debug_set_error_flag(e.h, 2)
    if how == "synchronize":
        with pytest.raises(FFT3DError):
            e.synchronize()
    else:
        e.reset()
    got.fill_(1)
    torch.cuda.synchronize()
    _group(e, dev, got, 4, k)
    torch.cuda.synchronize()
    assert np.array_equal(got[4:4 + k].cpu().numpy(), want[4:4 + k].cpu().numpy())
    ref.close()
    e.close()
