"""One-frame device calls on both sides of the lines between the kernels that
serve them.

Planes of many blocks take a warp per block (or a few blocks as one stream of
bin pairs), planes of few blocks a CTA per block, small planes one launch if
their output tiles are small enough; blocks with few rows take the forward
transform with a row per thread instead of two. Frame groups take none of the
first three, so that one frame per call must give their bytes; the wide blocks'
forward is held against the CPU restatement.
"""
import numpy as np
import pytest

from neo_fft3d_b200 import engine, synth
from neo_fft3d_b200.params import make_params, plane_descs
from oracle import restate

F = 7
SIZES = [(8, 8), (12, 12), (16, 16), (24, 24), (32, 32), (48, 48), (16, 24), (24, 16), (16, 32), (32, 16), (16, 48),
         (48, 16), (24, 32), (32, 24), (32, 48), (48, 32)]


def _clip(w, h, bits, seed):
    """Noise and a ramp (a clip that is quick to make)."""
    rng = np.random.default_rng(seed)
    a = rng.normal(110.0, 20.0, (F, h, w)) + np.linspace(0.0, 40.0, w) + np.arange(F)[:, None, None]
    if bits == 32:
        return (a / 255.0).clip(0.0, 1.0).astype(np.float32)
    return a.clip(0, 255).astype(np.uint8)


def _run(torch, a, bits, filt, group):
    h, w = a.shape[1:]
    dev = torch.from_numpy(a).cuda()
    out = torch.zeros_like(dev)
    torch.cuda.synchronize()
    pitch = w * a.itemsize
    e = engine.PlaneEngine(make_params(**filt), plane_descs([(h, w)], bits, F)[0])
    src = lambda m: dev[m].data_ptr() if 0 <= m < F else 0  # noqa: E731
    if group:
        e.filter_frames_device(0, [src(m) for m in range(-2, F + 2)], [pitch] * (F + 4), [out[m].data_ptr() for m in range(F)],
                               [pitch] * F)
    else:
        for n in range(F):
            e.filter_device(n, [src(n + d) for d in range(-2, 3)], [pitch] * 5, out[n].data_ptr(), pitch)
    e.synchronize()
    blocks = e.nblocks
    e.close()
    return out.cpu().numpy(), blocks


@pytest.mark.gpu
@pytest.mark.parametrize("bt", [-1, 0, 1, 2, 3, 4, 5])
@pytest.mark.parametrize("bw,bh", SIZES, ids=["%dx%d" % s for s in SIZES])
def test_many_blocks(gpu, bw, bh, bt):
    """More blocks than any line (67 x 63, no multiple of a warp's blocks), and
    a count between the lines of the shapes (31 x 29)."""
    import torch
    filt = dict(sigma=2.5, bt=bt, bw=bw, bh=bh, ow=bw // 2, oh=bh // 2)
    if bt != 0 or bw % 16 == 0:
        filt["sharpen"] = 0.4
    if bt == 0:
        filt["sigma2"] = 4.0  # noise by frequency
    for nox, noy in ((67, 63), (31, 29)):
        a = _clip((nox - 2) * (bw // 2) + bw // 2 - 1, (noy - 2) * (bh // 2) + bh // 2, 8, 70 + bt)
        one, blocks = _run(torch, a, 8, filt, False)
        assert blocks == nox * noy
        grp, _ = _run(torch, a, 8, filt, True)
        assert np.array_equal(one, grp), (nox, noy)


@pytest.mark.gpu
@pytest.mark.parametrize("w,h,bw,bh,ow,oh", [(273, 122, 24, 24, 2, 6), (272, 122, 24, 24, 2, 6), (201, 150, 32, 32, 10, 10),
                                             (202, 150, 32, 32, 10, 10), (401, 300, 48, 48, 16, 16), (400, 300, 48, 48, 2, 2),
                                             (121, 90, 16, 16, 0, 0)])
def test_tile_sizes(gpu, w, h, bw, bh, ow, oh):
    """Small planes whose output tiles lie on both sides of the one-launch
    frame's line (pixels of a tile over the pixels that go out together)."""
    import torch
    a = _clip(w, h, 8, 3)
    for bt in (1, 3):
        filt = dict(sigma=2.5, bt=bt, bw=bw, bh=bh, ow=ow, oh=oh)
        assert np.array_equal(_run(torch, a, 8, filt, False)[0], _run(torch, a, 8, filt, True)[0]), bt


@pytest.mark.gpu
@pytest.mark.parametrize("bits", [8, 32])
@pytest.mark.parametrize("bw,bh", [(32, 16), (48, 16), (48, 32), (24, 16)])
def test_wide_blocks_match_oracle(gpu, bw, bh, bits):
    import torch
    a = synth.make_clip(230, 117, F, noise_sigma=5.0, seed=12, planes=1)[0]
    if bits == 32:
        a = a.astype(np.float32) / 255.0
    filt = dict(sigma=2.5, bt=3, bw=bw, bh=bh, ow=bw // 2, oh=bh // 2, sharpen=0.3)
    want = restate.filter_clip([a], bits=bits, **filt)[0]
    for group in (False, True):
        got = _run(torch, a, bits, filt, group)[0]
        d = np.abs(got.astype(np.float64) - want.astype(np.float64)) * (255.0 if bits == 32 else 1.0)
        assert (d <= 1).mean() >= 0.999 and d.max() <= 3, ((d <= 1).mean(), d.max())
