"""RGB8 stitching (hm-cupano_gb300/csrc/hmp_rgb.cu) where it changes path, bit for bit against the
oracle: every kind, one to seven levels, blend regions with and without copy blocks (the switch gives
the same bits), odd canvases, frames and canvases at odd addresses and odd row pitches, seam values
and labels no image has, table entries outside the frames, frames past the resolved offsets' range, and
a captured call."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import make_stitcher, masks_for_rig

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    import build as hmp_build

    hmp_build.build()


def _rig(n, kind, w, h, seed, **kw):
    from hmpano import synth

    overlap = kw.pop("overlap", 0.22)
    return synth.make_rig(canvas_w=w, canvas_h=h, n=n, src_w=w // n + 120, src_h=int(h * 0.9), overlap=overlap, seed=seed,
                          kind=kind, **kw)


def _frames(rig, seed, batch):
    from hmpano import synth

    return [np.ascontiguousarray(f[..., :3]) for f in synth.rig_frames(rig, seed=seed, batch=batch)]


def _odd(f, pitch_extra=0):
    """The frames on the GPU one byte past the allocation's start, rows `pitch_extra` bytes apart."""
    import torch

    b, h, w, c = f.shape
    pitch = w * c + pitch_extra
    buf = torch.zeros(1 + b * h * pitch, dtype=torch.uint8, device="cuda")
    t = buf[1:].as_strided((b, h, w, c), (h * pitch, pitch, c, 1))
    t.copy_(torch.from_numpy(f).cuda())
    return t


def _check(rig, kind, levels, batch=1, minimize=True, pitch_extra=0):
    import torch
    from oracle import oracle

    frames = _frames(rig, 5, batch)
    st = make_stitcher(kind, masks_for_rig(rig), levels, batch, minimize=minimize)
    ref = oracle.Stitch.from_rig(rig, levels, batch, minimize_blend=minimize).run(frames)
    canvas = _odd(np.full(ref.shape, 77, np.uint8), pitch_extra)
    st._run([_odd(f, pitch_extra) for f in frames], canvas)
    torch.cuda.synchronize()
    out = canvas.cpu().numpy()
    if not np.array_equal(out, ref):
        d = np.argwhere((out != ref).any(-1))
        pytest.fail(f"{len(d)} pixels differ, first {d[:4].tolist()}: {[(out[tuple(i)], ref[tuple(i)]) for i in d[:2]]}")
    return st, frames, ref


@pytest.mark.parametrize("levels", [1, 2, 5, 7])
@pytest.mark.parametrize("n,kind,w,h", [(2, 2, 1203, 301), (2, 1, 900, 257), (3, 3, 1501, 203), (3, 1, 1501, 203),
                                        (5, 1, 2003, 305)])
def test_levels_and_kinds(oracle_lib, n, kind, w, h, levels):
    _check(_rig(n, kind, w, h, seed=n + levels), kind, levels, batch=2, pitch_extra=5)


@pytest.mark.parametrize("n,kind", [(2, 2), (4, 1)])
def test_whole_canvas_blend(oracle_lib, n, kind):
    _check(_rig(n, kind, 1301, 190, seed=3), kind, 4, minimize=False)


def test_entries_outside_the_frames(oracle_lib):
    _check(_rig(2, 2, 1200, 220, seed=9, oob_fraction=0.05), 2, 4)
    _check(_rig(4, 1, 1600, 220, seed=9, oob_fraction=0.05), 1, 4)


def test_seam_values_no_image_has(oracle_lib):
    for n, kind, value in ((2, 2, 3), (3, 3, 7), (4, 1, 200)):
        rig = _rig(n, kind, 1400, 200, seed=21)
        rig.seam[40:90, 200:420] = value
        rig.seam[120:140, 650:760] = value
        _check(rig, kind, 4)


def test_copy_blocks_switch_and_capture(oracle_lib):
    import torch
    from hmpano import _lib

    rig = _rig(3, 3, 2100, 400, seed=2)
    st, frames, ref = _check(rig, 3, 5)
    handle = st._handle_for(3, False)
    ins = [torch.from_numpy(f).cuda() for f in frames]
    for mode in (0, 1, 2):
        assert _lib.lib().hmp_stitcher_set_copy_blocks(handle, mode).code == 0
        out = st._run(ins)
        assert np.array_equal(out.cpu().numpy(), ref), mode
    canvas = torch.zeros_like(out)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        st._run(ins, canvas)
    g.replay()
    torch.cuda.synchronize()
    assert np.array_equal(canvas.cpu().numpy(), ref)


def test_frames_past_the_offset_range(oracle_lib):
    """Row pitches that put the frames' last pixels past 2^29 bytes."""
    import torch

    rig = _rig(2, 2, 1203, 301, seed=4)
    for levels in (0, 4):
        frames = _frames(rig, 5, 1)
        ref = oracle_lib.Stitch.from_rig(rig, levels, 1).run(frames)
        ins = []
        for f in frames:
            _, h, w, c = f.shape
            pitch = (1 << 29) // h + 4097
            buf = torch.zeros(h * pitch, dtype=torch.uint8, device="cuda")
            t = buf.as_strided((1, h, w, c), (h * pitch, pitch, c, 1))
            t.copy_(torch.from_numpy(f).cuda())
            ins.append(t)
        st = make_stitcher(2, masks_for_rig(rig), levels, 1)
        out = st._run(ins).cpu().numpy()
        assert np.array_equal(out, ref)
