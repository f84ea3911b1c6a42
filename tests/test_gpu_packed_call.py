"""process() calls that marshal their images in one pack against the checked path, form by form: the
same canvas, or the same exception with the same message."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import make_stitcher, masks_for_rig

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def setup():
    import build as hmp_build
    from hmpano import synth

    hmp_build.build()
    rig = synth.workload_rig("pano2_1280x720_to_2200x800", seed=3, kind=2, scale=0.4)
    return rig, {b: (make_stitcher(2, masks_for_rig(rig), 3, b), synth.rig_frames(rig, seed=1, batch=b)) for b in (1, 2)}


def _forms(torch, frames, canvas):
    ins = [torch.from_numpy(f).cuda() for f in frames]
    b, h, w, c = ins[0].shape
    wide = torch.zeros((b, h, w + 5, c), dtype=torch.uint8, device="cuda")[:, :, :w]
    wide.copy_(ins[0])
    yield "plain", ins, canvas
    yield "pitched", [wide, ins[1]], canvas
    if b == 1:
        yield "3-d", [t[0] for t in ins], canvas[0]
        yield "zero batch stride", [t[0].expand(1, -1, -1, -1) for t in ins], canvas
    yield "rgb", [t[..., :3].contiguous() for t in ins], canvas[..., :3].contiguous()
    yield "float", [t.float() for t in ins], canvas.float()
    yield "mixed types", [ins[0].float(), ins[1]], canvas
    yield "canvas type", ins, canvas.float()
    yield "half", [t.half() for t in ins], canvas.half()
    yield "two channels", [t[..., :2] for t in ins], canvas[..., :2]
    yield "transposed", [ins[0].transpose(1, 2), ins[1]], canvas
    yield "flipped channels", [ins[0][..., [2, 1, 0, 3]].permute(0, 1, 3, 2).contiguous().permute(0, 1, 3, 2), ins[1]], canvas
    yield "batch", [torch.cat([ins[0], ins[0]]), ins[1]], canvas
    yield "canvas batch", ins, torch.cat([canvas, canvas])
    yield "cpu input", [ins[0].cpu(), ins[1]], canvas
    yield "cpu canvas", ins, canvas.cpu()
    yield "2-d", [ins[0][0, ..., 0], ins[1]], canvas
    yield "one input", ins[:1], canvas
    yield "three inputs", [*ins, ins[0]], canvas
    yield "none", [None, ins[1]], canvas
    yield "canvas size", ins, canvas[:, :-1]


@pytest.mark.parametrize("batch", [1, 2])
def test_packed_call_equals_the_checked_one(setup, batch):
    import torch

    rig, by_batch = setup
    st, frames = by_batch[batch]
    shape = (batch, st.canvas_height(), st.canvas_width(), 4)
    results = {}
    for which in ("_run", "_run_checked"):
        for name, ins, canvas in _forms(torch, frames, torch.zeros(shape, dtype=torch.uint8, device="cuda")):
            fresh = make_stitcher(2, masks_for_rig(rig), 3, batch)  # a per-call error is sticky
            if name == "rgb":
                fresh._run_checked(ins)  # its stitcher exists
            try:
                out = getattr(fresh, which)(ins, canvas)
                got = (tuple(out.shape), out.cpu().numpy())
                assert out.data_ptr() == canvas.data_ptr()
            except Exception as e:
                got = (type(e).__name__, str(e))
            results.setdefault(name, []).append(got)
    assert isinstance(results["plain"][0][1], np.ndarray)
    for name, (a, b) in results.items():
        assert type(a[1]) is type(b[1]), (name, a, b)
        if isinstance(a[1], np.ndarray):
            assert a[0] == b[0] and np.array_equal(a[1], b[1]), name
        else:
            assert a == b, name


def test_sticky_status_on_both_paths(setup):
    import torch
    from hmpano import pano

    rig, by_batch = setup
    _, frames = by_batch[1]
    ins = [torch.from_numpy(f).cuda() for f in frames]
    st = make_stitcher(2, masks_for_rig(rig), 3, 1)
    good = torch.zeros((1, st.canvas_height(), st.canvas_width(), 4), dtype=torch.uint8, device="cuda")
    with pytest.raises(pano.CudaStatusError) as first:
        st._run(ins, good[:, :-1])
    for run in (st._run, st._run_checked):
        with pytest.raises(pano.CudaStatusError) as again:
            run(ins, good)
        assert str(again.value) == str(first.value)
        with pytest.raises(pano.CudaStatusError):  # the status comes before the frames' own faults
            run([t[..., :3].contiguous() for t in ins], good[..., :3].contiguous())
