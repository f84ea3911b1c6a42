"""StitchServer.submit: requests whose images hold another number of frames than the configuration, or
another pixel type, are refused before they reach the library (whose images carry neither), whether or
not their marshalling takes the packed form."""
from __future__ import annotations

import numpy as np
import pytest


def _bare_server(batch):
    """A server object without its native half, which a refused request never reaches."""
    from hmpano import pano

    srv = object.__new__(pano.StitchServer)
    srv._h, srv._live, srv._batch, srv._device = None, {}, {0: batch}, 0
    return srv


def _shapes(batch):
    """(what, input shapes and types, canvas shape and type) of requests that are refused."""
    b, u8, f32 = batch, "uint8", "float32"
    ok, canvas = ((b, 6, 8, 4), u8), ((b, 7, 9, 4), u8)
    yield "frames", [((b + 1, 6, 8, 4), u8), ok], canvas
    yield "frames of one input", [ok, ((b - 1 or 3, 6, 8, 4), u8)], canvas
    yield "canvas frames", [ok, ok], ((b + 1, 7, 9, 4), u8)
    yield "all one frame more", [((b + 1, 6, 8, 4), u8)] * 2, ((b + 1, 7, 9, 4), u8)
    if b > 1:
        yield "all one frame", [((1, 6, 8, 4), u8)] * 2, ((1, 7, 9, 4), u8)
        yield "no frame axis", [((6, 8, 4), u8)] * 2, ((7, 9, 4), u8)
    yield "float", [((b, 6, 8, 4), f32)] * 2, canvas
    yield "float canvas", [ok, ok], ((b, 7, 9, 4), f32)
    yield "rgb", [((b, 6, 8, 3), u8)] * 2, ((b, 7, 9, 3), u8)


@pytest.mark.parametrize("batch", [1, 2])
def test_refused_on_the_host(batch):
    import torch

    for what, ins, canvas in _shapes(batch):
        with pytest.raises(ValueError, match="batch size|pixel type|RGBA"):
            _bare_server(batch).submit(0, [torch.zeros(s, dtype=getattr(torch, t)) for s, t in ins],
                                       torch.zeros(canvas[0], dtype=getattr(torch, canvas[1])))
            pytest.fail(what)


@pytest.mark.gpu
@pytest.mark.parametrize("batch", [1, 2])
def test_packed_and_unpacked_requests_agree(batch, monkeypatch):
    import build as hmp_build
    import hmpano
    import torch
    from helpers import make_stitcher, masks_for_rig
    from hmpano import pano, synth

    hmp_build.build()
    rig = synth.workload_rig("pano2_1280x720_to_2200x800", seed=3, kind=2, scale=0.4)
    frames = [torch.from_numpy(f).cuda() for f in synth.rig_frames(rig, seed=1, batch=batch)]
    want = make_stitcher(2, masks_for_rig(rig), 3, batch)._run(frames).cpu().numpy()
    wide = torch.zeros((*frames[0].shape[:2], frames[0].shape[2] + 5, 4), dtype=torch.uint8, device="cuda")[:, :, :-5]
    wide.copy_(frames[0])
    forms = [("plain", frames), ("pitched", [wide, frames[1]])] + ([("3-d", [f[0] for f in frames])] if batch == 1 else [])
    pack, device = pano._pack_images, lambda t: torch.zeros(t[0], dtype=getattr(torch, t[1]), device="cuda")
    srv = hmpano.StitchServer(1 << 30, slots=2)
    for use in (pack, lambda *a: None):
        monkeypatch.setattr(pano, "_pack_images", use)
        cid = srv.add_config(2, masks_for_rig(rig), 3, batch_size=batch)
        for what, ins, canvas in _shapes(batch):
            with pytest.raises(ValueError, match="batch size|pixel type|RGBA"):
                srv.submit(cid, [device(t) for t in ins], device(canvas))
                pytest.fail(what)
        with pytest.raises(pano.CudaStatusError):
            srv.submit(cid + 7, frames, frames[0])
        with pytest.raises(pano.CudaStatusError):
            srv.submit(cid, frames[:1], frames[0])
        for what, ins in forms:
            out = torch.zeros(want.shape, dtype=torch.uint8, device="cuda")
            torch.cuda.synchronize()
            assert srv.wait(srv.submit(cid, ins, out)).ok()
            assert np.array_equal(out.cpu().numpy(), want), what
    srv.close()
