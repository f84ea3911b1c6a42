"""Captured and eager calls of one stitcher with frames of different geometries (row pitches, sizes):
every canvas equals the oracle's whatever ran in between, and a call captured before any eager one
(which reads the planned table entries instead of the resolved plane) equals the eager call over the
forms the canvas gather has."""
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

    return synth.make_rig(canvas_w=w, canvas_h=h, n=n, src_w=w // n + 120, src_h=int(h * 0.9), overlap=0.22, seed=seed,
                          kind=kind, **kw)


class _Calls:
    """A stitcher, its frames in two layouts (`wide` has the longer rows) and their canvases."""

    def __init__(self, oracle_lib, rig, levels, channels, batch=1, minimize=True, holes=False, **kw):
        import torch
        from hmpano import synth

        self.st = make_stitcher(rig.kind, masks_for_rig(rig), levels, batch, minimize=minimize, **kw)
        assert self.st.status.ok(), self.st.status
        self.st._handle_for(channels, False)  # the pixel type's stitcher exists before any capture
        self.ins, self.ref = {}, {}
        orc = oracle_lib.Stitch.from_rig(rig, levels, batch, minimize_blend=minimize)
        for seed, (name, extra) in enumerate((("tight", 0), ("wide", 9))):
            frames = [np.ascontiguousarray(f[..., :channels]) for f in synth.rig_frames(rig, seed=seed, batch=batch)]
            if holes:
                for f in frames:
                    f[:, 30:60, 40:-40, 3] = 0
            self.ref[name] = orc.run(frames) if not kw else None
            self.ins[name] = []
            for f in frames:
                b, h, w, c = f.shape
                t = torch.zeros((b, h, w + extra, c), dtype=torch.uint8, device="cuda")[:, :, :w]
                t.copy_(torch.from_numpy(f))
                self.ins[name].append(t)
        self.shape = (batch, rig.canvas_h, rig.canvas_w, channels)
        torch.cuda.synchronize()

    def canvas(self):
        import torch

        return torch.full(self.shape, 77, dtype=torch.uint8, device="cuda")

    def eager(self, name):
        import torch

        out = self.canvas()
        self.st._run(self.ins[name], out)
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy(), self.ref[name]), ("eager", name)

    def capture(self, name):
        import torch

        out, g = self.canvas(), torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            self.st._run(self.ins[name], out)

        def replay():
            out.fill_(78)
            g.replay()
            torch.cuda.synchronize()
            assert np.array_equal(out.cpu().numpy(), self.ref[name]), ("replay", name)

        return replay


FORMS = [(2, 2, 0, 3), (2, 2, 4, 3), (3, 3, 3, 3), (5, 1, 3, 3), (2, 2, 0, 4), (2, 2, 4, 4), (3, 3, 3, 4), (5, 1, 3, 4)]


@pytest.mark.parametrize("n,kind,levels,channels", FORMS)
def test_capture_then_other_geometry(oracle_lib, n, kind, levels, channels):
    c = _Calls(oracle_lib, _rig(n, kind, 420 * n + 3, 203, seed=n), levels, channels)
    c.eager("wide")
    wide = c.capture("wide")
    c.eager("tight")
    wide()
    c.eager("wide")
    tight = c.capture("tight")
    for step in (tight, wide, lambda: c.eager("tight"), wide, tight):
        step()


@pytest.mark.parametrize("n,kind,levels,channels", FORMS)
def test_first_call_captured(oracle_lib, n, kind, levels, channels):
    c = _Calls(oracle_lib, _rig(n, kind, 420 * n + 3, 203, seed=n), levels, channels)
    wide = c.capture("wide")
    c.eager("wide")
    wide()
    c.eager("tight")
    wide()
    tight = c.capture("tight")
    for step in (wide, tight, lambda: c.eager("wide"), tight):
        step()


@pytest.mark.parametrize("channels", [3, 4])
@pytest.mark.parametrize("kind,n,levels,minimize,rig_kw", [
    (2, 2, 3, False, {}), (1, 4, 3, False, {}), (1, 2, 1, True, {}), (2, 2, 0, True, {"oob_fraction": 0.05}),
    (2, 2, 3, True, {"oob_fraction": 0.05}), (3, 3, 2, True, {"oob_fraction": 0.05}), (1, 8, 4, True, {}), (1, 4, 0, True, {})])
def test_planned_entries_give_the_oracles_canvas(oracle_lib, kind, n, levels, minimize, rig_kw, channels):
    c = _Calls(oracle_lib, _rig(n, kind, 300 * n + 301, 157, seed=7, **rig_kw), levels, channels, batch=2, minimize=minimize)
    c.capture("tight")()


@pytest.mark.parametrize("n,kind", [(2, 2), (3, 3), (5, 1)])
def test_planned_entries_check_alpha(oracle_lib, n, kind):
    """Copy blocks with alpha 0 behind them: captured first (three gated launches), and eager beside a
    captured call of another geometry (the gate)."""
    c = _Calls(oracle_lib, _rig(n, kind, 420 * n + 3, 203, seed=n), 4, 4, holes=True)
    c.capture("wide")()
    c = _Calls(oracle_lib, _rig(n, kind, 420 * n + 3, 203, seed=n), 4, 4, holes=True)
    c.eager("wide")
    wide = c.capture("wide")
    c.eager("tight")
    c.eager("tight")
    wide()


@pytest.mark.parametrize("storage,filter", [("f16", "refbox"), ("f32", "binomial5")])
def test_planned_entries_other_pyramids(oracle_lib, storage, filter):
    import torch

    rig = _rig(2, 2, 903, 203, seed=5)
    c = _Calls(oracle_lib, rig, 4, 4, storage=storage, filter=filter)
    other = make_stitcher(2, masks_for_rig(rig), 4, 1, storage=storage, filter=filter)
    for name in ("tight", "wide"):
        c.ref[name] = other._run(c.ins[name]).cpu().numpy()
    torch.cuda.synchronize()
    c.capture("wide")()
    c.eager("tight")
    c.capture("tight")()
