"""The first replay of a captured call whose copy blocks do not hold (alpha 0 behind them), on a new
stitcher: its pyramid buffers outside the work lists hold nothing of these frames yet, so a fallback
kernel that reads ahead of the one before it shows as wrong pixels."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import make_stitcher, masks_for_rig

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,kind,levels", [(2, 2, 4), (3, 3, 3), (3, 3, 4), (3, 1, 5), (5, 1, 4)])
def test_first_replay_that_falls_back(oracle_lib, n, kind, levels):
    import build as hmp_build
    import torch
    from hmpano import synth

    hmp_build.build()
    rig = synth.make_rig(canvas_w=420 * n + 3, canvas_h=203, n=n, src_w=540, src_h=182, overlap=0.22, seed=n, kind=kind)
    orc = oracle_lib.Stitch.from_rig(rig, levels)
    cases = []
    for seed in (1, 2):
        frames = synth.rig_frames(rig, seed=seed)
        for f in frames:
            f[:, 30:60, 40:-40, 3] = 0
        cases.append(([torch.from_numpy(f).cuda() for f in frames], orc.run(frames)))
    other = [torch.from_numpy(f).cuda() for f in synth.rig_frames(rig, seed=9)]
    for i in range(12):
        st = make_stitcher(kind, masks_for_rig(rig), levels)
        ins, ref = cases[i % 2]
        mine, canvas = [t.clone() for t in other], torch.zeros(ref.shape, dtype=torch.uint8, device="cuda")
        st._run(mine, canvas)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            st._run(mine, canvas)
        for t, u in zip(mine, ins):
            t.copy_(u)
        g.replay()
        torch.cuda.synchronize()
        out = canvas.cpu().numpy()
        assert np.array_equal(out, ref), (i, np.argwhere((out != ref).any(-1))[[0, -1]].tolist())
