"""The stabiliser's tiled flow and bitmask corners where they change path, bit for bit against the
oracle: windows at the ends of the tiled range and past it, frames one pixel around the 64-pixel
tiles and the 128-pixel corner blocks, more corners in a tile than a CTA has threads, motions inside,
past and far past the staged margin, frames at odd addresses, and values whose window sums leave
FP32's comfortable range."""
from __future__ import annotations

import numpy as np
import pytest

from stab_frames import moving_pair

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    import build as hmp_build

    hmp_build.build()


CASES = [
    # h, w, shift, window, threshold, scale
    (64, 64, (1, 0), 15, 1e6, 1.0),
    (65, 129, (-2, 3), 15, 1e6, 1.0),
    (127, 257, (2, 2), 3, 1e6, 1.0),
    (90, 130, (0, -3), 20, 1e6, 1.0),
    (90, 130, (1, 1), 22, 1e6, 1.0),
    (70, 90, (1, 1), 1, 1e6, 1.0),
    (130, 200, (9, -7), 15, 1e6, 1.0),
    (130, 200, (26, 31), 15, 1e6, 1.0),
    (130, 200, (-14, 11), 21, 1e6, 1.0),
    (96, 128, (1, -1), 15, -1e38, 1.0),
    (80, 100, (2, 1), 15, 1e6, 3e17),
    (80, 100, (2, 1), 15, -1e38, 1e-21),
]


@pytest.mark.parametrize("h,w,shift,window,thr,scale", CASES)
def test_tiles_match_oracle(oracle_lib, h, w, shift, window, thr, scale):
    import hmpano
    import torch

    prev, nxt = moving_pair(h, w, shift, seed=h + w)
    prev, nxt = (prev * np.float32(scale)).astype(np.float32), (nxt * np.float32(scale)).astype(np.float32)
    with np.errstate(all="ignore"):
        ref = oracle_lib.Stabilize(threshold=thr, window=window).run(prev, nxt)
    st = hmpano.Stabilizer(w, h)
    # Frames four bytes past a 16-byte boundary.
    bufs = [torch.zeros(h * w + 1, device="cuda")[1:].view(h, w) for _ in range(3)]
    bufs[0].copy_(torch.from_numpy(prev))
    bufs[1].copy_(torch.from_numpy(nxt))
    st.run(bufs[0], bufs[1], bufs[2], threshold=thr, window_size=window)
    xy, flow, m = st.features()
    assert m.corners == ref["found"]
    np.testing.assert_array_equal(st.response(), ref["response"])
    np.testing.assert_array_equal(xy, ref["corners"].reshape(-1, 2))
    np.testing.assert_array_equal(flow, ref["flow"].reshape(-1, 2))
    np.testing.assert_array_equal(np.float32([m.dx, m.dy]), np.float32([ref["dx"], ref["dy"]]))
    np.testing.assert_array_equal(bufs[2].cpu().numpy(), ref["out"])
