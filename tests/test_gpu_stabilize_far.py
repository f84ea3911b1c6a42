"""Flow beyond the part of the next frame that the tiled kernel stages (kFlowPitch's margin around the
tile), bit for bit against the oracle: smooth content that Lucas-Kanade follows past half the margin and
past the margin, tiles with more features than a CTA has threads, unrelated frames whose flow scatters,
windows across the border, frames at each offset from a 16-byte boundary, odd widths."""
from __future__ import annotations

import numpy as np
import pytest

from stab_frames import texture

WINDOW_MARGIN = {3: 15, 9: 12, 15: 9, 21: 6}  # (96 - 64) / 2 - half


def pair(h, w, shift, seed, blur):
    dx, dy = shift
    m = max(abs(dx), abs(dy)) + 1
    big = texture(h + 2 * m, w + 2 * m, seed, blur)
    return (np.ascontiguousarray(big[m:m + h, m:m + w]),
            np.ascontiguousarray(big[m - dy:m - dy + h, m - dx:m - dx + w]))


def grid(h, w, step):
    return np.array([(x, y) for y in range(0, h, step) for x in range(0, w, step)], np.int32)


# h, w, motion (None: an unrelated frame), window, blur, feature spacing, offset of the frames in values
CASES = [
    (200, 260, (7, 3), 15, 9, 4, 0), (200, 260, (-11, 8), 15, 12, 4, 1), (131, 203, (12, -12), 15, 12, 5, 2),
    (200, 260, (8, -6), 21, 12, 4, 3), (131, 203, (20, 0), 9, 24, 5, 1), (131, 203, (24, 20), 3, 30, 5, 2),
    (131, 203, None, 15, 3, 5, 3), (131, 204, None, 21, 3, 5, 0), (70, 90, None, 9, 3, 3, 1), (40, 30, None, 15, 3, 2, 2),
]


def _frames(h, w, shift, blur):
    if shift is not None:
        return pair(h, w, shift, h + w, blur)
    return texture(h, w, 5, blur), texture(h, w, 6, blur)


@pytest.mark.parametrize("h,w,shift,window,blur,step,off", CASES)
def test_flows_leave_the_margin(oracle_lib, h, w, shift, window, blur, step, off):
    prev, nxt = _frames(h, w, shift, blur)
    xy = grid(h, w, step)
    flow = oracle_lib.Stabilize(window=window).run(prev, nxt, features=xy)["flow"]
    margin, far = WINDOW_MARGIN[window], np.abs(flow).max(1)
    assert np.isfinite(flow).all()
    assert (far > margin + 1).mean() > (0.25 if shift is None or max(map(abs, shift)) > margin else 0.0)
    if shift is not None:  # some tile's mean is past half the margin, where `next` is staged again
        tiles = (xy // 64) @ np.array([1, 100])
        assert max(np.abs(flow[tiles == t].mean(0)).max() for t in np.unique(tiles)) > margin / 2 + 1
        if step == 4:
            assert max((tiles == t).sum() for t in np.unique(tiles)) > 128


@pytest.mark.gpu
@pytest.mark.parametrize("h,w,shift,window,blur,step,off", CASES)
def test_far_flow_matches_oracle(oracle_lib, h, w, shift, window, blur, step, off):
    import build as hmp_build
    import hmpano
    import torch

    hmp_build.build()
    prev, nxt = _frames(h, w, shift, blur)
    xy = grid(h, w, step)
    ref = oracle_lib.Stabilize(window=window).run(prev, nxt, features=xy)
    dev = []
    for f in (prev, nxt):
        t = torch.zeros(h * w + off, device="cuda")[off:].view(h, w)
        t.copy_(torch.from_numpy(f))
        dev.append(t)
    st = hmpano.Stabilizer(w, h)
    st.set_features(xy)
    st.flow(*dev, window_size=window)
    _, flow, m = st.features()
    np.testing.assert_array_equal(flow, ref["flow"].reshape(-1, 2))
    np.testing.assert_array_equal(np.float32([m.dx, m.dy]), np.float32([ref["dx"], ref["dy"]]))
