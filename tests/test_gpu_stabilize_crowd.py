"""Features crowded into one flow tile, shared out in items of 128: counts around the items' edges, more
items than CTAs are resident, crowded tiles beside sparse ones and one place many times, bit for bit
against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

from stab_frames import moving_pair

pytestmark = pytest.mark.gpu

H, W = 150, 200


def _crowd(n, seed=1):
    return np.random.default_rng(seed).integers((64, 64), (128, 128), (n, 2)).astype(np.int32)


def _features():
    for n in (1, 127, 128, 129, 255, 256, 257, 385, 1000):
        yield f"{n} in a tile", _crowd(n)
    yield "one place", np.full((700, 2), 70, np.int32)
    rng = np.random.default_rng(2)
    yield "a crowd and the rest", np.concatenate([_crowd(900), rng.integers((0, 0), (W, H), (300, 2)).astype(np.int32), _crowd(5, 3)])
    yield "more items than CTAs", np.concatenate([_crowd(27000), np.tile(np.int32([[3, 140]]), (27000, 1)), _crowd(9000, 4)])


@pytest.mark.parametrize("window,shift", [(5, (1, -1)), (15, (2, 1)), (21, (7, -6))])
def test_crowded_tiles_match_oracle(oracle_lib, window, shift):
    import build as hmp_build
    import hmpano
    import torch

    hmp_build.build()
    prev, nxt = moving_pair(H, W, shift, seed=window)
    p, q = torch.from_numpy(prev).cuda(), torch.from_numpy(nxt).cuda()
    st = hmpano.Stabilizer(W, H)
    more = hmpano.Stabilizer(600, 200)  # holds more features than this frame has pixels
    p2, q2 = (torch.nn.functional.pad(t, (0, 600 - W, 0, 200 - H)).contiguous() for t in (p, q))
    for what, xy in _features():
        big = len(xy) > (H - 2) * (W - 2)
        s, a, b = (more, p2, q2) if big else (st, p, q)
        uniq, back = np.unique(xy, axis=0, return_inverse=True)
        ref = oracle_lib.Stabilize(window=window).run(a.cpu().numpy(), b.cpu().numpy(), features=uniq)["flow"]
        s.set_features(xy)
        s.flow(a, b, window_size=window)
        got, flow, _ = s.features()
        np.testing.assert_array_equal(got, xy)
        np.testing.assert_array_equal(flow, ref.reshape(-1, 2)[back.ravel()], err_msg=what)
