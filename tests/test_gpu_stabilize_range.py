"""Lucas-Kanade windows whose sums lie at the ends of the FP32 range, bit for bit against the oracle.
Every second line of the frames is a faint texture (the one that moves), the lines between are 0 and a
large value in turn, so that one gradient of a texture pixel is large and the other small. `upper`: sums
that double gradients overflow while the sums proper do not; `lower`: products that are subnormal, and
round differently doubled. The features are a grid over the frame, its borders included."""
from __future__ import annotations

import numpy as np
import pytest

from stab_frames import moving_pair


def frames(end: str, h: int, w: int, motion: int, window: int, seed: int):
    # upper: the squares of a whole window sum to 2e38 (doubled, 8e38); lower: to 2e36.
    scale, total = {"upper": (1 / 400, 2e38), "lower": (5e-23, 2e36)}[end]
    step = 2 * (total / (window * (window + 1) / 2)) ** 0.5
    a, b = moving_pair(w, h, (motion, 0), seed=seed) if end == "upper" else moving_pair(h, w, (motion, 0), seed=seed)
    out = []
    for f in (a, b):
        f = (f * np.float32(scale)).astype(np.float32)
        f[1::4] = 0
        f[3::4] = step
        out.append(f)
    if end == "upper":  # the lines are columns
        out = [np.ascontiguousarray(f.T) for f in out]
    return out


def grid(h: int, w: int):
    xs, ys = sorted({*range(0, w, 3), 1, w - 2, w - 1}), sorted({*range(0, h, 3), 1, h - 2, h - 1})
    return np.array([(x, y) for y in ys for x in xs], np.int32)


def first_sums(prev, nxt, xy, half, double):
    """The five sums of each window without displacement, in FP32 and the reference's order; `double`: of
    gradients without their factor 1/2, scaled afterwards."""
    h, w = prev.shape
    k, one = np.float32(1 if double else 0.5), np.float32(0.25)
    out = np.zeros((len(xy), 5), np.float32)
    for n, (px, py) in enumerate(xy):
        s = np.zeros(5, np.float32)
        for y in range(py - half, py + half + 1):
            for x in range(px - half, px + half + 1):
                if not (1 <= x < w - 1 and 1 <= y < h - 1):
                    continue
                ix, iy = (prev[y, x + 1] - prev[y, x - 1]) * k, (prev[y + 1, x] - prev[y - 1, x]) * k
                it = nxt[y, x] - prev[y, x]
                s = s + np.array([ix * ix, iy * iy, ix * iy, ix * it, iy * it], np.float32)
        out[n] = s * np.array([one, one, one, 2 * one, 2 * one], np.float32) if double else s
    return out


CASES = [("upper", 1, 15), ("upper", 3, 15), ("upper", 2, 9), ("lower", 1, 15), ("lower", 3, 15), ("lower", 2, 9)]


@pytest.mark.parametrize("end,motion,window", CASES)
def test_frames_reach_the_ends(oracle_lib, end, motion, window):
    """The inputs do what they are for: finite flows other than zero, past the first rounding too, from
    windows whose sums of doubled gradients are other bits than the sums proper."""
    h, w = 70, 84
    with np.errstate(all="ignore"):
        prev, nxt = frames(end, h, w, motion, window, seed=window + motion)
        xy = grid(h, w)
        flow = oracle_lib.Stabilize(window=window).run(prev, nxt, features=xy)["flow"]
        some = xy[:: len(xy) // 40]
        plain = first_sums(prev, nxt, some, window // 2, False)
        double = first_sums(prev, nxt, some, window // 2, True)
    assert np.isfinite(flow).all(1).mean() > 0.9
    assert (np.abs(flow).max(1) > 0.6).mean() > 0.2
    assert np.isfinite(plain).all()
    assert ((plain != double).any(1)).mean() > 0.5
    if end == "upper":
        assert (plain[:, 0] >= 1e37).mean() > 0.5
    else:
        assert ((plain[:, 0] > 0) & (plain[:, 0] < 1e-37)).mean() > 0.5


@pytest.mark.gpu
@pytest.mark.parametrize("end,motion,window", CASES)
def test_flow_at_the_ends(oracle_lib, end, motion, window):
    import build as hmp_build
    import hmpano
    import torch

    hmp_build.build()
    h, w = 140, 168
    xy = grid(h, w)
    with np.errstate(all="ignore"):
        prev, nxt = frames(end, h, w, motion, window, seed=window + motion)
        ref = oracle_lib.Stabilize(window=window).run(prev, nxt, features=xy)
    st = hmpano.Stabilizer(w, h)
    st.set_features(xy)
    st.flow(torch.from_numpy(prev).cuda(), torch.from_numpy(nxt).cuda(), window_size=window)
    _, flow, _ = st.features()
    np.testing.assert_array_equal(flow, ref["flow"].reshape(-1, 2))
