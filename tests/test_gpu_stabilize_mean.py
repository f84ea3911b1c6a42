"""The stabiliser's mean flow on sums that hover: a still pair with sensor noise, whose flow scatters
around zero, so that the running sums keep changing sign and binade over several of the mean's chunks.
The bits are those of the oracle's one sum after the other, at counts around the kernel's limits."""
from __future__ import annotations

import functools

import numpy as np
import pytest

from stab_frames import texture

H, W, WINDOW = 400, 480, 9
COUNTS = [1, 31, 4095, 4096, 4097, 11263, 11264, 11265, 30000, 48000]


@functools.lru_cache(None)
def still():
    rng = np.random.default_rng(3)
    base = texture(H, W, 7)
    prev, nxt = (np.round(base + rng.normal(0, 3, base.shape)).astype(np.float32) for _ in range(2))
    xy = np.array([(x, y) for y in range(0, H, 2) for x in range(0, W, 2)], np.int32)
    return prev, nxt, xy


def test_sums_hover(oracle_lib):
    prev, nxt, xy = still()
    flow = oracle_lib.Stabilize(window=WINDOW).run(prev, nxt, features=xy)["flow"]
    for part in (flow[:11264, 0], flow[:, 0], flow[:, 1]):
        sums = np.cumsum(part, dtype=np.float32)
        binades = np.sign(sums) * np.floor(np.log2(np.maximum(np.abs(sums), 1e-30)))
        assert (np.diff(binades) != 0).sum() > 60


@pytest.mark.gpu
def test_mean_of_hovering_sums(oracle_lib):
    import build as hmp_build
    import hmpano
    import torch

    hmp_build.build()
    prev, nxt, xy = still()
    st = hmpano.Stabilizer(W, H)
    p, q = torch.from_numpy(prev).cuda(), torch.from_numpy(nxt).cuda()
    for n in COUNTS:
        ref = oracle_lib.Stabilize(window=WINDOW).run(prev, nxt, features=xy[:n])
        st.set_features(xy[:n])
        st.flow(p, q, window_size=WINDOW)
        _, flow, m = st.features()
        np.testing.assert_array_equal(flow, ref["flow"].reshape(-1, 2))
        np.testing.assert_array_equal(np.float32([m.dx, m.dy]), np.float32([ref["dx"], ref["dy"]]))
