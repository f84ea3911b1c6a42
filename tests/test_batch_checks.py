"""Batch.add refuses what process() refuses of a call's batch size and pixel types (the library's images
carry neither, so a captured job would read and write past the tensors)."""
from __future__ import annotations

from types import SimpleNamespace

import pytest


@pytest.mark.parametrize("ins,canvas", [
    ([(1, 6, 8, 4), (2, 6, 8, 4)], (2, 7, 9, 4)), ([(2, 6, 8, 4)] * 2, (1, 7, 9, 4)), ([(1, 6, 8, 4)] * 2, (1, 7, 9, 4)),
    ([(6, 8, 4)] * 2, (7, 9, 4)), ([(2, 6, 8, 3), (2, 6, 8, 4)], (2, 7, 9, 4)), ([(2, 6, 8, 4)] * 2, (2, 7, 9, 3)),
])
def test_refused_on_the_host(ins, canvas):
    import torch
    from hmpano import pano

    job = object.__new__(pano.Batch)
    job._h, job._keep = None, []
    st = SimpleNamespace(_batch=2, _handle_for=lambda *a: pytest.fail("reached the library"))
    with pytest.raises(ValueError, match="batch size|pixel type"):
        job.add(st, [torch.zeros(s, dtype=torch.uint8) for s in ins], torch.zeros(canvas, dtype=torch.uint8))
