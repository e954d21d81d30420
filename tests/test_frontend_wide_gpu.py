"""Blur windows too wide for the tiles (R > 320) along the rows, with the median division that follows
them, against the oracle's restatement of the reference driver's frame preparation."""
import types

import numpy as np
import pytest

from oracle import frontend
from steadyscan_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,w", [(40, 720), (720, 721)])
@pytest.mark.parametrize("src", [np.uint16, np.float64])
@pytest.mark.parametrize("mednorm", [True, False])
def test_wide_windows_along_the_rows(h, w, src, mednorm):
    import torch
    sd = 36.0  # windows of 346 samples each side, clamped to half the padded length
    frames = np.random.default_rng(w).uniform(0, 60000, size=(h, w, 2)).astype(src)
    lay = types.SimpleNamespace(prevknotind=np.tile((np.arange(h) + 1)[:, None], (1, w)), frame_w=h,
                                cropping=[0, 0, 0, 0])
    dev = torch.from_numpy(np.ascontiguousarray(frames.transpose(2, 1, 0))).cuda().permute(2, 1, 0)
    got = api.prepare_frames(dev, lay, pregauss=sd, mednorm=mednorm).cpu().numpy()
    ref = frontend.set_bmdata(frames, lay.prevknotind, h, [0, 0, 0, 0], sd, mednorm)
    # the FFT and the direct sums round differently, each by a few 1e-16 of the largest sample
    np.testing.assert_allclose(got, ref, rtol=1e-12, atol=1e-12 * np.abs(ref).max())
