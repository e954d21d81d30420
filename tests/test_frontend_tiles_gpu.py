"""The tiled kernels of ss_prepare_frames at the edges of their tiles, against the oracle's restatement
of the reference driver's frame preparation."""
import types

import numpy as np
import pytest

from oracle import frontend
from steadyscan_b200 import api

pytestmark = pytest.mark.gpu


def _rows_layout(hc, wc, nb, crop):
    """Blocks of whole lines, as even as the line count allows."""
    blk = np.arange(hc) * nb // hc + 1
    return types.SimpleNamespace(prevknotind=np.tile(blk[:, None], (1, wc)), frame_w=nb, cropping=crop)


def _frames(h, w, n, dtype, seed=0):
    x = np.random.default_rng(seed).uniform(0, 60000, size=(h, w, n))
    return x.astype(dtype)


def _device(frames):
    import torch
    return torch.from_numpy(np.ascontiguousarray(frames.transpose(2, 1, 0))).cuda().permute(2, 1, 0)


# lines, pixels, blocks, cropping: tiles of 64 rows and columns full, one short and one over; 1 to 33
# lines per block (33: the general gather); blocks of unequal height; rows and columns off 16 bytes
MAPS = [(64, 64, 64, [0, 0, 0, 0]), (128, 65, 64, [0, 0, 0, 0]), (130, 63, 65, [1, 1, 1, 1]), (63, 129, 21, [0, 0, 0, 0]),
        (96, 70, 3, [0, 0, 0, 0]), (99, 40, 3, [0, 0, 0, 0]), (77, 130, 10, [2, 3, 8, 5]), (72, 96, 9, [4, 0, 8, 0]),
        (5, 3, 5, [0, 0, 0, 0]), (40, 1, 20, [0, 0, 0, 0])]


@pytest.mark.parametrize("h,w,nb,crop", MAPS)
@pytest.mark.parametrize("src,out", [(np.uint16, np.uint16), (np.uint16, np.float64), (np.float32, np.float32),
                                     (np.float64, np.float32), (np.float64, np.float64)])
def test_whole_line_blocks_are_copied_exactly(h, w, nb, crop, src, out):
    frames = _frames(h, w, 3, src)
    lay = _rows_layout(h - crop[2] - crop[3], w - crop[0] - crop[1], nb, crop)
    got = api.prepare_frames(_device(frames), lay, out_dtype=out).cpu().numpy()
    ref = frontend.set_bmdata(frames, lay.prevknotind, nb, crop, 0.0, False)
    np.testing.assert_array_equal(got, ref.astype(out))


def test_a_map_that_only_starts_like_whole_lines_is_gathered():
    """One entry off the row structure: the general gather, not the tiles."""
    h, w, nb = 64, 70, 16
    frames = _frames(h, w, 2, np.float32)
    lay = _rows_layout(h, w, nb, [0, 0, 0, 0])
    blk = lay.prevknotind.copy()
    blk[3, w - 1], blk[4, 0] = blk[4, 0], blk[3, w - 1]
    lay.prevknotind = blk
    got = api.prepare_frames(_device(frames), lay, out_dtype=np.float32).cpu().numpy()
    np.testing.assert_array_equal(got, frontend.set_bmdata(frames, blk, nb, [0, 0, 0, 0], 0.0, False).astype(np.float32))
