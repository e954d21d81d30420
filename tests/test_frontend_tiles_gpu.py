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


# a warp's 256 outputs down a column and a CTA's 64 columns full, one short and one over; windows that
# wrap more than once round a small frame; a window too wide for the tiles (R > 320)
BLURS = [(256, 64, 1.0), (257, 65, 2.0), (255, 63, 0.3), (7, 5, 1.5), (33, 129, 6.0), (720, 40, 36.0), (513, 9, 4.7)]


@pytest.mark.parametrize("h,w,sd", BLURS)
@pytest.mark.parametrize("src", [np.uint16, np.float32])
def test_blur_tiles_match_the_fft(h, w, sd, src):
    """The FFT and the direct sums round differently, each by a few 1e-16 of the largest sample."""
    frames = _frames(h, w, 2, src, seed=h)
    lay = _rows_layout(h, w, h, [0, 0, 0, 0])
    got = api.prepare_frames(_device(frames), lay, pregauss=sd).cpu().numpy()
    ref = frontend.set_bmdata(frames, lay.prevknotind, h, lay.cropping, sd, False)
    np.testing.assert_allclose(got, ref, rtol=1e-12, atol=1e-12 * np.abs(ref).max())


def _median_frames(kind, h, w):
    rng = np.random.default_rng(h * 7 + w)
    x = rng.uniform(10, 200, size=(h, w, 2))
    if kind == "ties":  # a few values, many samples each: no range of keys narrows to a few samples
        x = np.floor(x / 50) * 50 + 1
    elif kind == "halves":  # the two middle samples on either side of a gap
        x = np.where((np.arange(h * w) % 2 == 0).reshape(h, w)[:, :, None], 3.0, 1e9) * np.ones(2)
    elif kind == "constant":
        x = np.full_like(x, 4.25)
    elif kind == "wide":  # both signs, every binade, zeros of both signs and infinities
        x = np.ldexp(rng.standard_normal(x.shape), rng.integers(-900, 900, x.shape))
        x.reshape(-1)[::7] = 0.0
        x.reshape(-1)[3::11] = -0.0
        x[0, 0], x[-1, -1] = np.inf, -np.inf
        x += 1.5  # the median of symmetric samples would be next to zero
    elif kind == "nan":
        x[h // 2, w // 2, 1] = np.nan
    return x


# counts at and around the 1024 samples that are ranked at once, odd and even, one sample
@pytest.mark.parametrize("h,w", [(1, 1), (1, 2), (32, 32), (41, 25), (31, 33), (300, 217), (128, 512)])
@pytest.mark.parametrize("kind", ["plain", "ties", "halves", "constant", "wide", "nan"])
def test_median_is_exact(kind, h, w):
    frames = _median_frames(kind, h, w)
    lay = _rows_layout(h, w, h, [0, 0, 0, 0])
    got = api.prepare_frames(_device(frames), lay, mednorm=True).cpu().numpy()
    with np.errstate(all="ignore"):
        med = np.median(frames.reshape(h * w, 2, order="F"), axis=0)
        ref = frames / med
    np.testing.assert_array_equal(got, frontend.set_bmdata(ref, lay.prevknotind, h, lay.cropping, 0.0, False))


@pytest.mark.parametrize("src", [np.uint16, np.float32, np.float16])
def test_median_of_storage_types(src):
    frames = (np.random.default_rng(5).integers(1, 900, size=(90, 61, 3))).astype(src)
    lay = _rows_layout(90, 61, 30, [0, 0, 0, 0])
    got = api.prepare_frames(_device(frames), lay, mednorm=True, out_dtype=np.float32).cpu().numpy()
    f = frames.astype(np.float64)
    ref = frontend.set_bmdata(f / np.median(f.reshape(-1, 3, order="F"), axis=0), lay.prevknotind, 30, lay.cropping,
                              0.0, False)
    np.testing.assert_array_equal(got, ref.astype(np.float32))
