"""The block map of ss_prepare_frames is checked before any device work (no GPU needed: the device id is
out of range, which is only reported for a valid map)."""
import ctypes as C

import numpy as np
import pytest

from steadyscan_b200 import _lib
from steadyscan_b200._lib import SS_DEVICE, SS_U16, SSMatrix, SSPrepFrames


def _call(h, w, gather):
    g = np.asarray(gather, np.int32)
    hb, nb = g.shape
    g = np.asfortranarray(g)
    fake = 1 << 20  # never read
    p = SSPrepFrames()
    p.frames = SSMatrix(fake, h, w, SS_U16, SS_DEVICE)
    p.n_frames = 1
    p.gather = g.ctypes.data
    p.block_h, p.n_blocks = hb, nb
    p.out = SSMatrix(fake, hb, nb, SS_U16, SS_DEVICE)
    p.gpu_device_id = -1
    lib = _lib.load()
    rc = lib.ss_prepare_frames(C.byref(p))
    return rc, lib.ss_last_error().decode()


def _refused(r):
    return r[0] != 0 and "outside the cropped frame" in r[1]


# whole lines of a frame of 2^31 pixels and more: the last entry has wrapped below zero
@pytest.mark.parametrize("h,w", [(1 << 30, 3), (1 << 29, 5), ((1 << 30) + 1, 2)])
def test_a_map_whose_entries_wrap_is_refused(h, w):
    line = (np.arange(w, dtype=np.int64) * h + (h - 1 if w == 2 else 0)).astype(np.int64)
    assert line[-1] >= 1 << 31
    wrapped = (line & 0xFFFFFFFF).astype(np.uint32).view(np.int32)
    assert _refused(_call(h, w, wrapped[:, None]))


@pytest.mark.parametrize("bad", [-2, 12, 1 << 30, -(1 << 31), (1 << 31) - 1])
def test_an_entry_outside_the_frame_is_refused(bad):
    lines = np.arange(12, dtype=np.int64).reshape(4, 3, order="F")  # 3 columns of 4 rows: block b is row b
    g = lines.T.copy()
    for r in range(3):
        for b in range(4):
            m = g.copy()
            m[r, b] = bad
            assert _refused(_call(4, 3, m)), (r, b)
    assert not _refused(_call(4, 3, g))
