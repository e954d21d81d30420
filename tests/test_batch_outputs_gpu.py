"""Host outputs of a batch belong to the caller until they are collected: a run neither reads nor writes them."""
import ctypes
import mmap

import numpy as np
import pytest

from steadyscan_b200 import api
from tests.helpers import make_args

pytestmark = pytest.mark.gpu

PAGE = mmap.PAGESIZE


class _Pages:
    """Fresh anonymous pages, and which of them the process has touched (mincore)."""

    def __init__(self, n):
        self.n = n
        self.m = mmap.mmap(-1, n, flags=mmap.MAP_PRIVATE | mmap.MAP_ANONYMOUS)
        self.addr = ctypes.addressof(ctypes.c_char.from_buffer(self.m))
        self.libc = ctypes.CDLL(None, use_errno=True)

    def resident(self):
        vec = (ctypes.c_ubyte * (-(-self.n // PAGE)))()
        rc = self.libc.mincore(ctypes.c_void_p(self.addr), ctypes.c_size_t(self.n), vec)
        assert rc == 0, ctypes.get_errno()
        return sum(v & 1 for v in vec)


def test_a_run_leaves_the_outputs_alone():
    args, _, _ = make_args(nlines=64, linewidth=64, nknots=33, n_frames=40, frame_dtype=np.uint16,
                           settings={"max_iter": 4})
    b = api.Batch([args], want_mask=True)
    b.run()
    first = b.collect()[0]
    ref = {k: np.array(first[k]) for k in ("dx", "dy", "mask")}
    o = b._outs[0]
    pages = {"dx_knots": _Pages(ref["dx"].nbytes), "dy_knots": _Pages(ref["dy"].nbytes), "mask": _Pages(ref["mask"].size)}
    assert ref["mask"].size > 2 * 65536
    seen = _Pages(4 * PAGE)  # the measure itself: a written page shows
    assert seen.resident() == 0
    seen.m[PAGE] = 1
    assert seen.resident() >= 1
    for k, p in pages.items():  # new outputs for the next run
        setattr(o, k, p.addr)
        assert p.resident() == 0
    b.run()
    for k, p in pages.items():
        assert p.resident() == 0, k
    b.collect()
    got = np.frombuffer(pages["mask"].m, np.uint8, ref["mask"].size).reshape(ref["mask"].shape, order="F")
    np.testing.assert_array_equal(got.astype(bool), ref["mask"])
    for k in ("dx", "dy"):
        np.testing.assert_array_equal(np.frombuffer(pages[k + "_knots"].m, np.float64, ref[k].size), ref[k])


def test_a_mask_outlives_the_next_collect():
    args, _, _ = make_args(nlines=32, linewidth=32, nknots=9, n_frames=4, settings={"max_iter": 4})
    b = api.Batch([args], want_mask=True)
    b.run()
    first = b.collect()[0]["mask"]
    ref = first.copy()
    assert ref.any()
    first[:] = False  # the caller's own
    b.run()
    second = b.collect()[0]["mask"]
    np.testing.assert_array_equal(second, ref)
    assert not first.any() and second.flags.f_contiguous
