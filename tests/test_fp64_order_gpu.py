"""FP64 line searches compare a trial's error with the assembly's: both add a column's pixels in the same
order, so that a trial that moves no knot is no improvement. Geometries whose columns differ in tfrac (a
fractional number of lines per knot) are assembled row by row; the twin of each, whose first row (masked)
has another basex, is searched row by row too."""
import numpy as np
import pytest

from steadyscan_b200 import api
from tests.helpers import make_args

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,w,nk", [(38, 32, 9), (45, 32, 10), (40, 36, 10)])
@pytest.mark.parametrize("dtype", [np.float64, np.uint16])
def test_trials_add_in_the_assembly_order(h, w, nk, dtype):
    args, _, _ = make_args(nlines=h, linewidth=w, nknots=nk, n_frames=6, seed=h + 2, frame_dtype=dtype,
                           settings={"max_iter": 8, "gpu_flags": "e", "gpu_forced_precision": "D"})
    tf, bx = np.array(args["tfrac"]), np.array(args["basex"])
    assert tf.shape[0] % 4 == 0 and not (tf == tf[:, :1]).all() and (bx[:4, 0] == bx[0, 0]).all()
    bm = np.array(args["base_mask"])
    bm[0, 0] = 0
    twin_bx = bx.copy()
    twin_bx[0, 0] += 0.5
    # (a group's results do not depend on a masked pixel's position)
    a = api.align_group(dict(args, base_mask=bm), want_history=True)
    b = api.align_group(dict(args, base_mask=bm, basex=twin_bx), want_history=True)
    assert a["iter_used"] == b["iter_used"] and a["iter_used"] >= 3
    for k in ("dx", "dy", "mask", "iteration_errvals"):
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)
