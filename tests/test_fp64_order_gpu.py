"""FP64 line searches compare a trial's error with the assembly's: both add a column's pixels in the same
order, so that a trial that moves no knot is no improvement. Two block columns (more would add up over the
columns in another order), tables that the columns share and not (a fractional number of lines per knot),
runs of 4 rows per lane and single rows."""
import numpy as np
import pytest

from steadyscan_b200 import api
from tests.helpers import make_args

pytestmark = pytest.mark.gpu


# lines, pixels: 4 or more lines a knot in blocks of a multiple of 4 rows, alike and not; off 4 rows; 3 lines
@pytest.mark.parametrize("h,w", [(32, 32), (16, 36), (11, 24), (33, 32), (25, 40), (13, 31), (6, 32)])
@pytest.mark.parametrize("dtype", [np.float64, np.float32, np.uint16])
def test_trials_add_in_the_assembly_order(h, w, dtype):
    """The errors are recorded at an iteration's end: the first frame's is that of its last trial, the
    others' that of the assembly. A first run of frames that are all alike moves frame 0 in its first
    half-step; in a second run frame 1 starts at those knots, beside the neighbour that frame 0 had."""
    nk, nf = 3, 4
    args, _, _ = make_args(nlines=h, linewidth=w, nknots=nk, n_frames=1, seed=h, frame_dtype=dtype,
                           settings={"max_iter": 2, "gpu_flags": "et", "gpu_forced_precision": "D", "gpu_filter_id": 0})
    frame = np.asarray(args["bmData"])
    tf = np.asarray(args["tfrac"])
    W = tf.shape[1]
    assert W == 2
    zero = np.zeros((W + 1, nf))
    a4 = dict(args, bmData=np.asfortranarray(np.tile(frame, (1, nf))), nFrames=nf, est_dx_knots=zero, est_dy_knots=zero)
    first = api.align_group(a4, want_history=True)
    n = W * nf + 1
    after = first["rg_params"][:, 0]  # the chain after the first half-step: x, then y
    moved = [after[:W], after[n:n + W]]
    assert max(np.abs(m).max() for m in moved) > 0  # frame 0 has taken a step
    est = [zero.copy(), zero.copy()]
    for d in range(2):
        est[d][:W, 1] = moved[d]
        est[d][W, 0] = moved[d][0]  # (a frame's last knot and the next frame's first are one)
    second = api.align_group(dict(a4, est_dx_knots=est[0], est_dy_knots=est[1]), want_history=True)
    trial, assembled = first["iteration_errvals"][0, 0], second["iteration_errvals"][0, 1]
    assert trial < first["iteration_errvals"][0, 1]  # (frame 1's, assembled at the start)
    assert trial == assembled
