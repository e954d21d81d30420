"""The FP64 column evaluation at the edges of its row steps, against the oracle: runs of 4 rows per lane
(4 or more lines per knot) and single rows, steps cut short, block heights off 4 rows, few columns per
cluster CTA, geometry shared by the columns and not, every frame storage type."""
import numpy as np
import pytest

from oracle import oracle
from steadyscan_b200 import api
from tests.helpers import make_args

pytestmark = pytest.mark.gpu

# lines, pixels, knots, frames, storage, settings
CASES = [(64, 64, 17, 4, np.float64, {}),                  # 4 lines a knot: 2 steps of 128 rows
         (64, 50, 9, 3, np.uint16, {}),                    # 8 lines, 400 rows: the last step cut short
         (64, 33, 17, 2, np.float32, {}),                  # 4 lines, 132 rows
         (30, 33, 11, 4, np.uint16, {}),                   # 3 lines, 99 rows: off 4 rows
         (32, 31, 33, 2, np.float16, {}),                  # a line a knot, 31 rows: less than a warp
         (48, 40, 4, 5, np.float64, {}),                   # 3 columns of 640 rows
         (32, 48, 2, 2, np.uint16, {}),                    # a single column of 1536 rows
         (40, 36, 10, 4, np.float64, {}),                  # a fractional number of lines a knot: tables differ
         (64, 40, 17, 4, np.float32, {"isbidirectional": True}),
         (64, 64, 17, 4, np.float64, {"gpu_flags": "c"}),  # the difference-image state of flag c
         (64, 64, 17, 6, np.uint16, {"gpu_flags": "M", "haltcorr": 0.97})]


@pytest.mark.parametrize("h,w,nk,n,dtype,st", CASES)
def test_matches_the_oracle(h, w, nk, n, dtype, st):
    args, _, _ = make_args(nlines=h, linewidth=w, nknots=nk, n_frames=n, seed=h + w, frame_dtype=dtype,
                           settings=dict(st, max_iter=12))
    o = oracle.align_group(dict(args, flags="D" + st.get("gpu_flags", "")), n_threads=4)
    g = api.align_group(dict(args, flags="D" + st.get("gpu_flags", "")))
    assert g["iter_used"] == o["iterations"]
    np.testing.assert_array_equal(g["mask"], o["mask"])
    for k in ("dx", "dy", "frame_corr", "residrms"):
        np.testing.assert_allclose(g[k], o[k], rtol=0, atol=1e-6)
