"""What Batch.collect returns when a batch is run and collected again (no GPU: the library is a stub)."""
import types

import numpy as np

from steadyscan_b200 import api
from tests.helpers import make_args


def test_a_mask_of_an_earlier_collect_keeps_its_values():
    args, _, _ = make_args(nlines=12, linewidth=10, nknots=4, n_frames=2)
    o, a, d = api._outputs(args)
    b = object.__new__(api.Batch)
    b._outs, b._arrays, b._dims, b._h = [o], [a], [d], None
    fill = {"v": 1}

    def collect(handle):  # the library writes the batch's buffers in full
        a["mask"][:] = fill["v"]
        a["blocks_used"][:] = fill["v"]
        return 0

    b._lib = types.SimpleNamespace(ss_batch_collect=collect, ss_batch_destroy=lambda h: None)
    first = b.collect()[0]
    fill["v"] = 0
    second = b.collect()[0]
    assert first["mask"].dtype == np.bool_ and second["mask"].dtype == np.bool_
    assert first["mask"].all() and first["blocks_used"].all()
    assert not second["mask"].any()
    second["mask"][:] = True  # an edit stays the caller's own
    assert not a["mask"].any()
