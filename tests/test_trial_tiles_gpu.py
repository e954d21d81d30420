"""Trial rounds of precision 'S' whose tiles hold 8, 16 or 32 frames (chosen by how many block columns
are searching): a group's result is the same bits alone, where its rounds take the smallest tiles, and
in a batch large enough for the largest."""
import numpy as np
import pytest

from steadyscan_b200 import api
from tests.helpers import make_args

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw,copies", [(dict(nlines=256, linewidth=256, nknots=129, n_frames=20), 12),
                                       (dict(nlines=128, linewidth=128, nknots=129, n_frames=33), 20),
                                       (dict(nlines=64, linewidth=96, nknots=25, n_frames=9), 30)])
def test_tile_sizes_give_the_same_bits(kw, copies):
    args, _, _ = make_args(seed=kw["n_frames"], frame_dtype=np.uint16,
                           settings={"lambda": 5e-3, "gpu_forced_precision": "S", "max_iter": 12}, **kw)
    alone = api.align_group(args)
    for r in api.align_groups([args] * copies):
        assert r["iter_used"] == alone["iter_used"]
        for k in ("dx", "dy", "frame_corr", "residrms", "mask"):
            np.testing.assert_array_equal(r[k], alone[k])
