"""A reconstruction on a device whose memory is nearly taken: fewer iterates are kept (and the outputs'
swept again), then fewer frames at a time, before the call gives up. In a process of its own, whose work
pool holds nothing yet."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import sys
import numpy as np, torch
sys.path.insert(0, sys.argv[1])
from oracle import reconstruct as rc
from steadyscan_b200 import api, prep, synth
leave = int(sys.argv[2])
n, reps = 256, 16
rec = synth.make_recording(n, n, 4, 65, n_blobs=40, sigma=(2.0, 6.0), walk_sigma=0.1, clip_px=2.0, jumps_per_frame=0,
                           jump_px=0.0, seed=3, nlines=n, linewidth=n, noise=True)
s = prep.init_settings({"nknots": 65}, rec.template, n, n)
rng = np.random.default_rng(0)
nf = 4 * reps
fr = np.concatenate([rec.frames * (0.5 + 0.1 * k) for k in range(reps)], axis=2).astype(np.float32)
dx, dy = rng.normal(0, 0.4, (65, nf)), rng.normal(0, 0.4, (65, nf))
small = prep.init_settings({"nknots": 5}, rec.template[:24, :24], 24, 24)
for dt in (np.float32, np.float64):  # every kernel loaded before the memory is taken
    api.reconstruct_frames(fr[:24, :24, :2].astype(dt), dx[:5, :2], dy[:5, :2], small, (24, 24), out_dtype=dt)
torch.cuda.synchronize()
free = torch.cuda.mem_get_info()[0]
held = torch.empty(max(0, free - leave), dtype=torch.uint8, device="cuda") if leave else None
g = api.reconstruct_frames(fr, dx, dy, s, (n, n))
its, iv = [int(v) for v in g["iterations"]], 1
kept = []
for it in its:  # sweeps, and the sweep whose iterate is the output
    kept.append(it - iv)
    assert it > 0 and it % iv == 0
    iv = int(max(1, min(10, rc.round_half_away(np.sqrt(np.float32(it))))))
assert any(it - k >= 5 for it, k in zip(its, kept)), "no output further back than the shortest ring holds"
for f in (0, 1, 5, 22, 47, 63):
    out, mask, _ = rc.invert_bilinear_sampling(fr[:, :, f], dx[:, f:f + 1], dy[:, f:f + 1], s["basex"], s["basey"],
                                               s["tfrac"], s["prevknotind"], n, n, stop_at=[kept[f] + 1])
    np.testing.assert_array_equal(g["mask"][:, :, f], mask[:, :, 0])
    m = mask[:, :, 0]
    np.testing.assert_allclose(g["data_corrected"][:, :, f][m], out[:, :, 0][m], rtol=0,
                               atol=1e-4 * np.abs(out[:, :, 0][m]).max())
print("free", free >> 20, "MB, sweeps", sorted(set(its)))
print("child ok")
"""

# 64 frames of 256 x 256: the longest ring wants about 870 MB, the shortest one 500 MB; in 300 MB the frames
# run in parts
@pytest.mark.parametrize("leave", [0, 700 << 20, 300 << 20])
def test_a_call_fits_the_memory_that_is_left(leave):
    r = subprocess.run([sys.executable, "-c", CHILD, ROOT, str(leave)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "child ok" in r.stdout, r.stdout[-2000:] + r.stderr[-3000:]
