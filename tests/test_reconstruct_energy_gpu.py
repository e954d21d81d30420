"""The energies that stop a reconstruction, on templates of both parities each way: at every check before a
frame's stop the energy of the oracle's iterates in FP64 had decreased, and at its stop it had not, to
the rounding of the compared FP32 values; and the outputs are the oracle's iterates. The frames are dark
but for the lines or pixels that map to the template's last two rows or columns, so that the energy's
entries there (quads that the edge cuts, paired or single stencil loads) decide: one left out or taken
twice moves the stop."""
import numpy as np
import pytest

from oracle import reconstruct as rc
from steadyscan_b200 import api
from tests.helpers import make_args

pytestmark = pytest.mark.gpu

EPS32 = 2.0 ** -24


class _Frame:
    """One frame's system and its iterates (the oracle's, by replaying stops)."""

    def __init__(self, frame, dxk, dyk, s, shape):
        self.a = (frame, dxk[:, None], dyk[:, None], s["basex"], s["basey"], s["tfrac"], s["prevknotind"], *shape)
        self.kw = dict(regfac=s.get("ibs_regfac", 3e-3), aspect=s.get("ibs_template_pixel_aspect_ratio", 1.0))
        th, tw = shape
        wy, ww = rc.bilinear_map_linear_constraints(frame, dxk, dyk, *self.a[3:7], tw, th)
        self.q = (ww + rc.imageadjdiffquadmat(tw, th, 1.0 / self.kw["aspect"]) * self.kw["regfac"]).tocsr()
        self.wy = wy
        self.seen = {}

    def iterate(self, k):
        """(iterate k over the mask, mask); k >= 1"""
        if k not in self.seen:
            out, mask, _ = rc.invert_bilinear_sampling(*self.a, **self.kw, stop_at=[k + 1])
            m = mask.reshape(-1, order="F")
            self.seen[k] = out.reshape(-1, order="F")[m].astype(np.float64), m
        return self.seen[k]

    def energy(self, k):
        """Energy of iterate k and a bound on the rounding of its FP32 value: the linear term is an FP32 sum
        (at most 8 terms of a thread, 8 + 64 of the partial sums, a product each), the quadratic one FP64,
        their difference rounded once; and the two iterates may differ by FP32 rounding of a sweep's
        8-term sums, to which the energy reacts by its gradient."""
        x, m = self.iterate(k)
        q = self.q[m][:, m]
        qx, l = q @ x, self.wy[m]
        e = float(x @ qx - 2.0 * (l @ x))
        terms = np.abs(l * x).sum()
        rounding = EPS32 * (2 * (8 + 8 + 64 + 1) * terms + abs(e))
        moved = 16 * EPS32 * np.abs(x).max() * 2.0 * np.abs(qx - l).sum()
        return e, rounding + moved


@pytest.mark.parametrize("dh,dw", [(0, 0), (1, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("axis", [0, 1])
def test_stops_follow_the_energy(dh, dw, axis):
    args, rec, s = make_args(n_frames=3, seed=5)
    nk = args["tfrac"].shape[1] + 1
    rng = np.random.default_rng(0)
    dxk, dyk = rng.normal(0, 0.3, (nk, 3)), rng.normal(0, 0.3, (nk, 3))
    shape = (rec.template.shape[0] - dh, rec.template.shape[1] - dw)
    fr = rng.uniform(0, 1000, rec.frames.shape).astype(np.float32)
    at = np.arange(fr.shape[axis])
    lit = (at >= shape[axis] - 2) & (at < shape[axis])
    fr *= lit[:, None, None] if axis == 0 else lit[None, :, None]
    g = api.reconstruct_frames(fr, dxk, dyk, s, shape)
    n, clear = 1, 0
    for f, it in enumerate(int(v) for v in g["iterations"]):
        fm = _Frame(fr[:, :, f], dxk[:, f], dyk[:, f], s, shape)
        assert it % n == 0 and it > n
        for k in range(2 * n, it + 1, n):  # (iterate 0, the first guess, is not among the oracle's outputs)
            (e0, t0), (e1, t1) = fm.energy(k - n), fm.energy(k)
            if abs(e1 - e0) <= t0 + t1:
                continue  # within rounding: either decision
            clear += 1
            assert (e1 < e0) == (k < it), (f, k, it, e0, e1)
        x, m = fm.iterate(it - n)
        got = g["data_corrected"][:, :, f].reshape(-1, order="F")
        np.testing.assert_array_equal(g["mask"][:, :, f].reshape(-1, order="F"), m)
        np.testing.assert_allclose(got[m], x, rtol=0, atol=1e-4 * np.abs(x).max())
        n = int(max(1, min(10, rc.round_half_away(np.sqrt(np.float32(it))))))
    assert clear >= 6  # checks that rounding does not decide
