"""The workloads this package is timed on: calls of its public entry points with synthetic recordings.

A case is a dict of sizes and options; ``prepare`` builds what a program holds before the call (its
frames, template, settings, and the batch or session it keeps), ``run`` is one call. Recordings are
Gaussian-blob templates sampled along a per-line random walk with one jump per frame and Poisson
noise at a 200-photon peak, the statistics of ``steadyscan_b200.synth`` rendered on the GPU.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from steadyscan_b200 import api, prep, synth

DTYPES = {"u16": torch.uint16, "f16": torch.float16, "f32": torch.float32, "f64": torch.float64}
NP_DTYPES = {"u16": np.uint16, "f32": np.float32, "f64": np.float64}
BYTES = {"u16": 2, "f16": 2, "f32": 4, "f64": 8}

# frame sizes (lines x pixels) and knot spacings of the ragged batch
RAGGED_SIZES = [(128, 128), (256, 512), (512, 512), (796, 512)]
RAGGED_SPACING = [1, 2, 4]


def listed():
    return [
        # the smallest call: a few frames of a small field at the default settings (precision D, FP64
        # frames, as a MEX caller has them), where launches and host work count
        {"name": "group_tiny_d", "call": "group", "h": 64, "w": 64, "nk": 17, "n": 4, "dtype": "f64", "prec": "D",
         "lam": 0.0, "host": True},
        # one set per call from host memory, in FP64: 50 camera frames of 256 x 256, knots every 4 lines
        {"name": "group_256_d", "call": "group", "h": 256, "w": 256, "nk": 65, "n": 50, "dtype": "u16", "prec": "D",
         "lam": 1e-2, "host": True},
        # a session that keeps its template on the GPU and aligns the next 32 frames as they come
        {"name": "session_512_s", "call": "session", "h": 512, "w": 512, "nk": 257, "n": 32, "dtype": "u16", "prec": "S",
         "lam": 5e-3, "host": False},
        # a recording's groups in one call from page-locked host memory (upload and results included)
        {"name": "groups_512_s", "call": "groups", "h": 512, "w": 512, "nk": 257, "n": 640, "group": 64, "dtype": "u16",
         "prec": "S", "lam": 5e-3, "host": True},
        # the headline workload: 2000 frames in groups of 64, resident on the GPU, run again and again
        {"name": "batch_512_s", "call": "batch", "h": 512, "w": 512, "nk": 257, "n": 2000, "group": 64, "dtype": "u16",
         "prec": "S", "lam": 5e-3, "host": False},
        # groups of mixed length, frame size and knot spacing in one call
        {"name": "ragged_s", "call": "ragged", "groups": 24, "longest": 128, "dtype": "u16", "prec": "S",
         "lam": 1e-2},
        # a whole recording through the driver's estimate loop (sets with an overlap frame, validity
        # flags) at the default precision, its prefiltered FP64 frames already on the GPU
        {"name": "recording_d", "call": "recording", "h": 256, "w": 512, "nk": 65, "n": 400, "per_set": 100,
         "dtype": "f64", "prec": "D", "lam": 0.0, "host": False},
        # raw camera frames put into block-matrix order
        {"name": "reorder_u16", "call": "prepare", "h": 512, "w": 512, "nk": 257, "n": 1000, "dtype": "u16",
         "out": "u16", "sd": 0.0, "med": False, "crop": 0},
        # the full prefilter: blur, division by the frame's median, block order, FP64
        {"name": "prefilter_512", "call": "prepare", "h": 512, "w": 512, "nk": 257, "n": 256, "dtype": "u16",
         "out": "f64", "sd": 1.0, "med": True, "crop": 0},
        # odd sizes: FP32 frames with margins to crop, a wider blur, FP32 out
        {"name": "prefilter_odd", "call": "prepare", "h": 203, "w": 397, "nk": 28, "n": 30, "dtype": "f32",
         "out": "f32", "sd": 2.5, "med": True, "crop": 5},
        # motion-corrected images of one set
        {"name": "reconstruct_512", "call": "reconstruct", "h": 512, "w": 512, "nk": 257, "n": 64, "dtype": "f32"},
        # the knot-chain solve on its own: 64 frames of 256 knots
        {"name": "solve_16385", "call": "solve", "n": 16385},
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    call = rng.choice(["group", "session", "groups", "batch", "ragged", "recording", "prepare", "prepare",
                       "reconstruct", "solve"])
    if call == "solve":
        return {"call": call, "n": _log(rng, 40, 60000)}
    if call == "ragged":
        return {"call": call, "groups": rng.randint(4, 32), "longest": _log(rng, 8, 128), "dtype": "u16", "prec": "S",
                "lam": 1e-2}
    k = rng.choice([2, 4, 8])
    h = k * rng.randint(64 // k, 640 // k)
    # knots every 2, 4 or 8 lines, or (the timing model takes any count) at a fraction of a line
    nk = h // k + 1 if rng.random() < 0.75 else rng.randint(h // 8 + 1, h // 2)
    w = rng.randint(64, 640)
    c = {"call": call, "h": h, "w": w, "nk": nk}
    # never more pixels than 400 frames of 256 x 512 (precision D) or 600 of 512 x 512 (others)
    most_d, most = max(4, 400 * 256 * 512 // (h * w)), max(4, 600 * 512 * 512 // (h * w))
    if call == "prepare":
        dtype = rng.choice(["u16", "u16", "f32", "f64"])
        plain = rng.random() < 0.4
        c.update(n=_log(rng, 1, min(400, most)), dtype=dtype, out=dtype if plain else rng.choice(["f64", "f32"]),
                 sd=0.0 if plain else round(rng.uniform(0.5, 4.0), 2), med=(not plain) and rng.random() < 0.7,
                 crop=rng.choice([0, 0, 3]))
        return c
    if call == "reconstruct":
        c.update(n=_log(rng, 1, 64), dtype=rng.choice(["f32", "f64"]))
        return c
    if call == "group":
        prec = rng.choice(["D", "D", "S"])
        c.update(n=_log(rng, 2, 60), dtype=rng.choice(["u16", "f64", "f32"]), prec=prec, lam=rng.choice([0.0, 1e-2]),
                 host=True)
    elif call == "session":
        c.update(n=_log(rng, 2, 64), dtype=rng.choice(["u16", "f16", "f32"]), prec="S", lam=5e-3, host=False)
    elif call == "recording":
        c.update(n=_log(rng, 20, max(20, min(400, most_d))), per_set=rng.choice([50, 100, 500]),
                 dtype=rng.choice(["u16", "f64"]), prec="D", lam=0.0, host=False)
    else:
        prec = rng.choice(["S", "S", "D"])
        c.update(n=_log(rng, 16, max(16, min(600, most_d if prec == "D" else most))),
                 group=rng.choice([16, 32, 64, 100]), dtype=rng.choice(["u16", "u16", "f32"]), prec=prec, lam=5e-3,
                 host=call == "groups")
    return c


# ------------------------------------------------------------------------------------------------
# synthetic recordings

def _fold(v, clip):
    """A walk kept within +-clip by reflection at the ends."""
    return clip - ((v - clip) % (4 * clip) - 2 * clip).abs()


def _walk(n, h, sigma, clip, gen, dev):
    """Per-line (dx, dy) of n frames of h lines: a random walk with one jump of up to 4 px per frame."""
    steps = torch.randn((n * h, 2), generator=gen, device=dev, dtype=torch.float64) * sigma
    line = (torch.rand(n, generator=gen, device=dev, dtype=torch.float64) * h).long().clamp(max=h - 1)
    at = torch.arange(n, device=dev) * h + line
    ang = torch.rand(n, generator=gen, device=dev, dtype=torch.float64) * (2 * math.pi)
    mag = torch.rand(n, generator=gen, device=dev, dtype=torch.float64) * 4
    steps[at] += torch.stack([mag * torch.cos(ang), mag * torch.sin(ang)], 1)
    return _fold(torch.cumsum(steps, 0), clip).view(n, h, 2)


def _frames(tmpl, walk, h, w, dtype, gen, dev):
    """n frames as a (n, pixels, lines) tensor (each frame column-major) of photon counts."""
    T = torch.tensor(np.ascontiguousarray(tmpl), device=dev)
    th, tw = T.shape
    n = walk.shape[0]
    bg = T.min()
    out = torch.empty((n, w, h), dtype=dtype, device=dev)
    jj = torch.arange(w, device=dev, dtype=torch.float64)[None, :, None]
    ll = torch.arange(h, device=dev, dtype=torch.float64)[None, None, :]
    step = max(1, (16 << 20) // (h * w))
    for a in range(0, n, step):
        x = jj + walk[a:a + step, None, :, 0]
        y = ll + walk[a:a + step, None, :, 1]
        x0, y0 = torch.floor(x), torch.floor(y)
        fx, fy = x - x0, y - y0
        xl, yl = x0.long(), y0.long()
        inside = (xl >= 0) & (yl >= 0) & (xl < tw - 1) & (yl < th - 1)
        xl, yl = xl.clamp(0, tw - 2), yl.clamp(0, th - 2)
        v = (1 - fx) * ((1 - fy) * T[yl, xl] + fy * T[yl + 1, xl]) + fx * ((1 - fy) * T[yl, xl + 1]
                                                                           + fy * T[yl + 1, xl + 1])
        cnt = torch.poisson(torch.where(inside, v, bg), generator=gen).clamp(0, 65535)
        out[a:a + step] = cnt.to(torch.int32).to(dtype) if dtype == torch.uint16 else cnt.to(dtype)
    return out


def _block_map(blk, nblocks, dev):
    """Column-major pixel index of every entry (block, row) of the block matrix, -1 past a block's end."""
    blk = torch.tensor(np.ascontiguousarray(np.asarray(blk).T), device=dev).reshape(-1)
    order = torch.argsort(blk, stable=True)
    count = torch.bincount(blk, minlength=nblocks + 1)[1:]
    start = torch.cumsum(count, 0) - count
    row = torch.arange(int(count.max()), device=dev)[None, :]
    return torch.where(row < count[:, None], order[(start[:, None] + row).clamp(max=order.numel() - 1)], -1)


def _blocks(frames, idx):
    """(n, pixels, lines) frames in block order: n x blocks x rows, zeros past a block's end."""
    v = frames.reshape(frames.shape[0], -1)
    v = v.view(torch.int16) if v.dtype == torch.uint16 else v
    out = torch.where(idx >= 0, v[:, idx.clamp(min=0)], torch.zeros((), dtype=v.dtype, device=v.device))
    return out.view(frames.dtype)


def _template(h, w, rng):
    # column-major, as a caller that goes through the C ABI keeps it
    return np.asfortranarray(synth.make_template(h, w, max(2, round(400 * h * w / (512 * 512))), (2.0, 6.0), rng))


def _pinned(flat):
    host = torch.empty(flat.shape, dtype=flat.dtype, pin_memory=True)
    host.copy_(flat)
    return host


def _setup(h, w, nk, prec, lam, rng, more=None):
    tmpl = _template(h, w, rng)
    s = prep.init_settings(dict({"nknots": nk, "gpu_forced_precision": prec, "lambda": lam}, **(more or {})), tmpl, h,
                           w)
    return tmpl, s, prep.block_layout(s), prep.template_gradients(tmpl)


def _group(setup, h, w, n, dtype, host, sigma, gen, dev):
    tmpl, s, lay, grads = setup
    idx = _block_map(lay.prevknotind, lay.frame_w, dev)
    flat = _blocks(_frames(tmpl, _walk(n, h, sigma, 6.0, gen, dev), h, w, DTYPES[dtype], gen, dev), idx).reshape(-1)
    if host:
        keep = _pinned(flat)
        bm = keep.numpy().reshape(lay.frame_h, lay.frame_w * n, order="F")
    else:
        bm = flat.view(lay.frame_w * n, lay.frame_h).T
        keep = flat
    return prep.boundary_arguments(s, tmpl, bm, n, layout=lay, gradients=grads), keep


def _ragged(case):
    """Sizes, knot spacings and lengths of a ragged batch: of the case, not of the seed."""
    rng = np.random.default_rng([case["groups"], case["longest"]])
    for _ in range(case["groups"]):
        h, w = RAGGED_SIZES[int(rng.integers(len(RAGGED_SIZES)))]
        yield h, w, RAGGED_SPACING[int(rng.integers(len(RAGGED_SPACING)))], int(rng.integers(2, case["longest"] + 1))


def prepare(case, seed):
    dev = torch.device("cuda", 0)
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    call, st = case["call"], {"call": case["call"]}
    if call == "solve":
        n = case["n"]
        # normal equations of a chain of knots: every block of pixels couples its two knots
        g = torch.randn((n + 1, 24, 2), generator=gen, device=dev, dtype=torch.float64) * 8
        f = torch.rand((n + 1, 24), generator=gen, device=dev, dtype=torch.float64)
        own, nxt = 1 - f, f
        gg = torch.stack([g[..., 0] ** 2, g[..., 1] ** 2, g[..., 0] * g[..., 1]], -1)
        a = (gg * (own ** 2)[..., None]).sum(1)
        b = (gg * (nxt ** 2)[..., None]).sum(1)
        o = (gg * (own * nxt)[..., None]).sum(1)
        st["diag"] = (a[1:] + b[:-1] + torch.tensor([1e-2, 1e-2, 0.0], dtype=torch.float64, device=dev)).contiguous()
        st["coup"] = torch.stack([o[1:n, 0], o[1:n, 1], o[1:n, 2], o[1:n, 2]], -1).contiguous()
        st["rhs"] = torch.randn((n, 2), generator=gen, device=dev, dtype=torch.float64) * 100
        return st
    if call == "ragged":
        setups, groups, keep = {}, [], []
        for h, w, k, n in _ragged(case):
            if (h, w, k) not in setups:
                setups[h, w, k] = _setup(h, w, h // k + 1, case["prec"], case["lam"], rng,
                                         {"move_thresh": 1e-3, "max_iter": 30})
            a, t = _group(setups[h, w, k], h, w, n, case["dtype"], False, 0.15, gen, dev)
            groups.append(a)
            keep.append(t)
        st.update(groups=groups, keep=keep)
        return st
    h, w, nk, n = case["h"], case["w"], case["nk"], case["n"]
    if call == "prepare":
        c = case["crop"]
        # the block map of the cropped lines: block b holds lines ceil(b hc / nb) .. of nb blocks
        nb = nk - 1
        blk = np.arange(h - 2 * c) * nb // (h - 2 * c) + 1
        lay = prep.BlockLayout(nk, nb, 0, np.tile(blk[:, None], (1, w - 2 * c)), None, None, None, None, None,
                               [c, c, c, c])
        fr = _frames(_template(h, w, rng), _walk(n, h, 0.1, 6.0, gen, dev), h, w, DTYPES[case["dtype"]], gen, dev)
        st.update(frames=fr.permute(2, 1, 0), layout=lay, sd=case["sd"], med=case["med"], out=NP_DTYPES[case["out"]])
        return st
    if call == "reconstruct":
        tmpl, s, lay, _ = _setup(h, w, nk, "S", 0.0, rng)
        walk = _walk(n + 1, h, 0.1, 6.0, gen, dev)
        fr = _frames(tmpl, walk[:n], h, w, DTYPES[case["dtype"]], gen, dev)
        line = torch.round(torch.arange(nk, device=dev, dtype=torch.float64) * (h / (nk - 1))).long()
        at = torch.arange(n, device=dev)[:, None] * h + line[None, :]
        kn = walk.view(-1, 2)[at].permute(2, 1, 0).cpu().numpy()
        st.update(frames=fr.permute(2, 1, 0), dx=np.asfortranarray(kn[0]), dy=np.asfortranarray(kn[1]), settings=s,
                  shape=(h, w))
        return st
    setup = _setup(h, w, nk, case["prec"], case["lam"], rng)
    if call in ("group", "session", "recording"):
        a, keep = _group(setup, h, w, n, case["dtype"], case["host"], 0.1, gen, dev)
        st.update(args=a, keep=keep, per_set=case.get("per_set"))
        if call == "session":
            st["session"] = api.Session(a)
        return st
    groups, keep = [], []
    for f in range(0, n, case["group"]):
        a, t = _group(setup, h, w, min(case["group"], n - f), case["dtype"], case["host"], 0.1, gen, dev)
        groups.append(a)
        keep.append(t)
    st.update(groups=groups, keep=keep)
    if call == "batch":
        st["batch"] = api.Batch(groups)
    return st


# ------------------------------------------------------------------------------------------------
# one call

KEYS = ["dx", "dy", "frame_corr", "residrms", "blocks_used"]


def _all(results):
    out = {k: np.concatenate([np.asarray(r[k]).reshape(-1, order="F") for r in results]) for k in KEYS}
    out["iter_used"] = np.array([r["iter_used"] for r in results])
    out["stop_reason"] = np.array([r["stop_reason"] for r in results])
    return out


def run(st):
    call = st["call"]
    if call == "group":
        r = api.align_group(st["args"])
        return {k: r[k] for k in KEYS + ["iter_used", "stop_reason", "mask"]}
    if call == "session":
        b = api.Batch([st["args"]], sessions=[st["session"]])
        b.run()
        r = b.collect()
        b.close()
        return _all(r)
    if call in ("groups", "ragged"):
        return _all(api.align_groups(st["groups"], want_mask=False))
    if call == "batch":
        st["batch"].run()
        return _all(st["batch"].collect())
    if call == "recording":
        r = api.estimate_displacements(st["args"], frames_per_set=st["per_set"])
        return {k: v for k, v in r.items() if k != "n_sets"}
    if call == "prepare":
        r = api.prepare_frames(st["frames"], st["layout"], pregauss=st["sd"], mednorm=st["med"], out_dtype=st["out"])
        return r.view(torch.int16) if r.dtype == torch.uint16 else r  # the same bytes: torch indexes no uint16
    if call == "reconstruct":
        return api.reconstruct_frames(st["frames"], st["dx"], st["dy"], st["settings"], st["shape"])
    return api.solve_block_tridiagonal(st["diag"], st["coup"], st["rhs"])


# ------------------------------------------------------------------------------------------------
# what a call cannot do without, and its values in 64 bits

def work(case):
    """Inputs read once, outputs written once; the arithmetic of a search is that of one iteration:
    two half-steps (warp, sample, gradients and sums, then one trial) and the correlation."""
    call = case["call"]
    if call == "solve":  # 9 + 2 doubles in, 2 out; one 2x2 block elimination and substitution per knot
        return {"bytes": case["n"] * 13 * 8.0, "flops": case["n"] * 50.0}
    if call == "ragged":
        px = float(sum(h * w * n for h, w, _, n in _ragged(case)))
        return {"bytes": px * BYTES[case["dtype"]], "flops": px * 220.0}
    px = float(case["h"] * case["w"] * case["n"])
    if call == "prepare":
        inner = (case["h"] - 2 * case["crop"]) * (case["w"] - 2 * case["crop"]) * case["n"]
        taps = 2 * math.ceil(9.6 * case["sd"]) + 1 if case["sd"] else 0
        return {"bytes": px * BYTES[case["dtype"]] + float(inner) * BYTES[case["out"]], "flops": px * 4.0 * taps}
    if call == "reconstruct":
        return {"bytes": px * (BYTES[case["dtype"]] + 5), "flops": px * 100.0}
    knots = 2.0 * case["nk"] * case["n"] * 8
    mask = px if call == "group" else 0.0
    return {"bytes": px * BYTES[case["dtype"]] + mask + 2 * knots, "flops": px * 220.0}


def _exact_solve(st):
    """Block elimination along the chain, one 2x2 block at a time."""
    d = st["diag"].cpu().numpy()
    c = st["coup"].cpu().numpy()
    b = st["rhs"].cpu().numpy().copy()
    n = d.shape[0]
    D = np.stack([np.stack([d[:, 0], d[:, 2]], -1), np.stack([d[:, 2], d[:, 1]], -1)], 1)
    C = np.stack([np.stack([c[:, 0], c[:, 2]], -1), np.stack([c[:, 3], c[:, 1]], -1)], 1)
    for i in range(1, n):
        t = np.linalg.solve(D[i - 1], C[i - 1]).T
        D[i] -= t @ C[i - 1]
        b[i] -= t @ b[i - 1]
    x = np.empty_like(b)
    x[n - 1] = np.linalg.solve(D[n - 1], b[n - 1])
    for i in range(n - 2, -1, -1):
        x[i] = np.linalg.solve(D[i], b[i] - C[i] @ x[i + 1])
    return x


def _exact_prepare(case, st):
    fr = st["frames"].permute(2, 1, 0)  # n, pixels, lines
    n, w, h = fr.shape
    lay, sd, c = st["layout"], st["sd"], case["crop"]
    idx = _block_map(lay.prevknotind, lay.frame_w, fr.device)
    hb = idx.shape[1]
    out = torch.empty((n, lay.frame_w, hb), dtype=fr.dtype if st["out"] == np.uint16 else torch.float64,
                      device=fr.device)
    for f in range(n):
        v = fr[f] if st["out"] == np.uint16 else fr[f].to(torch.float64)
        if sd > 0:  # the periodic Gaussian on the frame padded by L zeros, in the frequency domain
            pad = math.ceil(math.sqrt(2 * sd ** 2 * math.log(10000 / (math.sqrt(2 * math.pi) * sd))))

            def gauss(m):
                d = torch.arange(m, device=fr.device, dtype=torch.float64)
                d = torch.minimum(d, m - d)
                g = torch.exp(-d * d / (2 * sd * sd))
                return g / g.sum()

            pw, ph = w + pad, h + pad
            kern = gauss(pw)[:, None] * gauss(ph)[None, :]
            v = torch.fft.irfft2(torch.fft.rfft2(v, s=(pw, ph)) * torch.fft.rfft2(kern), s=(pw, ph))[:w, :h]
        if st["med"]:
            q = torch.sort(v.reshape(-1)).values
            v = v / ((q[(q.numel() - 1) // 2] + q[q.numel() // 2]) / 2)
        out[f] = _blocks(v[None, c:w - c, c:h - c], idx)[0]
    out = out.view(n * lay.frame_w, hb).T
    return out.view(torch.int16) if out.dtype == torch.uint16 else out


def exact(case, seed):
    # The alignment and the reconstruction are searches that stop by their own rules (a trial is
    # accepted or halved, an iteration is the last when a threshold is met): their outputs are defined
    # by that path and have no closed value of their own.
    if case["call"] == "solve":
        return _exact_solve(prepare(case, seed))
    if case["call"] == "prepare":
        return _exact_prepare(case, prepare(case, seed))
    return None
