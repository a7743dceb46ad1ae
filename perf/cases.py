"""Performance cases of the tracking path.

Each case is one piece of work that a program has this framework do, through
the Python binding of the C ABI:

  pair      one frame pair tracked: restore the start state, track_frame, read
            the records back.  With "host" the two frames are handed over from
            page-locked host memory in every pass, as a program that decodes
            files does; otherwise they are resident.
  sequence  a short run with a reference change after every frame: start
            records and first frame in, then per frame load, optional lens
            remap, track, records out.  Frames come from page-locked host
            memory, or ("raw") as sensor mosaics in device memory.
  grad      the subpixel objective, and the objective with its gradient, for
            every grain at given positions.
  disto     the distortion-parameter fit over tracked grain pairs.

"form" names how pairs and sequences are tracked: "plain" is the default
configuration (exact search, Powell refinement), "fast" the tensor-core search
with the adjoint Levenberg-Marquardt refinement.  Frames and motions are the
seeded synthetic workloads of the package.
"""
from __future__ import annotations

import importlib
import math

import numpy as np
import torch

ptk = importlib.import_module("p-tracker_b200")
wl = importlib.import_module("p-tracker_b200.workloads")

RAW_LEFT, RAW_TOP = 24, 8  # margins of the sensor mosaics
STEPS_INC = 0.005          # radians between rotation steps


def _case(kind, dimx, dimy, n, r0, r1, **more):
    """A case with the defaults of the options that it does not give: grains
    of radius r0..r1, a fraction `big` of them of radius R0..R1."""
    c = dict(kind=kind, form="plain", dimx=dimx, dimy=dimy, n=n, r0=float(r0), r1=float(r1), big=0.0, R0=30.0, R1=40.0,
             bits=16, noise=2.0, zone=15, num_rot=10, disp=10.0, rot=0.05, pattern="grain_diameter", pa=1.0, pb=1.0,
             interp="cubic", host=False)
    c.update(more)
    return c


def listed():
    return [
        # the smallest call: a dozen grains in a small 8-bit frame (one view of a close-up), default form
        _case("pair", 256, 192, 12, 9, 13, name="plain_tiny", bits=8, zone=4, num_rot=4, disp=2.0, rot=0.02),
        # some tens of grains in a small 16-bit frame, default form
        _case("pair", 512, 384, 40, 10, 18, name="plain_small", big=0.4, R0=20.0, R1=26.0, zone=6, disp=5.0),
        # an ordinary laboratory pair: 8-bit camera, 400 discs, small motion, default form
        _case("pair", 2048, 1536, 400, 20, 30, name="plain_2048", bits=8, zone=8, disp=3.0, rot=0.02),
        # a full-size 16-bit camera pair with 2000 grains of mixed size, default form (the largest)
        _case("pair", 5616, 3744, 2000, 10, 18, name="plain_5616", big=0.4),
        # a run with jumps, rescue searches, lens remap and reference changes, default form
        _case("sequence", 1536, 1024, 80, 8, 40, name="plain_sequence", frames=3, rescue=40, jump=0.1, remap=True),
        # the small pair in the fast form: launches and latencies
        _case("pair", 512, 384, 40, 10, 18, name="fast_small", form="fast", big=0.4, R0=20.0, R1=26.0, zone=6, disp=5.0),
        # the laboratory pair in the fast form with both frames uploaded in every pass (the host loop)
        _case("pair", 2048, 1536, 400, 20, 30, name="fast_2048_host", form="fast", bits=8, zone=8, disp=3.0, rot=0.02,
              host=True),
        # the full-size pair in the fast form, frames resident
        _case("pair", 5616, 3744, 2000, 10, 18, name="fast_5616", form="fast", big=0.4),
        # the full-size sequence: 5000 grains, remap, jumps and rescues, reference changes, uploads
        _case("sequence", 5616, 3744, 5000, 8, 40, name="fast_sequence", form="fast", frames=2, rescue=40, jump=0.03,
              remap=True),
        # raw camera mosaics demosaiced and rescaled on the device, then tracked
        _case("sequence", 2048, 1536, 400, 20, 30, name="fast_raw_sequence", form="fast", frames=2, raw=-2, zone=8),
        # objective and gradient of the full-size pair's grains
        _case("grad", 5616, 3744, 2000, 10, 18, name="grad_5616", big=0.4),
        # fit of the leading radial term from 2000 grains tracked in 3 images (with the next one free too, the length
        # of the minimisation varies tenfold with the tracking noise)
        _case("disto", 5616, 3744, 2000, 0, 0, name="disto_fit", images=3, dist=1000.0),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["pair"] * 6 + ["sequence"] * 3 + ["grad", "disto"])
    area = _log(rng, 256 * 192, 5616 * 3744)
    dimx = min(5616, max(256, int(math.sqrt(area * rng.uniform(1.2, 1.7)))))
    dimy = min(3744, max(192, int(area / dimx)))
    if kind == "disto":
        n = int(_log(rng, 100, 2000))
        return _case("disto", max(dimx, 1024), max(dimy, 768), n, 0, 0, images=rng.randint(1, 4 if n < 1400 else 3),
                     dist=rng.uniform(300.0, 1000.0))
    form = rng.choice(["plain", "fast"])
    r0 = rng.uniform(8.0, 24.0)
    r1 = r0 + rng.uniform(2.0, 16.0)
    big = rng.choice([0.0, 0.2, 0.4])
    zone = rng.randint(3, 15)
    disp = min(10.0, 0.7 * zone)
    cell = 2.0 * max(r1, 40.0 if big else 0.0) + 2.0 * disp + 12.0
    fit = max(4.0, 0.55 * dimx * dimy / (cell * cell))
    n = int(min(_log(rng, max(4.0, fit / 4.0), fit), 2000.0))
    more = dict(form=form, big=big, zone=zone, num_rot=rng.randint(3, 10), disp=disp, rot=rng.choice([0.02, 0.05]),
                bits=rng.choice([8, 16]), noise=rng.choice([2.0, 2.0, 12.0]))
    if rng.random() < 0.25:
        more.update(rng.choice([dict(pattern="circ", pa=float(rng.randint(8, 16))),
                                dict(pattern="rect", pa=float(rng.randint(6, 14)), pb=float(rng.randint(6, 14))),
                                dict(pattern="ring", pa=3.0, pb=float(rng.randint(8, 16)))]))
    if form == "plain" and rng.random() < 0.2:
        more["interp"] = rng.choice(["linear", "quintic"])
    if kind == "pair":
        more["host"] = rng.random() < 0.3
    if kind == "sequence":
        # a rescue zone needs room round the grains: frames of a megapixel and more, fewer grains in the default form
        more.update(frames=rng.randint(2, 3), bits=16, remap=rng.random() < 0.5, noise=2.0)
        if rng.random() < 0.5 and min(dimx, dimy) >= 900:
            more.update(rescue=rng.randint(24, 40), jump=0.05)
        elif rng.random() < 0.4:
            more.update(raw=rng.choice([-1, -2, -20]), remap=False)
        n = min(n, 200 if form == "plain" else 2000)
    return _case(kind, dimx, dimy, n, round(r0, 2), round(r1, 2), **more)


def _preset(c):
    """The case as a workload description of the package."""
    s = 256.0 if c["bits"] == 16 else 1.0
    mix = [(1.0 - c["big"], c["r0"], c["r1"])] + ([(c["big"], c["R0"], c["R1"])] if c["big"] else [])
    p = dict(dimx=c["dimx"], dimy=c["dimy"], maxval=65535 if c["bits"] == 16 else 255, n=c["n"], mix=mix, sig=(1.5, 3.0),
             density=0.02, amp=(60.0 * s, 220.0 * s), bg=10.0 * s, noise=c["noise"] * s, disp=c["disp"], rot=c["rot"],
             zone=c["zone"], num_rot=c["num_rot"], inc_rot=STEPS_INC, rescue_zone=c.get("rescue", 0))
    if c["kind"] == "sequence":
        # the shear of the whole 50-frame run spread over its frames: a few pixels a frame
        p.update(frames=c["frames"] + 1, shear=min(0.5 * c["zone"], 6.0) * c["frames"] / 2.0, rot_walk=0.01, jump=25.0,
                 jump_frac=c.get("jump", 0.0), gap=20.0, disp=0.0, rot=0.0)
        if c.get("remap"):
            p["disto"] = (-2e-9, 1e-16)
    return p


def _tracker(c, p, iraz):
    form = dict(search_method=ptk.SEARCH_BF16, subpix_method=ptk.SUBPIX_ADJOINT_LM) if c["form"] == "fast" else {}
    o = wl.tracker_options(p)
    return ptk.Tracker(c["dimx"], c["dimy"], image_interpolator=c["interp"], iraz=iraz, **form, **o)


def _mosaic(frame):
    """A sensor mosaic on the device that holds the frame at its margins."""
    h, w = frame.shape
    m = np.zeros((h + 2 * RAW_TOP, (w + 2 * RAW_LEFT + 7) // 8 * 8), dtype=np.uint16)
    m[RAW_TOP:RAW_TOP + h, RAW_LEFT:RAW_LEFT + w] = frame
    return torch.from_numpy(m.view(np.int16)).cuda()


def _disto_case(c, seed):
    return wl.make_disto_case(seed=seed, n=c["n"], n_tracked=c["images"], dimx=c["dimx"], dimy=c["dimy"])


def _disto_pairs(d, dist):
    return ptk.disto_pairs(d["refx"], d["refy"], 0.0, dist)


def prepare(case, seed):
    c = case
    if c["kind"] == "disto":
        d = _disto_case(c, seed)
        start, step = d["X"].copy(), np.zeros(14)
        start[2:4] = 0.0
        step[2] = 1e-10
        fit = ptk.DistoFit(d["dimx"], d["dimy"], d["refx"], d["refy"], d["dx"], d["dy"], d["ncc"], 0.7,
                           _disto_pairs(d, c["dist"]))
        return dict(case=c, fit=fit, start=start, step=step)
    p = _preset(c)
    if c["kind"] == "sequence":
        s = wl.make_sequence(p, seed=seed)
        t = _tracker(c, p, iraz=0)
        t.set_grains(s["rec"])
        t.make_patterns(c["pattern"], c["pa"], c["pb"])
        if s["disto"] is not None:
            t.set_distortion(s["disto"])
        frames = [_mosaic(f) if c.get("raw") else ptk.pinned_copy(f) for f in s["frames"]]
        return dict(case=c, t=t, rec=s["rec"], frames=frames)
    s = wl.make_pair(p, seed=seed)
    t = _tracker(c, p, iraz=1000)
    t.set_grains(s["rec"])
    t.make_patterns(c["pattern"], c["pa"], c["pb"])
    ref, cur = ptk.pinned_copy(s["ref"]), ptk.pinned_copy(s["cur"])
    t.load_frame(0, ref)
    t.load_frame(1, cur)
    t.snapshot_grains()
    state = dict(case=c, t=t, ref=ref, cur=cur)
    if c["kind"] == "grad":
        t.precompute()
        state["X"] = _positions(s, seed)
    t.synchronize()
    return state


def _positions(s, seed):
    """Where objective and gradient are wanted: near each grain's motion, as a
    minimiser of the caller's own steps."""
    off = np.random.default_rng(seed + 17).uniform(-0.4, 0.4, s["truth"].shape) * np.array([1.0, 1.0, 0.01])
    return s["truth"] - s["rec"][:, 4:7] + off


def _records(t):
    """The grains' records column by column, as a program reads them back."""
    g = t.get_grains_structs()
    names = ("refx", "refy", "refrot", "dx", "dy", "drot", "upix", "vpix", "rot_inc", "NCC", "NCC_rescue", "NCC_subpix",
             "status")
    return {k: g[k] for k in names}


def _load(t, c, slot, frame):
    if c.get("raw"):
        h, w = frame.shape
        t.load_frame_raw_device(slot, frame.data_ptr(), w, h, RAW_LEFT, RAW_TOP, c["raw"], True)
    else:
        t.load_frame(slot, frame)
    if c.get("remap"):
        t.remap(slot)


def run(state):
    c = state["case"]
    if c["kind"] == "disto":
        x, ini, end, _ = state["fit"].fit(state["start"], state["step"])
        return dict(params=x, index_ini=ini, index_end=end)
    t = state["t"]
    if c["kind"] == "grad":
        f = t.objective(state["X"])
        f2, g = t.grad(state["X"])
        return dict(objective=f, value=f2, gradient=g)
    if c["kind"] == "sequence":
        t.set_grains(state["rec"])
        t.set_iref(0)
        _load(t, c, 0, state["frames"][0])
        out = []
        for k in range(1, len(state["frames"])):
            _load(t, c, 1, state["frames"][k])
            t.track_frame(k)
            out.append(_records(t))
        return out
    if c["host"]:
        t.load_frame(0, state["ref"])
        t.load_frame(1, state["cur"])
    t.restore_grains()
    t.track_frame(1)
    return _records(t)


# ---- what a pass cannot do without ------------------------------------------

def _mean_points(c):
    """Expected points of a grain's pattern."""
    if c["pattern"] == "circ":
        return math.pi * c["pa"] ** 2
    if c["pattern"] == "ring":
        return math.pi * (c["pb"] ** 2 - c["pa"] ** 2)
    if c["pattern"] == "rect":
        return (2.0 * c["pa"] + 1.0) * (2.0 * c["pb"] + 1.0)
    sq = lambda a, b: (a * a + a * b + b * b) / 3.0  # noqa: E731  mean of r^2, r uniform in a..b
    return math.pi * ((1.0 - c["big"]) * sq(c["r0"], c["r1"]) + c["big"] * sq(c["R0"], c["R1"]))


SAMPLE_FLOPS = 5 * 21 + 8  # one bicubic sample: five cubics, and its position
EVALS = {"plain": 100, "fast": 5}  # objective evaluations a refinement takes, about


def work(case):
    """Frames read once and records read and written once; six operations per
    pattern pixel and candidate of the search (three multiply-adds), and the
    bicubic samples of the refinement."""
    c = case
    if c["kind"] == "disto":
        pairs = 0.5 * c["n"] ** 2 * min(1.0, math.pi * c["dist"] ** 2 / (c["dimx"] * c["dimy"]))
        points = c["n"] * (c["images"] + 1)
        evals = 1000.0  # objective evaluations of the minimisation, about
        return {"bytes": 8.0 * pairs + 24.0 * points, "flops": evals * (25.0 * pairs * c["images"] + 60.0 * points)}
    points, frame = _mean_points(c), float(c["dimx"] * c["dimy"])
    if c["kind"] == "grad":
        return {"bytes": c["n"] * (10.0 * points + 80.0), "flops": c["n"] * points * (3.0 * SAMPLE_FLOPS + 40.0)}
    nrot = 2 * c["num_rot"] + 1
    search = 6.0 * points * nrot * (2 * c["zone"] + 1) ** 2
    if c.get("rescue"):
        search += c["jump"] / c["frames"] * 6.0 * points * nrot * (2 * c["rescue"] + 1) ** 2
    refine = EVALS[c["form"]] * points * (SAMPLE_FLOPS + 9.0)
    frames = c.get("frames", 1)
    pixels = frame * (frames + 1) * (c["bits"] // 8) * (2.0 if c["kind"] == "sequence" else 1.0)
    flops = frames * c["n"] * (search + refine)
    if c.get("remap"):
        flops += (frames + 1) * frame * SAMPLE_FLOPS
        pixels += (frames + 1) * frame * 16.0
    return {"bytes": pixels + frames * c["n"] * (4.0 * points + 208.0), "flops": flops}


# ---- the same values in 64 bits, from numpy and torch alone ------------------

def _pattern(c, r):
    k = c["pattern"]
    if k == "rect":
        h, w = int(c["pb"]), int(c["pa"])
        y, x = np.mgrid[-h:h + 1, -w:w + 1]
        return x.ravel().astype(np.float64), y.ravel().astype(np.float64)
    lo, R = (c["pa"], int(c["pb"])) if k == "ring" else (0.0, int(c["pa"]) if k == "circ" else max(int(r * c["pa"]), int(c["pb"])))
    y, x = np.mgrid[-R:R + 1, -R:R + 1]
    d = np.sqrt(x * x + y * y)
    keep = (d <= R) & (d >= lo)
    return x[keep].astype(np.float64), y[keep].astype(np.float64)


def _steps(num, inc):
    """Angles that the double loop from -|inc num| in steps of inc visits."""
    out, d, top = [], -abs(inc * num), abs(inc * num)
    while d <= top:
        out.append(d)
        d += inc
    return np.array(out)


def _best_ncc(c, s):
    """The best NCC of every grain over the level-0 zone and rotation steps."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    ref, cur = (torch.from_numpy(s[k].astype(np.float64)).to(dev) for k in ("ref", "cur"))
    z, steps, flat, width = c["zone"], _steps(c["num_rot"], STEPS_INC), cur.reshape(-1), cur.shape[1]
    span = torch.arange(-z, z + 1, device=dev)
    cand = (span[None, :] * width + span[:, None]).reshape(1, -1, 1)
    best = torch.zeros(len(s["rec"]), dtype=torch.float64, device=dev)
    away = lambda v: np.sign(v) * np.floor(np.abs(v) + 0.5)  # noqa: E731  round half away from zero
    for i, rec in enumerate(s["rec"]):
        x, y = _pattern(c, rec[3])
        X0, Y0 = int(rec[0]), int(rec[1])
        a = ref[Y0 + torch.from_numpy(y.astype(np.int64)).to(dev), X0 + torch.from_numpy(x.astype(np.int64)).to(dev)]
        a = a - a.mean()
        co, si = np.cos(steps)[:, None], np.sin(steps)[:, None]
        rx, ry = away(co * x + si * y), away(-si * x + co * y)
        at = (Y0 + int(away(rec[5])) + ry) * width + X0 + int(away(rec[4])) + rx
        at = torch.from_numpy(at.astype(np.int64)).to(dev)[:, None, :]
        for k in range(0, len(steps), 4):
            w = flat[at[k:k + 4] + cand]
            w = w - w.mean(-1, keepdim=True)
            ncc = (w @ a) / torch.sqrt((a @ a) * (w * w).sum(-1))
            best[i] = torch.maximum(best[i], torch.nan_to_num(ncc, nan=0.0).max())
    return best.cpu().numpy()


def _cubic(p, x):
    """Catmull-Rom through p[1] (x = 0) and p[2] (x = 1), and its derivative."""
    c, d1 = 0.5 * (p[2] - p[0]), 0.5 * (p[3] - p[1])
    b, a = -3.0 * p[1] + 3.0 * p[2] - 2.0 * c - d1, 2.0 * p[1] - 2.0 * p[2] + c + d1
    return ((a * x + b) * x + c) * x + p[1], (3.0 * a * x + 2.0 * b) * x + c


def _objective(c, s, X):
    """1 - NCC through bicubic interpolation, and its gradient, per grain."""
    cur = s["cur"].astype(np.float64)
    f, g = np.zeros(len(X)), np.zeros((len(X), 3))
    for i, rec in enumerate(s["rec"]):
        x, y = _pattern(c, rec[3])
        a = s["ref"][int(rec[1]) + y.astype(int), int(rec[0]) + x.astype(int)].astype(np.float64)
        a = a - a.mean()
        co, si = math.cos(rec[6] + X[i, 2]), math.sin(rec[6] + X[i, 2])
        xs = rec[0] + rec[4] + X[i, 0] + co * x + si * y
        ys = rec[1] + rec[5] + X[i, 1] - si * x + co * y
        ix, iy = np.floor(xs).astype(int), np.floor(ys).astype(int)
        cols = [_cubic([cur[iy - 1 + k, ix - 1 + j] for k in range(4)], ys - iy) for j in range(4)]
        v, vx = _cubic([q[0] for q in cols], xs - ix)
        vy, _ = _cubic([q[1] for q in cols], xs - ix)
        b = v - v.mean()
        den, ratio = math.sqrt((a @ a) * (b @ b)), (a @ b) / (b @ b)
        dn = (a - ratio * b) / den
        f[i] = 1.0 - (a @ b) / den
        g[i] = -(dn @ vx), -(dn @ vy), -(dn @ (vx * (-si * x + co * y) + vy * (-co * x - si * y)))
    return f, g


def exact(case, seed):
    """Pairs: the pixel stage's best NCC (the refined positions are where an
    iterative minimiser stops: no value of their own).  Objective and
    gradient; the distortion criterion at the start of the fit, where the lens
    is the identity.  Sequences: none (each frame starts from the last one's
    refined state)."""
    c = case
    if c["kind"] == "disto":
        d = _disto_case(c, seed)
        rx, ry = d["refx"].astype(np.float64), d["refy"].astype(np.float64)
        pr = _disto_pairs_exact(rx, ry, c["dist"])
        abx, aby = rx[pr[1]] - rx[pr[0]], ry[pr[1]] - ry[pr[0]]
        ab = np.sqrt(abx * abx + aby * aby)
        ddx, ddy = d["dx"][:, pr[1]] - d["dx"][:, pr[0]], d["dy"][:, pr[1]] - d["dy"][:, pr[0]]
        e = abx / ab * ddx + aby / ab * ddy
        ok = (d["ncc"][:, pr[0]] >= 0.7) & (d["ncc"][:, pr[1]] >= 0.7)
        return dict(params=None, index_ini=float((e[ok] ** 2).sum() / c["images"]), index_end=None)
    if c["kind"] == "sequence" or c["interp"] != "cubic":
        return None
    s = wl.make_pair(_preset(c), seed=seed)
    if c["kind"] == "grad":
        f, g = _objective(c, s, _positions(s, seed))
        return dict(objective=f, value=f, gradient=g)
    none = dict.fromkeys(("refx", "refy", "refrot", "dx", "dy", "drot", "upix", "vpix", "rot_inc", "NCC_rescue",
                          "NCC_subpix", "status"))
    return dict(none, NCC=_best_ncc(c, s))


def _disto_pairs_exact(rx, ry, dist):
    i, j = np.triu_indices(len(rx), 1)
    near = np.hypot(rx[i] - rx[j], ry[i] - ry[j]) <= dist
    return i[near], j[near]
