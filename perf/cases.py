"""The work that programs have this library do, as cases that can be timed.

A case is a dict of plain values.  `listed()` gives the named ones, `draw()`
more of the same ranges, `prepare()` what a program holds before the call,
`run()` one pass through the public entry points, `work()` the bytes and
operations a pass cannot do without, and `exact()` the same results computed
in 64 bits with torch alone.

Kinds of case:
  locate  gpu_tracking.batch_device on a movie that is on the device
  host    gpu_tracking.batch_rust on a movie in host memory
  many    batched.batch_many on a list of uneven movies
  link    gpu_tracking.link_rust on a table of positions
  refine  adjoint.refine and its backward pass at given peaks
  tracks  trajectories.filter_stubs, steps and imsd on a linked table

Movies: Poisson background 100 and Gaussian read noise 5, Gaussian spots of
amplitude 150 to 1500 that diffuse and blink (2 %), the spot model of
tracking_optimizations_b200/synth.py, drawn on the device from the seed.
"""
import math

import numpy as np
import torch
from torch.nn import functional as F

BACKGROUND, READ_NOISE, BLINK = 100.0, 5.0, 0.02
AMP_LO, AMP_HI = 150.0, 1500.0


def _locate(name, T, H, W, spots, d, dtype="u16", sep=0, sr=0.0, memory=0, sigma=1.2, step=1.5, minmass=0.0, cpu=False,
            char=False, sig=0.0, bg=0.0, kind="locate"):
    return dict(name=name, kind=kind, T=T, H=H, W=W, spots=spots, diameter=d, dtype=dtype, separation=sep or d + 1,
                search_range=sr, memory=memory, sigma=sigma, step=step, minmass=minmass, cpu_processed=cpu,
                characterize=char, sig_radius=sig, bg_radius=bg)


def listed():
    return [
        # a frame as a camera delivers it, located at once: the latency of a call
        _locate("frame", 1, 256, 256, 50, 9, sigma=1.5, minmass=500.0),
        # a short movie with linking, the smallest configuration of synth.py
        _locate("short movie", 10, 256, 256, 50, 9, sr=5.0, sigma=1.5, step=1.0, minmass=500.0),
        # the movie of the benchmark: 1000 frames, linked with memory
        _locate("movie", 1000, 512, 512, 500, 7, sr=5.0, memory=2, minmass=300.0, cpu=True),
        # float frames (the only type that the pyo3 module takes) of the size of the lab's recording
        _locate("float movie", 200, 524, 800, 420, 9, dtype="f32", sr=5.0, memory=1, minmass=500.0, cpu=True),
        # a large sensor, few frames, no linking, with the shader's own characterisation
        _locate("large frames", 12, 2048, 2560, 8000, 11, minmass=700.0, char=True),
        # larger features on a cropped sensor (odd sides), raw signal and background columns
        _locate("wide features", 100, 389, 517, 90, 15, sep=12, sr=6.0, memory=1, sigma=2.5, minmass=2000.0, sig=6.0,
                bg=9.0),
        # dense linking: 20000 spots a frame, search range 7, memory 3
        _locate("dense movie", 200, 2048, 2048, 20000, 9, sr=7.0, memory=3, sigma=1.5, step=2.5),
        # the call of the Python module on a numpy array
        _locate("host movie", 200, 512, 512, 500, 7, sr=5.0, memory=2, minmass=300.0, cpu=True, kind="host"),
        # a screening plate: movies of several sizes and diameters in one call
        dict(name="uneven movies", kind="many", movies=12, frames=120, side=1024, spread=3),
        # linking of positions that were located elsewhere
        dict(name="table to link", kind="link", T=500, per_frame=800, side=700, search_range=5.0, memory=2),
        # one step of a fit through the refinement: positions, loss, gradients
        dict(name="refine step", kind="refine", T=256, H=512, W=512, spots=400, diameter=7, sigma=1.2),
        # what the lab pipeline does with linked rows: stubs, steps, mean squared displacements
        dict(name="tracks", kind="tracks", particles=2500, frames=600, mean_length=150, threshold=20, max_lagtime=300),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["locate", "locate", "locate", "host", "many", "link", "refine", "tracks"])
    if kind == "many":
        return dict(kind=kind, movies=rng.randint(2, 16), frames=_logint(rng, 10, 160), side=rng.choice([256, 512, 1024]),
                    spread=rng.randint(1, 1000))
    if kind == "link":
        per_frame = _logint(rng, 20, 3000)
        side = int(math.sqrt(per_frame / rng.uniform(0.0005, 0.0025))) + 8
        return dict(kind=kind, T=_logint(rng, 5, 500), per_frame=per_frame, side=side,
                    search_range=round(rng.uniform(3.0, 6.0), 2), memory=rng.randint(0, 3))
    if kind == "refine":
        H, W = _logint(rng, 64, 800), _logint(rng, 64, 800)
        return dict(kind=kind, T=_logint(rng, 2, 256), H=H, W=W,
                    spots=max(2, int(H * W * rng.uniform(0.0005, 0.002))), diameter=rng.choice([5, 7, 9, 11]),
                    sigma=round(rng.uniform(1.0, 2.0), 2))
    if kind == "tracks":
        length = _logint(rng, 10, 300)
        return dict(kind=kind, particles=_logint(rng, 50, 2500), frames=2 * length + rng.randint(1, 200),
                    mean_length=length, threshold=rng.randint(2, length), max_lagtime=_logint(rng, 10, 300))
    pixels = _logint(rng, 1 << 14, 1 << 22)
    H = max(48, int(math.sqrt(pixels) * math.exp(rng.uniform(-0.35, 0.35))))
    W = max(48, pixels // H)
    if rng.random() < 0.6:  # sensors and crops whose sides are multiples of 16
        H, W = max(48, H // 16 * 16), max(48, W // 16 * 16)
    T = max(1, min(_logint(rng, 1, 1000), (1 << 27) // (H * W)))
    d = rng.choice([5, 7, 7, 9, 9, 11, 11, 13, 15])
    c = _locate("", T, H, W, max(4, int(H * W * rng.uniform(0.0005, 0.003))), d,
                dtype="u16" if kind == "host" else rng.choice(["u16", "u16", "f32"]),
                sep=rng.choice([d + 1, d + 1, d]), sr=round(rng.uniform(3.0, 6.0), 2) if rng.random() < 0.75 else 0.0,
                memory=rng.randint(0, 3), sigma=round(rng.uniform(0.9, 0.2 * d), 2), minmass=6.0 * d * d,
                cpu=rng.random() < 0.5, char=rng.random() < 0.2, sig=round(d / 2.0, 1) if rng.random() < 0.2 else 0.0,
                kind=kind)
    c["bg_radius"] = c["sig_radius"] + 3.0 if c["sig_radius"] and rng.random() < 0.5 else 0.0
    del c["name"]
    return c


def _params(c):
    p = dict(diameter=c["diameter"], separation=c["separation"])
    if c["minmass"]:
        p["minmass"] = c["minmass"]
    if c["search_range"]:
        p.update(search_range=c["search_range"], memory=c["memory"])
    if c["cpu_processed"]:
        p["cpu_processed"] = True
    if c["characterize"]:
        p["characterize"] = True
    if c["sig_radius"]:
        p["sig_radius"] = c["sig_radius"]
    if c["bg_radius"]:
        p["bg_radius"] = c["bg_radius"]
    return p


def _columns(p):
    names = ["frame", "mass", "y", "x"]
    names += ["particle"] if "search_range" in p else []
    names += ["Rg", "ecc", "signal"] if p.get("cpu_processed") else []
    names += ["raw_mass"] if p.get("sig_radius") else []
    names += ["raw_bg_median", "raw_mass_corrected"] if p.get("bg_radius") else []
    names += ["Rg_gpu", "raw_mass_gpu", "signal_gpu", "ecc_gpu"] if p.get("characterize") else []
    return names


# ---- inputs ----

def _row_capacity(c):
    """Rows that a program sets aside for a movie's table."""
    return int(1.2 * c["T"] * c["spots"]) + 256


def _generator(seed, device="cuda"):
    g = torch.Generator(device=device)
    g.manual_seed(int(seed))
    return g


def _fold(x, lim):
    """Positions reflected at 0 and lim."""
    x = x.remainder(2 * lim)
    return torch.where(x > lim, 2 * lim - x, x)


def _positions(g, T, N, H, W, step):
    """(T, N, 2) float64 positions of N spots that diffuse."""
    start = torch.rand((1, N, 2), generator=g, device="cuda", dtype=torch.float64)
    start = start * torch.tensor([H - 1.0, W - 1.0], device="cuda", dtype=torch.float64)
    walk = torch.randn((T, N, 2), generator=g, device="cuda", dtype=torch.float64) * step
    walk[0] = 0
    pos = start + walk.cumsum(0)
    return torch.stack([_fold(pos[..., 0], H - 1.0), _fold(pos[..., 1], W - 1.0)], dim=-1)


def _movie(g, T, H, W, spots, sigma, step, dtype):
    """A (T, H, W) movie on the device and the spots' positions.  The spots
    are added in whole 1/64 counts, so that the sum's order cannot matter."""
    pos = _positions(g, T, spots, H, W, step)
    amp = AMP_LO + (AMP_HI - AMP_LO) * torch.rand((1, spots), generator=g, device="cuda")
    amp = amp * (torch.rand((T, spots), generator=g, device="cuda") >= BLINK)
    R = int(math.ceil(4 * sigma))
    off = torch.arange(-R, R + 1, device="cuda")
    dy, dx = off.repeat_interleave(2 * R + 1), off.repeat(2 * R + 1)
    out = torch.empty((T, H, W), dtype=torch.float32 if dtype == "f32" else torch.int16, device="cuda")
    chunk = max(1, min(T, (1 << 26) // (H * W), (1 << 25) // (spots * len(dy)) + 1))
    background = torch.full((1,), BACKGROUND, device="cuda")
    for t0 in range(0, T, chunk):
        p, a = pos[t0:t0 + chunk], amp[t0:t0 + chunk]
        n = p.shape[0]
        img = torch.zeros(n * H * W, dtype=torch.int32, device="cuda")
        c = p.round().long()
        rows, cols = c[..., 0, None] + dy, c[..., 1, None] + dx
        r2 = (rows - p[..., 0, None]).float() ** 2 + (cols - p[..., 1, None]).float() ** 2
        val = (64.0 * a[..., None] * torch.exp(-r2 / (2.0 * sigma * sigma))).round().to(torch.int32)
        ok = (rows >= 0) & (rows < H) & (cols >= 0) & (cols < W)
        idx = (torch.arange(n, device="cuda")[:, None, None] * H + rows) * W + cols
        img.index_add_(0, idx[ok], val[ok])
        noise = torch.poisson(background.expand(n * H * W), generator=g)
        noise += READ_NOISE * torch.randn(n * H * W, generator=g, device="cuda")
        frame = (img.float() / 64.0 + noise).clamp_(0, 30000)
        out[t0:t0 + n] = (frame if dtype == "f32" else frame.round()).view(n, H, W).to(out.dtype)
    return (out if dtype == "f32" else out.view(torch.uint16)), pos


def _many_specs(c):
    """Uneven movies: sides from side / 8 to side, aspect 1 or 2, diameters 5 to 11."""
    r = np.random.Generator(np.random.PCG64(c["spread"]))
    specs = []
    for _ in range(c["movies"]):
        H = max(64, c["side"] >> int(r.integers(0, 4)))
        W = min(c["side"], H * int(r.integers(1, 3)))
        T = max(2, int(c["frames"] * r.uniform(0.25, 1.0)))
        d = int(r.choice([5, 7, 9, 11]))
        specs.append(_locate("", T, H, W, max(4, int(H * W * r.uniform(0.0005, 0.003))), d,
                             sr=round(float(r.uniform(3.0, 8.0)), 2), memory=int(r.integers(0, 4)), minmass=6.0 * d * d))
    return specs


def _link_table(c, seed):
    g = _generator(seed)
    pos = _positions(g, c["T"], c["per_frame"], c["side"], c["side"], 1.5)
    mass = 100.0 + 1000.0 * torch.rand((c["T"], c["per_frame"], 1), generator=g, device="cuda", dtype=torch.float64)
    frame = torch.arange(c["T"], device="cuda", dtype=torch.float64)[:, None, None].expand(-1, c["per_frame"], 1)
    # one in twenty is missed, as many in every frame
    missed = torch.rand((c["T"], c["per_frame"]), generator=g, device="cuda").argsort(dim=1) < c["per_frame"] // 20
    return torch.cat([frame, mass, pos], dim=-1)[~missed].float().cpu().numpy()


def _tracks_table(c, seed):
    """Rows (particle, frame, x, y) in frame order: trajectories of
    exponential length, one frame in fifty missing.  Lengths, starts and gaps
    come from the sizes alone, the particles' numbers and paths from the
    seed, so that the results of every seed have as many rows."""
    n = c["particles"]
    r = np.random.Generator(np.random.PCG64(n))
    length = np.minimum(1 + r.exponential(c["mean_length"], n).astype(np.int64), c["frames"])
    start = (r.random(n) * (c["frames"] - length + 1)).astype(np.int64)
    first = np.cumsum(length) - length
    pid = np.repeat(np.arange(n), length)
    frame = np.arange(len(pid)) - np.repeat(first, length) + np.repeat(start, length)
    keep = r.random(len(pid)) >= 0.02
    keep[first] = keep[first + length - 1] = True
    r = np.random.Generator(np.random.PCG64(seed))
    paths = np.cumsum(r.normal(0.0, 1.0, (len(pid), 2)), axis=0)
    xy = (r.random((n, 2)) * 500.0 - paths[first])[pid] + paths
    xy = xy.astype(np.float32)
    pid = r.permutation(n)[pid]
    order = np.lexsort((pid, frame))
    order = order[keep[order]]
    return pid[order].astype(np.int64), frame[order].astype(np.int64), xy[order, 0].copy(), xy[order, 1].copy()


def _refine_inputs(c, seed):
    """Float frames, the walk records of the spots at their nearest pixels, and the true positions."""
    g = _generator(seed)
    movie, pos = _movie(g, c["T"], c["H"], c["W"], c["spots"], c["sigma"], 1.5, "f32")
    c0 = pos.round()
    t = torch.arange(c["T"], device="cuda", dtype=torch.float64)[:, None].expand(-1, c["spots"])
    walk = torch.stack([t, c0[..., 0], c0[..., 1], c0[..., 0], c0[..., 1]], dim=-1).reshape(-1, 5)
    return movie, walk.to(torch.int32).contiguous(), pos.reshape(-1, 2)


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind in ("locate", "host"):
        movie, _ = _movie(_generator(seed), c["T"], c["H"], c["W"], c["spots"], c["sigma"], c["step"], c["dtype"])
        rows = torch.zeros((_row_capacity(c), len(_columns(_params(c)))), dtype=torch.float32, device="cuda")
        if kind == "host":
            movie, rows = np.ascontiguousarray(movie.cpu().numpy()), rows.cpu().numpy()
        return dict(kind=kind, params=_params(c), frames=movie, rows=rows)
    if kind == "many":
        g = _generator(seed)
        movies = [(_movie(g, s["T"], s["H"], s["W"], s["spots"], s["sigma"], s["step"], s["dtype"])[0], _params(s))
                  for s in _many_specs(c)]
        from tracking_optimizations_b200 import batched

        return dict(kind=kind, movies=movies, outs=[b.zero_() for b in batched.output_buffers(movies)])
    if kind == "link":
        return dict(kind=kind, table=_link_table(c, seed), search_range=c["search_range"], memory=c["memory"])
    if kind == "refine":
        movie, walk, pos = _refine_inputs(c, seed)
        return dict(kind=kind, frames=movie.requires_grad_(True), walk=walk, target=pos.float(), diameter=c["diameter"],
                    noise_size=torch.tensor(1.1, dtype=torch.float64, device="cuda", requires_grad=True))
    pid, frame, x, y = _tracks_table(c, seed)
    return dict(kind=kind, pid=pid, frame=frame, x=x, y=y, threshold=c["threshold"], max_lagtime=c["max_lagtime"])


def run(state):
    kind = state["kind"]
    if kind in ("locate", "host"):
        from tracking_optimizations_b200 import gpu_tracking

        if kind == "locate":
            table = gpu_tracking.batch_device(state["frames"], **state["params"])
        else:
            table, _ = gpu_tracking.batch_rust(state["frames"], **state["params"])
        # the program keeps the movie's rows in its own array
        rows = state["rows"]
        rows[:len(table)] = table
        return dict(count=len(table), **{n: rows[:, i] for i, n in enumerate(_columns(state["params"]))})
    if kind == "many":
        from tracking_optimizations_b200 import batched

        tables = batched.batch_many(state["movies"], outs=state["outs"])
        return [[b[:, :4], b[:, 4], len(t)] for b, (t, _) in zip(state["outs"], tables)]
    if kind == "link":
        from tracking_optimizations_b200 import gpu_tracking

        return gpu_tracking.link_rust(state["table"], state["search_range"], state["memory"])
    if kind == "refine":
        from tracking_optimizations_b200 import adjoint

        yxm = adjoint.refine(state["frames"], state["walk"], state["diameter"], noise_size=state["noise_size"])
        loss = ((yxm[:, :2] - state["target"]) ** 2).sum(dim=1).mean()
        grads = torch.autograd.grad(loss, [state["frames"], state["noise_size"]])
        return dict(yxm=yxm.detach(), grad_frames=grads[0], grad_noise_size=grads[1])
    from tracking_optimizations_b200 import trajectories

    pid = state["pid"]
    keep = trajectories.filter_stubs(pid, state["threshold"])
    pid, frame, x, y = pid[keep], state["frame"][keep], state["x"][keep], state["y"][keep]
    xs, ys, x_step, y_step, length, order = trajectories.steps(pid, x, y, 0.1)
    lag, particle, msd = trajectories.imsd(pid, frame, x, y, 0.1, 10.0, max_lagtime=state["max_lagtime"])
    return dict(keep=keep, xs=xs, ys=ys, x_step=x_step, y_step=y_step, length=length, order=order, lag=lag,
                particle=particle, msd=msd)


def work(case):
    c, kind = case, case["kind"]
    if kind in ("locate", "host"):
        return _movie_work(c)
    if kind == "many":
        each = [_movie_work(s) for s in _many_specs(c)]
        return {"bytes": sum(w["bytes"] for w in each), "flops": sum(w["flops"] for w in each)}
    if kind == "link":
        n = c["T"] * c["per_frame"]
        return {"bytes": n * (16 + 8), "flops": n * 9 * 5}
    if kind == "refine":
        n, k = c["T"] * c["spots"], 2 * (c["diameter"] // 2) + 1
        px = c["T"] * c["H"] * c["W"]
        # frames read, gradient written; peaks and their results.  A peak's
        # bandpass is evaluated twice, its gradient passes back once
        return {"bytes": 8 * px + n * (20 + 12 + 8), "flops": n * 3 * 4 * (2 * k) * k * k}
    rows = c["particles"] * c["mean_length"]
    lags = min(c["max_lagtime"], c["mean_length"])
    return {"bytes": rows * (8 + 1 + 8 + 8 + 4 + 4 + 8 + 24 + 8) + c["particles"] * lags * 20,
            "flops": 8.0 * c["particles"] * lags * c["mean_length"]}


def _movie_work(c):
    px, k = c["T"] * c["H"] * c["W"], 2 * (c["diameter"] // 2) + 1
    # frames read, table written (of a spot in ten the row is lost to a
    # neighbour); two separable passes of the Gaussian (multiply and add) and
    # the box (running sums), the local maximum in both directions
    return {"bytes": px * (2 if c["dtype"] == "u16" else 4) + 0.9 * c["T"] * c["spots"] * 4 * len(_columns(_params(c))),
            "flops": px * (2 * (2 * k + 2) + 8)}


# ---- the same results in 64 bits ----

def _circle(radius):
    b = int(math.ceil(radius))
    return [(i, j) for i in range(-b, b + 1) for j in range(-b, b + 1) if i * i + j * j <= radius * radius]


def _taps(k, s):
    i = torch.arange(-(k // 2), k // 2 + 1, device="cuda", dtype=torch.float64)
    w = torch.exp(-i * i / (2.0 * s))
    return w / w.sum()


def _symmetric(n, r):
    """Indices of a line of n pixels with r mirrored ones at both ends."""
    i = torch.arange(-r, n + r, device="cuda")
    i = torch.where(i < 0, -i - 1, i)
    return torch.where(i >= n, 2 * n - i - 1, i)


def _bandpass(x, k, s):
    """Gaussian of variance s (zero outside) minus the box mean of side k (mirrored outside)."""
    r = k // 2
    H, W = x.shape[1:]
    a = _taps(k, s)
    z = F.pad(x, (r, r, r, r))
    z = sum(a[j] * z[:, :, j:j + W] for j in range(2 * r + 1))
    z = sum(a[j] * z[:, j:j + H] for j in range(2 * r + 1))
    m = x[:, _symmetric(H, r)][:, :, _symmetric(W, r)]
    m = sum(m[:, :, j:j + W] for j in range(2 * r + 1))
    m = sum(m[:, j:j + H] for j in range(2 * r + 1))
    return z - m / float(k * k)


def _at(plane, t, u, v, offsets):
    """plane[t, u + i, v + j] for the offsets (i, j), 0 outside."""
    H, W = plane.shape[1:]
    o = torch.tensor(offsets, device="cuda")
    uu, vv = u[:, None] + o[:, 0], v[:, None] + o[:, 1]
    ok = (uu >= 0) & (uu < H) & (vv >= 0) & (vv < W)
    return torch.where(ok, plane[t[:, None], uu.clamp(0, H - 1), vv.clamp(0, W - 1)], 0.0), ok


def _centroid(plane, t, u, v, rc, border):
    H, W = plane.shape[1:]
    offs = _circle(rc)
    o = torch.tensor(offs, device="cuda", dtype=torch.float64)
    p, _ = _at(plane, t, u, v, offs)
    inside = (u - border >= 0) & (u + border < H) & (v - border >= 0) & (v + border < W)
    m = torch.where(inside, p.sum(1), 0.0)
    safe = torch.where(m != 0, m, 1.0)
    return torch.where(inside, (p * o[:, 0]).sum(1) / safe, 0.0), torch.where(inside, (p * o[:, 1]).sum(1) / safe, 0.0), m


def _exact_frames(x, c, t0):
    """The rows of the frames x (float64), without the particle column."""
    n, H, W = x.shape
    d, sep = c["diameter"], float(c["separation"])
    P = _bandpass(x, d, 1.0).clamp_min(0.0)
    D = int(2.0 * sep / math.sqrt(2.0))
    o = int(D / 2.0 - 0.5)
    top = F.pad(P, (o, D - 1 - o, o, D - 1 - o), value=-math.inf)
    top = F.max_pool2d(F.max_pool2d(top[:, None], (1, D), 1), (D, 1), 1)[:, 0]
    t, u0, v0 = torch.nonzero((P >= top) & (P > 0), as_tuple=True)
    u, v = u0.clone(), v0.clone()
    w0, w1, m = (torch.zeros(len(t), device="cuda", dtype=torch.float64) for _ in range(3))
    active = torch.arange(len(t), device="cuda")
    for _ in range(10):
        a, b, mm = _centroid(P, t[active], u[active], v[active], (d - 1) // 2, d // 2)
        w0[active], w1[active], m[active] = a, b, mm
        du = ((a > 0.6) & (u[active] < H - 1)).long() - ((a < -0.6) & (u[active] > 0)).long()
        dv = ((b > 0.6) & (v[active] < W - 1)).long() - ((b < -0.6) & (v[active] > 0)).long()
        u[active] += du
        v[active] += dv
        active = active[(du != 0) | (dv != 0)]
    ok = (m > c["minmass"]) & (m != 0)
    t, u0, v0, y, x_, m = t[ok], u0[ok], v0[ok], (u + w0)[ok], (v + w1)[ok], m[ok]
    keep = torch.ones(len(t), dtype=torch.bool, device="cuda")
    ends = torch.searchsorted(t, torch.arange(n + 1, device="cuda")).tolist()
    for a, b in zip(ends[:-1], ends[1:]):
        near = (y[a:b, None] - y[None, a:b]) ** 2 + (x_[a:b, None] - x_[None, a:b]) ** 2 < sep * sep
        i = torch.arange(b - a, device="cuda")
        worse = (m[a:b, None] < m[None, a:b]) | ((m[a:b, None] == m[None, a:b]) & (i[:, None] > i[None]))
        keep[a:b] = ~(near & worse).any(1)
    t, u0, v0, y, x_, m = t[keep], u0[keep], v0[keep], y[keep], x_[keep], m[keep]
    out = dict(frame=(t + t0).double(), mass=m, y=y, x=x_)
    circle = _circle(d // 2)
    o = torch.tensor(circle, device="cuda", dtype=torch.float64)
    r2, th = (o * o).sum(1), torch.atan2(o[:, 1], o[:, 0])
    p, _ = _at(P, t, u0, v0, circle)
    mid, sn, cs = P[t, u0, v0], (p * torch.sin(2 * th)).sum(1), (p * torch.cos(2 * th)).sum(1)
    if c["cpu_processed"]:
        out.update(Rg=((p * r2).sum(1) / m).sqrt(), ecc=(sn * sn + cs * cs).sqrt() / (m - mid), signal=p.max(1).values)
    if c["sig_radius"]:
        # half away from zero, as the table's rounding
        mr, mc = (y + 0.5).floor().long(), (x_ + 0.5).floor().long()
        raw, _ = _at(x, t, mr, mc, _circle(c["sig_radius"]))
        out["raw_mass"] = raw.sum(1)
        if c["bg_radius"]:
            ring = [q for q in _circle(c["bg_radius"]) if q[0] ** 2 + q[1] ** 2 >= c["sig_radius"] ** 2]
            raw, ok = _at(x, t, mr, mc, ring)
            s = torch.where(ok, raw, math.inf).sort(1).values
            nv = ok.sum(1)
            lo = s.gather(1, ((nv - 1) // 2).clamp_min(0)[:, None])[:, 0]
            hi = s.gather(1, (nv // 2).clamp_max(len(ring) - 1)[:, None])[:, 0]
            out["raw_bg_median"] = 0.5 * (lo + hi)
            out["raw_mass_corrected"] = out["raw_mass"] - out["raw_bg_median"] * len(_circle(c["sig_radius"]))
    if c["characterize"]:
        raw, _ = _at(x, t, u0, v0, circle)
        own = p.sum(1)
        out.update(Rg_gpu=((p * r2).sum(1) / own).sqrt(), raw_mass_gpu=raw.sum(1), signal_gpu=p.max(1).values,
                   ecc_gpu=(sn * sn + cs * cs).sqrt() / (own - mid))
    return out


def _exact_movie(movie, c, rows):
    chunk = max(1, (1 << 24) // (c["H"] * c["W"]))
    parts = []
    for t0 in range(0, c["T"], chunk):
        x = movie[t0:t0 + chunk]
        x = x.double() if x.dtype == torch.float32 else x.view(torch.int16).double()
        parts.append(_exact_frames(x, c, t0))
    got = {n: torch.cat([p[n] for p in parts]) for n in parts[0]}
    return {n: F.pad(got[n], (0, rows - len(got[n]))) if n in got else None for n in _columns(_params(c))}


def _exact_refine(c, seed):
    movie, walk, target = _refine_inputs(c, seed)
    k, H, W = c["diameter"], c["H"], c["W"]
    s = torch.tensor(1.1, dtype=torch.float64, device="cuda", requires_grad=True)
    n = len(walk)
    per = c["spots"]
    yxm, grad_frames, grad_s = [], torch.empty_like(movie, dtype=torch.float64), 0.0
    chunk = max(1, (1 << 23) // (H * W))
    for t0 in range(0, c["T"], chunk):
        x = movie[t0:t0 + chunk].detach().double().requires_grad_(True)
        w = walk[t0 * per:(t0 + chunk) * per].long()
        P = _bandpass(x, k, s).clamp_min(0.0)
        a, b, m = _centroid(P, w[:, 0] - t0, w[:, 1], w[:, 2], (k - 1) // 2, k // 2)
        y, xx = w[:, 3] + a, w[:, 4] + b
        tg = target[t0 * per:(t0 + chunk) * per].float().double()
        loss = ((y - tg[:, 0]) ** 2 + (xx - tg[:, 1]) ** 2).sum() / n
        gx, gs = torch.autograd.grad(loss, [x, s])
        grad_frames[t0:t0 + chunk] = gx
        grad_s = grad_s + gs
        yxm.append(torch.stack([y, xx, m], dim=1).detach())
    return dict(yxm=torch.cat(yxm), grad_frames=grad_frames, grad_noise_size=grad_s)


def _exact_tracks(c, seed):
    pid, frame, x, y = _tracks_table(c, seed)
    keep = np.bincount(pid, minlength=c["particles"])[pid] >= c["threshold"]
    pid, frame, x, y = pid[keep], frame[keep], x[keep].astype(np.float64) * 0.1, y[keep].astype(np.float64) * 0.1
    order = np.argsort(pid, kind="stable")
    p, f, gx, gy = pid[order], frame[order], x[order], y[order]
    first = np.r_[True, p[1:] != p[:-1]] if len(p) else np.zeros(0, bool)
    x_step = np.where(first, 0.0, gx - np.r_[0.0, gx[:-1]])
    y_step = np.where(first, 0.0, gy - np.r_[0.0, gy[:-1]])
    lags, parts, msds = [], [], []
    bounds = np.r_[np.flatnonzero(first), len(p)]
    for a, b in zip(bounds[:-1], bounds[1:]):
        span = int(f[b - 1] - f[a]) + 1
        ax = np.full((span, 2), np.nan)
        ax[f[a:b] - f[a]] = np.stack([gx[a:b], gy[a:b]], 1)
        for lag in range(1, min(c["max_lagtime"], span - 1) + 1):
            sq = (ax[lag:] - ax[:-lag]) ** 2
            sq = sq[~np.isnan(sq[:, 0])]
            if len(sq):
                lags.append(lag)
                parts.append(p[a])
                msds.append(sq.mean(0).sum())
    lags, parts, msds = np.array(lags), np.array(parts), np.array(msds)
    at = np.lexsort((parts, lags)) if len(lags) else np.zeros(0, np.int64)
    return dict(keep=None, xs=x, ys=y, x_step=x_step, y_step=y_step, length=np.sqrt(y_step ** 2 + x_step ** 2), order=None,
                lag=lags[at] / 10.0 if len(lags) else np.zeros(0), particle=None, msd=msds[at] if len(lags) else np.zeros(0))


def exact(case, seed):
    """What run() returns for prepare(case, seed), in 64 bits; None in the
    place of particle ids and counts, which are whole numbers.  None for
    movies of over a million rows, where some pair lies so near the
    separation that the last bit decides which rows there are."""
    c, kind = case, case["kind"]
    if kind in ("locate", "host") and c["T"] * c["spots"] > 1000000:
        return None
    if kind in ("locate", "host"):
        movie, _ = _movie(_generator(seed), c["T"], c["H"], c["W"], c["spots"], c["sigma"], c["step"], c["dtype"])
        return dict(count=None, **_exact_movie(movie, c, _row_capacity(c)))
    if kind == "many":
        g = _generator(seed)
        out = []
        for s in _many_specs(c):
            movie, _ = _movie(g, s["T"], s["H"], s["W"], s["spots"], s["sigma"], s["step"], s["dtype"])
            e = _exact_movie(movie, s, max(1024, s["T"] * max(64, s["H"] * s["W"] // 256)))
            out.append([torch.stack([e[n] for n in ("frame", "mass", "y", "x")], dim=1), None, None])
        return out
    if kind == "refine":
        return _exact_refine(c, seed)
    if kind == "tracks":
        return _exact_tracks(c, seed)
    return None
