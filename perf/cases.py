"""The calls that the performance figures stand for.

Every case is one call of a public entry point (`batch`, `LoG`, `batch_videos`,
`characterize_points`, `link`, `batch_learned`, `ProposalNet.train`) on a
synthetic recording: Gaussian spots (sigma about a sixth of the diameter,
log-normal peak signal-to-noise ratios) that diffuse, blink, vanish and
appear, on a flat or vignetted background with shot or read noise -- the
distributions of the benchmark's workloads.  Each spot keeps to a cell of its
own and stands clear of the noise, so a movie's table has the same number of
rows whatever the seed.  Inputs follow from the case and a seed alone, bit
for bit (spots are summed as integers, so the order of the sum does not
matter).

`listed` names the cases, `draw` gives others of the same ranges, `prepare`
makes what a program has in hand before the call, `run` makes the call and
returns its table as arrays, `work` counts the bytes and operations that the
call cannot do without, and `exact` gives the float columns in 64 bits, from
torch alone, where a table's rows follow from one frame at a time.
"""
import math

import numpy as np
import torch

import gpu_tracking_b200 as gt
from gpu_tracking_b200 import learned

DEV = "cuda:0"


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # choosing parameters on one frame: the call that is made most often, all latency
        _movie("look_512_u16", frames=1, height=512, width=512, spots=125, diameter=11),
        # the same on the full chip of a large sensor
        _movie("look_2048_u16", frames=1, height=2048, width=2048, spots=2000, diameter=11),
        # an 8-bit camera movie of an uneven size in a numpy array, linked without memory
        _movie("movie_601x803_u8_host", frames=240, height=601, width=803, spots=300, diameter=9, dtype="u8",
               bg=30.0, link=5.0, host=True),
        # float frames (already corrected by the caller's program), linked with memory
        _movie("movie_1024_f32", frames=160, height=1024, width=1024, spots=500, diameter=9, dtype="f32", bg=50.0,
               link=6.0, memory=2),
        # the benchmark's recording: large sensor, 16 bit, linked with memory 3
        _movie("movie_2048_u16", frames=512, height=2048, width=2048, spots=2000, diameter=11, link=7.0, memory=3),
        # uneven illumination: division by the smoothed mean, thresholds from the frames' noise
        _movie("vignette_1024_u16", frames=64, height=1024, width=1024, spots=500, diameter=11, link=7.0, memory=1,
               vignette=True, snr=0.3),
        # blobs of many sizes in float frames: the LoG scale space
        dict(name="log_1024_f32", kind="log", frames=64, height=1024, width=1024, spots=600, min_radius=2.0,
             max_radius=8.0, n_radii=10, link=6.0, memory=0),
        # a folder of recordings of uneven size and length in one call, for their trajectories alone
        dict(name="folder_10_videos", kind="videos", videos=10, side_lo=256, side_hi=2048, frames_lo=13,
             frames_hi=125, diameter=11, link=7.0, memory=3),
        # properties of given points (found by another program) in every frame of a movie
        dict(name="points_1024_u16", kind="points", frames=64, height=1024, width=1024, spots=500, diameter=11,
             dtype="u16", bg=100.0),
        # detections that exist already, linked on their own
        dict(name="link_400x2000", kind="link", frames=400, side=2048, spots=2000, link=7.0, memory=3),
        # walk seeds from the proposal network at twice the density
        dict(name="learned_2048_u16", kind="learned", frames=64, height=2048, width=2048, spots=4000, diameter=11,
             link=7.0, memory=3),
        # training that network: forward, backward, update
        dict(name="train_256x128", kind="train", frames=16, side=512, spots=125, batch=256, crop=128, steps=12),
    ]


def _movie(name, **kw):
    case = dict(name=name, kind="batch", dtype="u16", bg=100.0, link=0.0, memory=0, host=False, vignette=False,
                snr=0.0)
    case.update(kw)
    return case


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges above (batch calls as often as all others together)."""
    kind = rng.choice(["batch"] * 5 + ["log", "videos", "points", "link", "learned", "train"])
    density = math.exp(rng.uniform(math.log(2e-4), math.log(8e-4)))
    if kind == "batch":
        corrected = rng.random() < 0.15
        if corrected:  # the frames' noise level needs a power-of-two size
            h = w = rng.choice([512, 1024])
        else:
            h, w = _log_int(rng, 256, 2048), _log_int(rng, 256, 2048)
        frames = 1 if rng.random() < 0.3 else _log_int(rng, 8, min(512, (1 << 29) // (h * w)))
        dtype = "u16" if corrected else rng.choice(["u16", "u16", "u8", "f32"])
        return _drop_name(_movie("", frames=frames, height=h, width=w, spots=max(8, int(density * h * w)),
                                 diameter=rng.choice([9, 11, 13]), dtype=dtype,
                                 bg={"u16": 100.0, "u8": 30.0, "f32": 50.0}[dtype],
                                 link=rng.choice([5.0, 6.0, 7.0]) if frames > 1 else 0.0, memory=rng.randint(0, 3),
                                 host=rng.random() < 0.25, vignette=corrected, snr=0.3 if corrected else 0.0))
    if kind == "log":
        h, w = _log_int(rng, 300, 1400), _log_int(rng, 300, 1400)
        return dict(kind="log", frames=_log_int(rng, 4, 64), height=h, width=w,
                    spots=max(8, int(0.8 * density * h * w)), min_radius=2.0, max_radius=rng.choice([5.0, 6.5, 8.0]),
                    n_radii=rng.randint(4, 10), link=6.0, memory=rng.randint(0, 2))
    if kind == "videos":
        return dict(kind="videos", videos=rng.randint(3, 10), side_lo=256, side_hi=_log_int(rng, 700, 2048),
                    frames_lo=10, frames_hi=_log_int(rng, 20, 100), diameter=rng.choice([9, 11]), link=7.0,
                    memory=rng.randint(0, 3))
    if kind == "points":
        h, w = _log_int(rng, 256, 2048), _log_int(rng, 256, 2048)
        dtype = rng.choice(["u16", "u8", "f32"])
        return dict(kind="points", frames=_log_int(rng, 1, min(64, (1 << 27) // (h * w))), height=h, width=w,
                    spots=max(8, int(density * h * w)), diameter=rng.choice([9, 11, 15]), dtype=dtype,
                    bg={"u16": 100.0, "u8": 30.0, "f32": 50.0}[dtype])
    if kind == "link":
        side = _log_int(rng, 512, 2048)
        return dict(kind="link", frames=_log_int(rng, 20, 400), side=side,
                    spots=max(8, int(min(density, 4.8e-4) * side * side)), link=rng.choice([5.0, 6.0, 7.0]),
                    memory=rng.randint(0, 3))
    if kind == "learned":
        h, w = _log_int(rng, 512, 2048), _log_int(rng, 512, 2048)
        return dict(kind="learned", frames=_log_int(rng, 4, 64), height=h, width=w,
                    spots=max(8, int(density * h * w)), diameter=rng.choice([9, 11]), link=7.0,
                    memory=rng.randint(0, 3))
    return dict(kind="train", frames=_log_int(rng, 4, 16), side=512, spots=_log_int(rng, 60, 200),
                batch=rng.choice([64, 128, 256]), crop=rng.choice([64, 96, 128]), steps=rng.randint(4, 12))


def _drop_name(case):
    return {k: v for k, v in case.items() if k != "name"}


# --------------------------------------------------------------- the recordings
def _tracks(rng, case_rng, frames, height, width, spots, gap, diffusion=1.0, turnover=0.02, blink=0.02):
    """Positions (frames, spots, 2) and which spots are there, (frames, spots):
    Brownian steps reflected inside a cell of the spot's own, `gap` pixels clear
    of the next; a fraction of the spots starts afresh elsewhere in the cell, or
    is dark, in a frame."""
    down = max(1, round(math.sqrt(spots * height / width)))
    across = -(-spots // down)
    edge = 12.0
    cell = np.array([(height - 2 * edge) / down, (width - 2 * edge) / across])
    corner = np.stack(np.divmod(rng.permutation(down * across)[:spots], across), axis=1) * cell + edge + gap / 2.0
    size = np.maximum(cell - gap, 1.0)
    walk = np.cumsum(rng.normal(0.0, math.sqrt(2.0 * diffusion), (frames, spots, 2)), axis=0)
    fresh = rng.random((frames, spots)) < turnover
    fresh[0] = True
    born = np.maximum.accumulate(np.where(fresh, np.arange(frames)[:, None], 0), axis=0)
    start = rng.random((frames, spots, 2)) * size
    cols = np.arange(spots)[None, :]
    pos = start[born, cols] + walk - walk[born, cols]
    pos = np.abs(pos) % (2 * size)
    return corner + np.where(pos > size, 2 * size - pos, pos), case_rng.random((frames, spots)) >= blink


def _peaks(rng, spots, snr):
    lo, hi = math.log(snr[0]), math.log(snr[1])
    return np.exp(np.clip(rng.normal(0.5 * (lo + hi), (hi - lo) / 4.0, spots), lo, hi))


def _frames(seed, tracks, height, width, dtype, bg, sigma, snr, vignette=False):
    """The movie of the tracks on the GPU, (frames, height, width)."""
    tracks, there = tracks
    rng = np.random.default_rng([seed, 1])
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    count, spots = tracks.shape[:2]
    noise = 5.0 if dtype == "f32" else math.sqrt(bg)
    pos = torch.from_numpy(tracks).to(DEV, torch.float32)
    sig = torch.from_numpy(rng.uniform(sigma[0], sigma[1], spots)).to(DEV, torch.float32)
    amp = torch.from_numpy(_peaks(rng, spots, snr) * noise * there).to(DEV, torch.float32)
    reach = int(math.ceil(4 * sigma[1]))
    off = torch.arange(-reach, reach + 1, device=DEV, dtype=torch.float32)
    kind = {"u16": torch.uint16, "u8": torch.uint8, "f32": torch.float32}[dtype]
    movie = torch.empty((count, height, width), dtype=kind, device=DEV)
    if vignette:
        yy = (torch.arange(height, device=DEV, dtype=torch.float32) / height - 0.5) ** 2
        xx = (torch.arange(width, device=DEV, dtype=torch.float32) / width - 0.5) ** 2
        light = 1.0 / (1.0 + 0.8 * (yy[:, None] + xx[None, :]))
    step = max(1, min(32, (1 << 26) // (height * width), (1 << 24) // (spots * len(off) ** 2)))
    ph, pw = height + 2 * reach, width + 2 * reach  # a spot near the edge falls on the padding
    for t in range(0, count, step):
        p = pos[t:t + step]
        n = len(p)
        base = torch.floor(p)
        frac = p - base
        ey = torch.exp(-(off - frac[..., 0:1]) ** 2 / (2 * sig[None, :, None] ** 2)) * amp[t:t + n, :, None]
        ex = torch.exp(-(off - frac[..., 1:2]) ** 2 / (2 * sig[None, :, None] ** 2))
        val = (ey[..., :, None] * ex[..., None, :] * 65536.0).to(torch.int32)
        at = ((torch.arange(n, device=DEV)[:, None] * ph + base[..., 0].long() + reach) * pw
              + base[..., 1].long() + reach)
        spread = (off.long()[:, None] * pw + off.long()[None, :])
        img = torch.zeros(n * ph * pw, dtype=torch.int32, device=DEV)
        img.index_add_(0, (at[..., None, None] + spread).reshape(-1), val.reshape(-1))
        img = img.view(n, ph, pw)[:, reach:reach + height, reach:reach + width].float() / 65536.0 + bg
        if vignette:
            img *= light
        if dtype == "f32":
            movie[t:t + n] = img + noise * torch.randn(img.shape, generator=g, device=DEV)
        else:
            top = 255 if dtype == "u8" else 65535
            movie[t:t + n] = torch.poisson(img, generator=g).clamp_(0, top).to(torch.int32).to(kind)
    return movie


def _sigma(diameter):
    return diameter / 9.0, diameter / 5.0


def _snr(diameter, kind):
    """Peak over noise, from what the smoothing of the diameter still tells from noise."""
    lowest = {"learned": 12.0, "vignette": 15.0}.get(kind, 9.0)
    return max(lowest, 9.0 * (11.0 / diameter) ** 2), 35.0


def _minmass(diameter, noise):
    """Well above the mass of the noise's maxima and below that of the dimmest spots."""
    return round(27.0 * (diameter / 9.0) ** 1.35 * noise, 2)


def _options(case):
    kw = dict(tqdm=False)
    kind = case["kind"]
    if kind in ("batch", "videos", "learned"):
        noise = 5.0 if case.get("dtype") == "f32" else math.sqrt(case.get("bg", 100.0))
        if case.get("snr"):
            noise = 0.12  # of the frames divided by the smoothed mean
            kw.update(snr=case["snr"], correct_illumination=True)
        kw["minmass"] = _minmass(case["diameter"], noise)
        if kind == "videos":
            kw.update(characterize=False, doughnut_correction=False)
    elif kind == "log":
        kw.update(n_radii=case["n_radii"], log_spacing=True, minmass=150.0)
    if case.get("link") and kind != "link":
        kw.update(search_range=case["link"], memory=case["memory"])
    return kw


def _blob_net(net):
    """Weights that make the network a blob finder: the mean of each 4x4 cell,
    suppressed where one of the eight cells around it is brighter.  They stand
    for trained ones: the same layers and as many proposals as spots."""
    shapes = [(32, 16), (32, 32), (32, 32), (3, 32)]
    layers = [(np.zeros((co, ci, 9), np.float32), np.zeros(co, np.float32)) for co, ci in shapes]
    layers[0][0][0, :, 4] = 1.0 / 16.0
    layers[1][0][0, 0, 4] = 1.0
    around = [k for k in range(9) if k != 4]
    for c, k in enumerate(around):
        layers[1][0][1 + c, 0, k] = 1.0
        layers[1][0][1 + c, 0, 4] = -1.0
    layers[2][0][0, 0, 4] = 1.0
    layers[2][0][1, 1:9, 4] = 1.0
    layers[3][0][0, 0, 4] = 1.0
    layers[3][0][0, 1, 4] = -8.0
    net.params = np.concatenate([np.concatenate([w.ravel(), b]) for w, b in layers])
    net.set_normalization(100.0, 0.1)
    net.threshold = 0.6


def prepare(case, seed):
    rng = np.random.default_rng([seed, 0])
    fixed = np.random.default_rng(20)
    kind = case["kind"]
    state = {"case": case, "kw": _options(case)}
    if kind == "link":
        # given points keep no distance from one another
        side = case["side"]
        tracks, seen = _tracks(rng, fixed, case["frames"], side, side, case["spots"], 0.0)
        tracks = tracks + rng.normal(0.0, 0.1, tracks.shape)
        number = np.broadcast_to(np.arange(case["frames"])[:, None], seen.shape)
        state["rows"] = np.column_stack([number[seen], tracks[seen]]).astype(np.float32)
    elif kind == "videos":
        d = case["diameter"]
        state["videos"] = []
        for k, (t, h, w, density) in enumerate(_video_shapes(case)):
            tracks = _tracks(rng, fixed, t, h, w, max(1, int(density * h * w)), d + 4.0,
                             diffusion=rng.uniform(0.2, 2.0))
            state["videos"].append(_frames(seed * 64 + k, tracks, h, w, "u16", 100.0, _sigma(d), _snr(d, kind)))
    elif kind == "train":
        side = case["side"]
        tracks = _tracks(rng, fixed, case["frames"], side, side, case["spots"], 8.0)
        state["movie"] = _frames(seed, tracks, side, side, "u16", 100.0, _sigma(11), _snr(11, kind))
        number = np.broadcast_to(np.arange(case["frames"])[:, None], tracks[1].shape)
        state["labels"] = {"frame": number[tracks[1]], "y": tracks[0][tracks[1]][:, 0],
                           "x": tracks[0][tracks[1]][:, 1]}
        state["net"] = learned.ProposalNet(seed=seed % 1000)
        state["net"].set_normalization(100.0, 0.1)
        state["start"] = state["net"].params
    else:
        h, w = case["height"], case["width"]
        d = case.get("diameter", 9)
        tracks = _tracks(rng, fixed, case["frames"], h, w, case["spots"], d + 4.0)
        dtype = case.get("dtype", "f32" if kind == "log" else "u16")
        sigma = (2.0 / math.sqrt(2.0), case["max_radius"] / math.sqrt(2.0)) if kind == "log" else _sigma(d)
        bg = 50.0 if kind == "log" else case.get("bg", 100.0)
        state["movie"] = _frames(seed, tracks, h, w, dtype, bg, sigma,
                                 _snr(d, "vignette" if case.get("vignette") else kind), case.get("vignette", False))
        if case.get("host"):
            state["movie"] = state["movie"].cpu().numpy()
        if kind == "points":
            number = np.repeat(np.arange(case["frames"]), case["spots"])
            found = tracks[0] + rng.normal(0.0, 0.3, tracks[0].shape)
            state["points"] = np.column_stack([number, found.reshape(-1, 2)]).astype(np.float32)
        if kind == "learned":
            state["net"] = learned.ProposalNet(seed=0)
            _blob_net(state["net"])
    return state


def _video_shapes(case):
    """Sizes and lengths of the folder's recordings: part of the case, the same for every seed."""
    rng = np.random.default_rng(case["videos"] * 1000 + case["side_hi"])
    sides = [s for s in (256, 331, 512, 700, 1024, 1536, 2048) if case["side_lo"] <= s <= case["side_hi"]]
    return [(int(rng.integers(case["frames_lo"], case["frames_hi"] + 1)), int(rng.choice(sides)),
             int(rng.choice(sides)), float(rng.uniform(1e-4, 8e-4))) for _ in range(case["videos"])]


def _columns(table):
    return {name: table[name].to_numpy() for name in table.columns}


def _padded(columns, rows):
    out = {}
    for name, col in columns.items():
        out[name] = np.zeros(rows, col.dtype)
        out[name][:len(col)] = col[:rows]
    return out


def run(state):
    case, kw = state["case"], state["kw"]
    kind = case["kind"]
    if kind == "batch":
        return _columns(gt.batch(state["movie"], case["diameter"], **kw))
    if kind == "log":
        # how many blobs a frame has depends on its noise: the columns end in zeros
        return _padded(_columns(gt.LoG(state["movie"], case["min_radius"], case["max_radius"], **kw)),
                       2 * case["frames"] * case["spots"] + 1000)
    if kind == "videos":
        return [_columns(table) for table in gt.batch_videos(state["videos"], case["diameter"], **kw)]
    if kind == "points":
        return _columns(gt.characterize_points(state["movie"], state["points"], case["diameter"], has_frames=True,
                                               **kw))
    if kind == "link":
        return gt.link(state["rows"], case["link"], case["memory"])
    if kind == "learned":
        return _columns(learned.batch_learned(state["movie"], case["diameter"], state["net"], **kw))
    net = state["net"]
    net.params = state["start"]
    loss = net.train(state["movie"], state["labels"], steps=case["steps"], batch=case["batch"], crop=case["crop"])
    return {"loss": loss, "params": net.params}


# ------------------------------------------------------------------ what it takes
def work(case):
    kind = case["kind"]
    size = {"u8": 1, "u16": 2, "f32": 4}
    if kind == "link":
        rows = case["frames"] * case["spots"]
        return {"bytes": rows * (12 + 8), "flops": rows * 20 * (case["memory"] + 1)}
    cell_flops = 2 * 9 * (16 * 32 + 32 * 32 + 32 * 32 + 32 * 3)
    if kind == "train":
        cells = case["steps"] * case["batch"] * (case["crop"] // 4) ** 2
        # forward, and the backward pass of every layer's weights and (but the first's) inputs
        return {"bytes": cells * 16 * 2, "flops": cells * (3 * cell_flops - 2 * 9 * 16 * 32)}
    if kind == "videos":
        pixels = sum(t * h * w for t, h, w, _ in _video_shapes(case))
        rows = sum(t * int(density * h * w) for t, h, w, density in _video_shapes(case))
        taps, itemsize = case["diameter"], 2
    else:
        pixels = case["frames"] * case["height"] * case["width"]
        rows = case["frames"] * case["spots"]
        taps, itemsize = case.get("diameter", 17), size[case.get("dtype", "f32" if kind == "log" else "u16")]
    out = rows * ((4 if kind == "videos" else 11) + 2 * bool(case.get("link"))) * 4
    per_pixel = 2 * 2 * taps + 12  # two tap passes, two running sums, the window maxima
    if kind == "learned":
        per_pixel = cell_flops / 16
    elif kind == "points":
        per_pixel = 0  # only the pixels around the points are needed
        out += rows * 3 * 4
        return {"bytes": min(pixels, rows * (2 * taps) ** 2) * itemsize + out, "flops": rows * 400 * taps}
    elif kind == "log":
        lo, hi, n = case["min_radius"], case["max_radius"], case["n_radii"]
        radii = [lo * (hi / lo) ** (k / (n - 1)) for k in range(n)]
        per_pixel += sum(2 * 4 * (2 * int(4.0 * r / math.sqrt(2.0) + 0.5) + 1) for r in radii)
    return {"bytes": pixels * itemsize + out, "flops": pixels * per_pixel}


# ------------------------------------------------------------------ in 64 bits
def _bandpass64(img, diameter):
    """Gaussian (noise size 1, taps off the frame left out) minus boxcar (edge
    pixels repeated), values under 1/255 set to 0."""
    r = diameter // 2
    x = torch.arange(-r, r + 1, device=img.device, dtype=torch.float64)
    taps = torch.exp(-x * x / 2.0)
    norm = taps.sum()
    pad = torch.nn.functional.pad
    z = pad(img[None, None], (r, r, r, r))[0, 0]
    e = pad(img[None, None], (r, r, r, r), mode="replicate")[0, 0]
    h, w = img.shape
    rows = sum(taps[k] * z[:, k:k + w] for k in range(2 * r + 1)) / norm
    gauss = sum(taps[k] * rows[k:k + h] for k in range(2 * r + 1)) / norm
    ones = sum(e[:, k:k + w] for k in range(2 * r + 1))
    box = sum(ones[k:k + h] for k in range(2 * r + 1))
    out = gauss - box / float(diameter * diameter)
    return torch.where(out < 1.0 / 255.0, torch.zeros_like(out), out)


def _around(img, u, v, off):
    """Pixels at the offsets around (u, v), and which of them lie in the frame."""
    h, w = img.shape
    a, b = u[:, None] + off[:, 0], v[:, None] + off[:, 1]
    ok = (a >= 0) & (a < h) & (b >= 0) & (b < w)
    return torch.where(ok, img[a.clamp(0, h - 1), b.clamp(0, w - 1)], torch.zeros((), dtype=img.dtype,
                                                                                device=img.device)), ok


def _disk(outer, inner=-1.0):
    b = int(math.ceil(outer))
    return torch.tensor([(i, j) for i in range(-b, b + 1) for j in range(-b, b + 1)
                         if inner * abs(inner) <= i * i + j * j <= outer * outer], device=DEV)


def _describe64(img, proc, y, x, mass, diameter):
    """The columns of points at (y, x), from the raw and the processed frame."""
    off = _disk(float((diameter - 1) // 2))
    u, v = torch.round(y).long(), torch.round(x).long()
    p, _ = _around(proc, u, v, off)
    if mass is None:
        mass = p.sum(1)
    r2 = (off ** 2).sum(1).double()
    theta = torch.atan2(off[:, 1].double(), off[:, 0].double())
    rest = (r2 > 0).double()
    es = (p * torch.sin(2 * theta) * rest).sum(1)
    ec = (p * torch.where(r2 > 0, torch.cos(2 * theta), torch.ones_like(theta))).sum(1)
    middle, _ = _around(proc, u, v, torch.zeros((1, 2), dtype=torch.long, device=DEV))
    out = {"y": y, "x": x, "mass": mass, "Rg": torch.sqrt((p * r2).sum(1) / mass),
           "raw": _around(img, u, v, off)[0].sum(1), "signal": p.amax(1),
           "ecc": torch.sqrt(es * es + ec * ec) / (mass - middle[:, 0])}
    # the doughnut: the disk of half the diameter against the median of the ring to twice that
    radius = diameter / 2.0
    u, v = torch.floor(y + 0.5).long(), torch.floor(x + 0.5).long()
    disk, ok = _around(img, u, v, _disk(radius))
    ring, inside = _around(img, u, v, _disk(2 * radius, radius))
    ring = torch.where(inside, ring, torch.full_like(ring, math.inf)).sort(1).values
    median = ring.gather(1, (inside.sum(1, keepdim=True) // 2))[:, 0]
    out.update(raw_mass=disk.sum(1), raw_bg_median=median, raw_mass_corrected=disk.sum(1) - median * ok.sum(1))
    return out


def _locate64(img, diameter, minmass):
    """One frame of `batch`: local maxima, centroid walk, the brighter of close neighbours."""
    proc = _bandpass64(img, diameter)
    h, w = img.shape
    sep = diameter + 1
    size = int(2.0 * sep / math.sqrt(2.0))
    left = int(size / 2.0 - 0.5)
    pads = (left, size - 1 - left, left, size - 1 - left)
    top = torch.nn.functional.max_pool2d(torch.nn.functional.pad(proc[None, None], pads, value=-math.inf), size, 1)[0, 0]
    margin = max(diameter // 2, sep // 2 - 1)
    edge = torch.zeros_like(proc, dtype=torch.bool)
    edge[margin:h - margin, margin:w - margin] = True
    u, v = torch.nonzero((top <= proc) & edge & (proc > 0), as_tuple=True)
    r = (diameter - 1) // 2
    off = _disk(float(r))
    done = torch.zeros_like(u, dtype=torch.bool)
    cy = cx = mass = torch.zeros(len(u), dtype=torch.float64, device=DEV)
    for _ in range(10):
        p, _ = _around(proc, u, v, off)
        m = p.sum(1)
        dy, dx = (p * off[:, 0]).sum(1) / m, (p * off[:, 1]).sum(1) / m
        live = ~done
        mass = torch.where(live, m, mass)
        cy, cx = torch.where(live, dy, cy), torch.where(live, dx, cx)
        su = ((dy > 0.6) & (u < h - 1 - r)).long() - ((dy < -0.6) & (u > r)).long()
        sv = ((dx > 0.6) & (v < w - 1 - r)).long() - ((dx < -0.6) & (v > r)).long()
        done = done | ((su == 0) & (sv == 0))
        u, v = u + torch.where(done, 0, su), v + torch.where(done, 0, sv)
    keep = mass >= minmass
    y, x, mass = (cy + u)[keep], (cx + v)[keep], mass[keep]
    near = ((y[:, None] - y) ** 2 + (x[:, None] - x) ** 2 < sep * sep)
    order = torch.arange(len(y), device=DEV)
    beats = (mass[None, :] > mass[:, None]) | ((mass[None, :] == mass[:, None]) & (order[None, :] < order[:, None]))
    keep = ~(near & beats).any(1)
    return _describe64(img, proc, y[keep], x[keep], mass[keep], diameter)


def exact(case, seed):
    """The float columns of `batch` and `characterize_points`; the others have
    none (ids are whole, the scale space, the noise thresholds and the 16-bit
    network decide row by row what a table holds) or take too long."""
    if case["kind"] not in ("batch", "points") or case.get("snr"):
        return None
    if case["frames"] * case["height"] * case["width"] > 1.5e8:
        return None
    state = prepare(case, seed)
    movie = state["movie"]
    if isinstance(movie, np.ndarray):
        movie = torch.from_numpy(movie).to(DEV)
    found = []
    for t in range(case["frames"]):
        img = movie[t].to(torch.float64)
        if case["kind"] == "points":
            pts = torch.from_numpy(state["points"][state["points"][:, 0] == t]).to(DEV, torch.float64)
            found.append(_describe64(img, _bandpass64(img, case["diameter"]), pts[:, 1], pts[:, 2], None,
                                     case["diameter"]))
        else:
            found.append(_locate64(img, case["diameter"], state["kw"]["minmass"]))
    out = {name: torch.cat([f[name] for f in found]).cpu().numpy() for name in found[0]}
    out.update(frame=None)
    if case.get("link"):
        out.update(particle=None, duration=None)
    return out
