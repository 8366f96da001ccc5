"""The cleaning workloads whose speed this repository cares about.

Each case is one call (or one execution of a kept plan) through the public
entry points, on seeded synthetic scenes of the kind ``cusmic_b200.scenes``
describes (sky and read noise, Gaussian stars, cosmic-ray hits and tracks,
masked pixels, non-finite pixels), drawn on the GPU here because the inputs are
made many times over.  ``exact`` is L.A.Cosmic as the published chain of
full-frame filters, in float64 torch operations of its own.
"""

import ctypes
import math

import numpy as np
import torch

from cusmic_b200 import _native, remove_cosmics
from cusmic_b200.autograd import remove_cosmics_differentiable
from cusmic_b200.plan import Batch, Plan

CONTRAST, CR, NEIGHBOR = 3.0, 5.0, 3.0
GAIN, READNOISE = 2.0, 5.0
STAR_SIGMA = 2.5 / (2.0 * math.sqrt(2.0 * math.log(2.0)))
BORDERS = ("mirror", "reflect", "nearest", "wrap", "constant")

# Fields of a case and what most calls have.  api: "call" (remove_cosmics on
# device tensors), "plan" (a kept Plan with its graph, executed on frames in
# place), "grad" (the differentiable call and its backward), "host" (the C
# ABI's batch call on page-locked host buffers).  noise: "error" (one map shared
# by the frames), "scalar" (gain and read noise), "maps" (maps of both).
# stars, rays: per 512 x 512 pixels; tracks: the share of rays that are tracks.
DEFAULTS = dict(api="call", frames=1, height=512, width=512, ragged=False, shape_seed=0, lo=0,
                hi=0, noise="error", masked=0.0, holes=0.0, background="none", border="mirror",
                maxiter=4, stars=40.0, rays=150.0, tracks=0.4, shortest=2.0, longest=8.0, clip=0.0)


def _case(name, **fields):
    return dict(DEFAULTS, name=name, **fields)


def listed():
    return [
        # The smallest call: a cutout around one object, cleaned on its own in
        # an interactive session or a per-object loop.  Launches and latency.
        _case("cutout_128", height=128, width=128),
        # A small detector's frame with the textbook noise model.
        _case("frame_512", noise="scalar"),
        # One exposure of an ordinary camera from a reduction pipeline: error
        # map, bad-pixel mask, a few non-finite pixels.
        _case("frame_2048", height=2048, width=2048, masked=0.005, holes=0.001, stars=25.0,
              rays=75.0),
        # A trimmed detector (odd sides) with flat-field maps of gain and read
        # noise and a sky background map.
        _case("maps_1531x1023", height=1531, width=1023, noise="maps", background="map",
              masked=0.005, border="reflect"),
        # A short sequence of trimmed frames in one call, no two of whose rows
        # start alike, the noise model and a constant background.
        _case("sequence_5x1018x1001", frames=5, height=1018, width=1001, noise="scalar",
              masked=0.005, background="scalar", border="nearest"),
        # A night's stack of one camera, the benchmark's workload, on a kept
        # plan whose results are read in stream order.
        _case("stack_2048", api="plan", frames=16, height=2048, width=2048, masked=0.005,
              holes=0.001, stars=25.0, rays=75.0),
        # Frames of 64 different cameras or windows in one plan, each with its
        # own gain, read noise and background.
        _case("ragged_64", api="plan", ragged=True, frames=64, lo=256, hi=4096, noise="scalar",
              background="scalar"),
        # Many small cutouts of a survey in one plan.
        _case("stamps_256", api="plan", ragged=True, frames=256, shape_seed=1, lo=40, hi=200,
              noise="scalar", background="scalar"),
        # Wide-field mosaics: full-size error map, 2% masked, saturated stars,
        # long tracks.
        _case("mosaic_8192", api="plan", frames=2, height=8192, width=8192, masked=0.02, stars=0.8,
              rays=11.7, tracks=0.1, shortest=10.0, longest=40.0, clip=65535.0),
        # A reduction inside a differentiable pipeline: forward and backward.
        _case("adjoint_1024", api="grad", frames=8, height=1024, width=1024, noise="scalar"),
        # The same with one error map and a fitted sky map, whose gradient
        # comes back too.
        _case("adjoint_sky_777", api="grad", frames=3, height=777, width=900, background="map",
              masked=0.005),
        # Frames that arrive in and go back to host memory.
        _case("host_4x2048", api="host", frames=4, height=2048, width=2048, masked=0.005,
              holes=0.001, stars=25.0, rays=75.0),
    ]


def draw(rng):
    """One more case: sides and counts over the listed cases' whole range."""
    side = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    api = rng.choice(["call", "call", "call", "plan", "plan", "ragged", "ragged", "grad", "host"])
    c = dict(DEFAULTS)
    c["noise"] = rng.choice(["error", "error", "scalar", "scalar", "maps"])
    c["masked"] = rng.choice([0.0, 0.005, 0.02])
    c["holes"] = rng.choice([0.0, 0.0, 0.001])
    c["background"] = rng.choice(["none", "none", "scalar", "map"])
    c["border"] = rng.choice(("mirror", "mirror") + BORDERS)
    c["stars"], c["rays"] = rng.uniform(1, 40), rng.uniform(12, 150)
    c["tracks"] = rng.uniform(0.1, 0.4)
    if api == "ragged":
        c.update(api="plan", ragged=True, shape_seed=rng.randrange(1 << 20), noise="scalar",
                 masked=0.0, background=rng.choice(["none", "scalar"]))
        c["frames"] = side(8, 256)
        c["lo"] = side(40, 256)
        # The expected area keeps a batch below the listed one's.
        c["hi"] = side(2 * c["lo"], max(2 * c["lo"] + 1, min(4096, int(1.5e4 / math.sqrt(c["frames"])))))
        return c
    c["api"] = api
    c["height"], c["width"] = side(64, 4096), side(64, 4096)
    if rng.random() < 0.4:  # detectors' sides are often multiples of 64
        c["height"], c["width"] = -(-c["height"] // 64) * 64, -(-c["width"] // 64) * 64
    most = {"call": 8, "plan": 16, "grad": 8, "host": 4}[api]
    room = {"call": 3e7, "plan": 6e7, "grad": 1e7, "host": 1.7e7}[api]
    c["frames"] = max(1, min(side(1, most), int(room / (c["height"] * c["width"]))))
    return c


def _shapes(case):
    if not case["ragged"]:
        return [(case["height"], case["width"])] * case["frames"]
    rng = np.random.default_rng(case["shape_seed"])
    lo, hi = math.log(case["lo"]), math.log(case["hi"])
    hs = np.exp(rng.uniform(lo, hi, case["frames"])).astype(int)
    ws = np.exp(rng.uniform(lo, hi, case["frames"])).astype(int)
    return list(zip(hs.tolist(), ws.tolist()))


def _merge(cells, values):
    """Sums per distinct cell (on the host, so their order is fixed)."""
    at, inverse = np.unique(cells, return_inverse=True)
    return at, np.bincount(inverse, weights=values, minlength=at.size)


def _stars(rng, case, h, w):
    n = max(1, round(case["stars"] * h * w / 512 ** 2))
    ys, xs = rng.uniform(0, h, n), rng.uniform(0, w, n)
    lo, hi = (20000.0, 200000.0) if case["clip"] else (200.0, 20000.0)
    peaks = np.exp(rng.uniform(math.log(lo), math.log(hi), n))
    r = np.arange(-6, 7)
    py = ys.astype(int)[:, None, None] + r[None, :, None]
    px = xs.astype(int)[:, None, None] + r[None, None, :]
    r2 = (py - ys[:, None, None]) ** 2 + (px - xs[:, None, None]) ** 2
    v = peaks[:, None, None] * np.exp(-0.5 * r2 / STAR_SIGMA ** 2)
    ok = (py >= 0) & (py < h) & (px >= 0) & (px < w)
    return _merge((py * w + px)[ok], v[ok])


def _rays(rng, case, h, w):
    n = max(1, round(case["rays"] * h * w / 512 ** 2))
    ys, xs = rng.integers(0, h, n), rng.integers(0, w, n)
    amps = rng.uniform(500.0, 15000.0, n)
    length = np.where(rng.random(n) < case["tracks"],
                      rng.uniform(case["shortest"], case["longest"], n), 0.0)
    angle = rng.uniform(0, math.pi, n)
    s = np.linspace(-0.5, 0.5, 2 * math.ceil(case["longest"]))[None, :] * length[:, None]
    py = np.clip(np.rint(ys[:, None] + s * np.sin(angle)[:, None]).astype(int), 0, h - 1)
    px = np.clip(np.rint(xs[:, None] + s * np.cos(angle)[:, None]).astype(int), 0, w - 1)
    hit = np.unique(np.arange(n)[:, None] * (h * w) + py * w + px)  # a ray's cells once each
    return _merge(hit % (h * w), amps[hit // (h * w)])


def _scene(case, seed):
    """The inputs of a case on the GPU, as dict: frames (a list, views of
    `stack` when the shapes agree), error, mask, gain, readnoise, background
    (maps or per-frame scalars)."""
    rng = np.random.default_rng([seed, 1])
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    shapes = _shapes(case)
    total = sum(h * w for h, w in shapes)
    flat = torch.randn(total, generator=gen, device=dev, dtype=torch.float64)
    s = dict(frames=[], error=None, mask=None, gain=None, readnoise=None, background=None)
    scalars, at = [], 0
    for f, (h, w) in enumerate(shapes):
        gain, rn = (rng.uniform(1, 4), rng.uniform(2, 10)) if case["ragged"] else (GAIN, READNOISE)
        scalars.append((gain, rn, rng.uniform(0, 200)))
        sky = rng.uniform(500, 3000) if case["noise"] == "error" and not case["clip"] else 1000.0
        px = flat[at:at + h * w]
        at += h * w
        px.mul_(math.sqrt(sky * gain + rn * rn) / gain).add_(sky)
        star_at, star = (torch.from_numpy(a).to(dev) for a in _stars(rng, case, h, w))
        px[star_at] += star
        if f == 0 and case["noise"] == "error":
            model = torch.full((h * w,), sky, dtype=torch.float64, device=dev)
            model[star_at] += star
            if case["clip"]:
                model.clamp_(max=case["clip"])
            s["error"] = (model / 2 + 2.5 ** 2).sqrt().view(h, w)
        ray_at, ray = (torch.from_numpy(a).to(dev) for a in _rays(rng, case, h, w))
        px[ray_at] += ray
        s["frames"].append(px.view(h, w))
    if case["clip"]:
        flat.clamp_(max=case["clip"])
    if case["holes"]:
        flat[torch.rand(total, generator=gen, device=dev) < case["holes"]] = math.nan
    h, w = shapes[0]
    if case["masked"]:
        s["mask"] = torch.rand((h, w), generator=gen, device=dev) < case["masked"]
        s["mask"][:, rng.choice(w, 2, replace=False).tolist()] = True
    if case["noise"] == "maps":
        ripple = torch.rand((2, h, w), generator=gen, device=dev, dtype=torch.float64)
        s["gain"], s["readnoise"] = GAIN * (0.95 + 0.1 * ripple[0]), READNOISE * (0.9 + 0.2 * ripple[1])
    elif case["noise"] == "scalar":
        s["gain"], s["readnoise"] = ([q[k] for q in scalars] for k in (0, 1))
    if case["background"] == "scalar":
        s["background"] = [q[2] for q in scalars] if case["ragged"] else [scalars[0][2]] * len(shapes)
    elif case["background"] == "map":
        y = torch.linspace(0, 3, h, dtype=torch.float64, device=dev)[:, None]
        x = torch.linspace(0, 2, w, dtype=torch.float64, device=dev)[None, :]
        s["background"] = scalars[0][2] + 40 * torch.sin(x + y)
    if not case["ragged"]:
        s["stack"] = flat.view(len(shapes), h, w)
    s["flat"] = flat
    return s


def _one(v):
    """A map, or the scalar that every frame of a same-shaped case has."""
    return v[0] if isinstance(v, list) else v


def prepare(case, seed):
    s = _scene(case, seed)
    options = dict(contrast=CONTRAST, cr_threshold=CR, neighbor_threshold=NEIGHBOR,
                   maxiter=case["maxiter"])
    api = case["api"]
    if api in ("call", "grad"):
        data = s["stack"][0] if case["frames"] == 1 and api == "call" else s["stack"]
        kw = dict(options, error=s["error"], mask=s["mask"], background=_one(s["background"]),
                  effective_gain=_one(s["gain"]), readnoise=_one(s["readnoise"]),
                  border_mode=case["border"])
        st = dict(api=api, data=data, kw=kw)
        if api == "grad":
            gen = torch.Generator(device="cuda")
            gen.manual_seed(seed + 1)
            st["weight"] = torch.randn(data.shape, generator=gen, device="cuda", dtype=torch.float64)
            st["wrt"] = [data.requires_grad_()]
            if case["background"] == "map":
                st["wrt"].append(kw["background"].requires_grad_())
        return st
    if api == "plan":
        num = lambda v, i: v[i] if isinstance(v, list) else None
        nf = case["frames"]
        if case["ragged"]:
            scalars = [(num(s["gain"], i), num(s["readnoise"], i), num(s["background"], i))
                       for i in range(nf)]
            batch, more = Batch.ragged(s["frames"], scalars=scalars), {}
        else:
            is_map = lambda v: v if isinstance(v, torch.Tensor) else None
            batch = Batch.stack(s["stack"], error=s["error"], mask=s["mask"], gain=is_map(s["gain"]),
                                readnoise=is_map(s["readnoise"]), background=is_map(s["background"]))
            more = {k: _one(s[n]) for k, n in (("gain", "gain"), ("readnoise", "readnoise"),
                                               ("background", "background")) if isinstance(s[n], list)}
        return dict(api=api, batch=batch,
                    plan=Plan(batch, graph=True, border=case["border"], **options, **more))
    # Host buffers: a stack that several calls of the C ABI would share.
    pin = lambda t: None if t is None else t.detach().to("cpu").pin_memory()
    host = dict(data=pin(s["stack"]), error=pin(s["error"]),
                mask=pin(None if s["mask"] is None else s["mask"].to(torch.uint8)))
    for k in ("gain", "readnoise", "background"):
        host[k] = pin(s[k]) if isinstance(s[k], torch.Tensor) else None
    host["clean"] = torch.empty(host["data"].shape, dtype=torch.float64).pin_memory()
    host["flags"] = torch.empty(host["data"].shape, dtype=torch.uint8).pin_memory()
    o = _native.default_options()
    o.contrast, o.cr_threshold, o.neighbor_threshold = CONTRAST, CR, NEIGHBOR
    o.maxiter, o.border = case["maxiter"], _native.BORDERS[case["border"]]
    for k in ("gain", "readnoise", "background"):
        if isinstance(s[k], list):
            setattr(o, k, s[k][0])
    nf, (h, w) = case["frames"], _shapes(case)[0]
    ptr = lambda t: None if t is None else t.data_ptr()
    ims = (_native.Image * nf)()
    for f in range(nf):
        ims[f] = _native.Image(host["data"][f].data_ptr(), ptr(host["error"]), ptr(host["gain"]),
                               ptr(host["readnoise"]), ptr(host["background"]), ptr(host["mask"]), w, h)
    return dict(api=api, host=host, options=o, ims=ims, nf=nf)


def run(state):
    if state["api"] == "call":
        return remove_cosmics(state["data"], **state["kw"])
    if state["api"] == "plan":
        state["plan"].execute()
        return state["batch"].clean, state["batch"].mask_out
    if state["api"] == "grad":
        clean, mask = remove_cosmics_differentiable(state["data"], **state["kw"])
        grads = torch.autograd.grad(clean, state["wrt"], state["weight"])
        return (clean.detach(), mask) + grads
    host = state["host"]
    msg = ctypes.create_string_buffer(256)
    status = _native.lib().cusmic_batch_host(state["ims"], state["nf"], ctypes.byref(state["options"]),
                                             None, host["clean"].data_ptr(), host["flags"].data_ptr(),
                                             msg, 256)
    _native.raise_for(status, msg)
    return host["clean"].numpy(), host["flags"].numpy()


def work(case):
    shapes = _shapes(case)
    px, one = sum(h * w for h, w in shapes), shapes[0][0] * shapes[0][1]
    maps = 8 * ((case["noise"] == "error") + 2 * (case["noise"] == "maps") +
                (case["background"] == "map")) + (case["masked"] > 0)
    grad = (16 * px + 8 * one * (case["background"] == "map")) if case["api"] == "grad" else 0
    # Pixels in and out, the mask out, each map once; the Laplacian's about
    # twenty operations per pixel are what no evaluation can leave out.
    return {"bytes": 17 * px + maps * one + grad, "flops": 20 * px}


# --------------------------------------------------------------------------
# The same cleaning in 64 bits from torch operations, one frame at a time.

def _border(n, r, mode):
    """Source index of positions -r .. n + r - 1 (-1: zero)."""
    x = np.arange(-r, n + r)
    if mode == "nearest":
        x = x.clip(0, n - 1)
    elif mode == "wrap":
        x = x % n
    elif mode == "constant":
        x = np.where((x < 0) | (x >= n), -1, x)
    elif n == 1:
        x = np.zeros_like(x)
    elif mode == "reflect":
        x = x % (2 * n)
        x = np.where(x >= n, 2 * n - 1 - x, x)
    else:
        x = x % (2 * (n - 1))
        x = np.where(x >= n, 2 * (n - 1) - x, x)
    return x


def _pad(a, r, mode):
    iy, ix = (torch.from_numpy(_border(n, r, mode)).to(a.device) for n in a.shape)
    out = a[iy.clamp(min=0)][:, ix.clamp(min=0)]
    if mode == "constant":
        out[iy < 0] = 0
        out[:, ix < 0] = 0
    return out


def _exchanges(n):
    """Batcher's merge-exchange sort of n values, kept only where it can reach
    the middle one."""
    pairs, t = [], max(1, math.ceil(math.log2(n)))
    p = 1 << (t - 1)
    while p > 0:
        q, r, d = 1 << (t - 1), 0, p
        while d > 0:
            pairs += [(i, i + d) for i in range(n - d) if i & p == r]
            d, q, r = q - p, q >> 1, p
        p >>= 1
    need, kept = {n // 2}, []
    for i, j in reversed(pairs):
        if i in need or j in need:
            kept.append((i, j, i in need, j in need))
            need |= {i, j}
    return kept[::-1]


_NETWORKS = {n * n: _exchanges(n * n) for n in (3, 5, 7)}


def _median(a, n, mode):
    h, w = a.shape
    p = _pad(a, n // 2, mode)
    v = [p[i:i + h, j:j + w] for i in range(n) for j in range(n)]
    for i, j, low, high in _NETWORKS[n * n]:
        x, y = v[i], v[j]
        if low:
            v[i] = torch.minimum(x, y)
        if high:
            v[j] = torch.maximum(x, y)
    return v[n * n // 2]


def _laplacian(a, mode):
    mode = "nearest" if mode in ("mirror", "reflect") else mode
    p = _pad(a, 1, mode) / 4
    c = a / 4
    up, down = c - p[:-2, 1:-1], c - p[2:, 1:-1]
    left, right = c - p[1:-1, :-2], c - p[1:-1, 2:]
    pos = lambda v: v.clamp(min=0)
    return (pos(up + left) + pos(up + right)) + (pos(down + left) + pos(down + right))


def _dilate(b):
    p = torch.nn.functional.pad(b, (1, 1, 1, 1))
    h, w = b.shape
    out = torch.zeros_like(b)
    for i in range(3):
        for j in range(3):
            out |= p[i:i + h, j:j + w]
    return out


def _donor_medians(clean, targets, donors):
    """For each target pixel the two central donors (linear indices) of the
    smallest clipped window (radius 2, 3, ...) that holds one, and whether the
    count is even; donors ordered by value, ties by index."""
    h, w = clean.shape
    pix = targets.flatten().nonzero()[:, 0]
    lo, hi = torch.zeros_like(pix), torch.zeros_like(pix)
    even = torch.zeros_like(pix, dtype=torch.bool)
    left = torch.arange(pix.numel(), device=pix.device)
    r = 2
    while left.numel():
        if r > max(h, w):
            raise ValueError("no finite replacement donors")
        d = torch.arange(-r, r + 1, device=pix.device)
        y = (pix[left] // w)[:, None, None] + d[:, None]
        x = (pix[left] % w)[:, None, None] + d
        inside = ((y >= 0) & (y < h) & (x >= 0) & (x < w)).flatten(1)
        at = (y.clamp(0, h - 1) * w + x.clamp(0, w - 1)).flatten(1)
        ok = inside & donors.view(-1)[at]
        value, order = torch.where(ok, clean.view(-1)[at], math.inf).sort(dim=1, stable=True)
        n = ok.sum(1)
        some = n > 0
        pick = lambda k: at.gather(1, order.gather(1, k[:, None].clamp(min=0)))[:, 0]
        lo[left[some]], hi[left[some]] = pick((n - 1) // 2)[some], pick(n // 2)[some]
        even[left[some]] = (n % 2 == 0)[some]
        left = left[~some]
        r += 1
    return pix, lo, hi, even


def _replace(clean, targets, donors):
    pix, lo, hi, even = _donor_medians(clean, targets, donors)
    v = clean.view(-1)
    v[pix] = torch.where(even, v[lo] / 2 + v[hi] / 2, v[lo])


def _clean_exact(data, error, mask, gain, rn, bg, mode, maxiter):
    """(cleaned, flags, working pixels' donors) of one frame."""
    hole = ~torch.isfinite(data)
    excluded = hole | mask if mask is not None else hole
    clean = torch.where(hole, 0.0, data)
    if bg is not None:
        clean = clean + bg
    if hole.any():
        _replace(clean, hole, ~excluded)
    crmask = torch.zeros_like(hole)
    for _ in range(maxiter):
        noise = error
        if noise is None:
            noise = (rn * rn + gain * _median(clean, 5, mode).clamp(min=1e-5)).sqrt() / gain
        raw = _laplacian(clean, mode) / (2 * noise)
        sig = torch.where(hole, 0.0, raw - _median(raw, 5, mode))
        med3 = _median(clean, 3, mode)
        fine = ((med3 - _median(med3, 7, mode)) / noise).clamp(min=0.01)
        seed = ~excluded & (sig > CR) & (sig / fine > CONTRAST)
        grown = _dilate(_dilate(seed) & (sig > CR)) & (sig > NEIGHBOR)
        if not (grown & ~crmask).any():
            break
        crmask |= grown
        _replace(clean, crmask, ~excluded & ~crmask)
    out = clean if bg is None else clean - bg
    return torch.where(hole, data, out), crmask, ~excluded & ~crmask


def exact(case, seed):
    s = _scene(case, seed)
    mode, outs, flags, grads = case["border"], [], [], []
    sky = case["api"] == "grad" and case["background"] == "map"
    g_sky = torch.zeros_like(s["background"]) if sky else None
    if case["api"] == "grad":
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed + 1)
        weight = torch.randn(s["stack"].shape, generator=gen, device="cuda", dtype=torch.float64)
    at = lambda v, f: v[f] if isinstance(v, list) else v
    for f, data in enumerate(s["frames"]):
        bg = at(s["background"], f)
        out, crmask, donors = _clean_exact(data, s["error"], s["mask"], at(s["gain"], f),
                                           at(s["readnoise"], f), bg, mode, case["maxiter"])
        outs.append(out)
        flags.append(crmask)
        if case["api"] == "grad":
            # Flagged pixels send their gradient to their donors, the others
            # pass it on.
            g = weight[f].masked_fill(crmask, 0.0).view(-1)
            work = data if bg is None else data + bg
            pix, lo, hi, even = _donor_medians(work, crmask, donors)
            share = weight[f].view(-1)[pix]
            half = torch.where(even, share / 2, share)
            moved = torch.zeros_like(g)
            moved.index_add_(0, lo, half)
            moved.index_add_(0, hi[even], half[even])
            grads.append((g + moved).view_as(data))
            if sky:
                moved[pix] -= share
                g_sky += moved.view_as(data)
    if case["ragged"]:
        return torch.cat([o.reshape(-1) for o in outs]), torch.cat([q.reshape(-1) for q in flags])
    clean, mask = torch.stack(outs), torch.stack(flags)
    if case["api"] == "call" and case["frames"] == 1:
        return clean[0], mask[0]
    if case["api"] == "grad":
        return (clean, mask, torch.stack(grads)) + ((g_sky,) if sky else ())
    return clean, mask
