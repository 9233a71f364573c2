"""Timed cases: the calls that programs using this framework make, over the range they make them.

A case is a plain dict; ``prepare`` builds what a program holds before the call (inputs from the
seed, and the batch or emulsion it keeps), ``run`` is one pass through the public entry points and
returns every result, ``exact`` gives the results that plain numpy / torch can form in 64 bits.

Exposure images are blurred noise stretched to the whole range of a photograph (0 to 1), so tiles
hold unexposed, partly and fully developed regions; film pixels are 1 / grain micrometres wide with
each stock's grain size at 35 mm.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import fgrain_gb300 as fg
from fgrain_gb300 import fast, film, image

STOCKS = ("tri-x", "t-max", "hp5")
# Per stock: half-dimension statistics and shape of the uploaded crystal sets (depth um, r_min,
# mean radius, log-normal width, thickness ratio, base sensitivity).
SETS = {"tri-x": (14.0, 1.2, 0.55, 0.40, 1.0, 1.2), "t-max": (8.0, 0.9, 0.40, 0.20, 6.5, 0.8),
        "hp5": (12.5, 1.1, 0.50, 0.30, 1.0, 1.1)}
OTF_TAPS = (0.035, 0.93, 0.035)


def listed():
    return [
        # One preview-sized tile, plan to pixels in one blocking call: the smallest render, where
        # launches and latency count.
        {"name": "tile_small", "kind": "tile", "stock": "tri-x", "w": 64, "h": 64, "push": 0.0},
        # The last tile of a row and column of an image (odd sizes), pushed, through the same call.
        {"name": "tile_ragged", "kind": "tile", "stock": "t-max", "w": 187, "h": 301, "push": 1.0},
        # A 1024 x 1024 photograph at supersample 2: the 49 tiles in one batch that the program
        # keeps (cubic grains).
        {"name": "image_trix", "kind": "image", "stock": "tri-x", "w": 2048, "h": 2048, "push": 0.0},
        # One layer of a fine-grained photograph (tabular grains, about 19 M crystals): the largest.
        {"name": "image_tmax", "kind": "image", "stock": "t-max", "w": 1600, "h": 1600, "push": 0.0},
        # An album: images of different sizes, stocks and push in one batch.
        {"name": "album", "kind": "album", "images": 10, "side": 400},
        # A photograph from RGB pixels to a finished gray image, and one to three dye layers at
        # supersample 2, each one call from host pixels to host pixels.
        {"name": "film_gray", "kind": "film", "stock": "tri-x", "w": 750, "h": 533, "color": False, "ss": 1, "push": 0.0},
        {"name": "film_color", "kind": "film", "stock": "t-max", "w": 231, "h": 317, "color": True, "ss": 2, "push": 0.0},
        # A demonstration patch stage by stage: synthesis, exposure, development, scan.
        {"name": "emulsion", "kind": "emulsion", "stock": "hp5", "um": 90.0, "px": 384, "spp": 4},
        # Exposure of a crystal set that the program uploaded (FP64 records).
        {"name": "expose", "kind": "expose", "stock": "tri-x", "um": 130.0, "px": 312},
        # One optimisation step over the scan: forward, loss gradient, backward.
        {"name": "gradient", "kind": "gradient", "stock": "t-max", "w": 701, "h": 640, "spp": 4},
        # The fast approximation of a 1024 x 1024 image.
        {"name": "fast", "kind": "fast", "stock": "tri-x", "w": 1024, "h": 1024, "push": 0.0},
        # The image stages around the tiles, one by one, as a custom pipeline calls them.
        {"name": "stages", "kind": "stages", "stock": "tri-x", "w": 1501, "h": 1003},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("tile", "image", "album", "film", "emulsion", "expose", "gradient", "fast", "stages"))
    stock = rng.choice(STOCKS)
    push = rng.choice((0.0, 0.0, round(rng.uniform(0.0, 3.0), 2)))
    c = {"kind": kind}
    if kind == "tile":
        c.update(stock=stock, w=_log(rng, 40, 384), h=_log(rng, 40, 384), push=push)
    elif kind == "image":
        top = 1400 if stock == "t-max" else 1800
        c.update(stock=stock, w=_log(rng, 300, top), h=_log(rng, 300, top), push=push)
    elif kind == "album":
        c.update(images=rng.randint(3, 12), side=_log(rng, 100, 400))
    elif kind == "film":
        color, ss = rng.random() < 0.4, rng.randint(1, 3)
        top = (500 if color else 900) // ss
        c.update(stock=stock, w=_log(rng, 80, top), h=_log(rng, 80, top), color=color, ss=ss, push=push)
    elif kind == "emulsion":
        c.update(stock=stock, um=round(rng.uniform(20.0, 120.0), 1), px=_log(rng, 64, 512), spp=rng.choice((1, 4, 9, 16)))
    elif kind == "expose":
        c.update(stock=stock, um=round(rng.uniform(20.0, 140.0), 1), px=_log(rng, 48, 384))
    elif kind == "gradient":
        c.update(stock=stock, w=_log(rng, 100, 900), h=_log(rng, 100, 900), spp=rng.choice((1, 4, 4, 9)))
    elif kind == "fast":
        c.update(stock=stock, w=_log(rng, 100, 1100), h=_log(rng, 100, 1100), push=push)
    else:
        c.update(stock=stock, w=_log(rng, 200, 1600), h=_log(rng, 200, 1600))
    return c


# ---- inputs ----

def _photo(rng, h, w, sigma):
    """Blurred uniform noise (Gaussian, periodic) stretched to [0, 1], float64 [h, w]."""
    fy, fx = np.fft.fftfreq(h)[:, None], np.fft.rfftfreq(w)[None, :]
    g = np.exp(-2.0 * (np.pi * sigma) ** 2 * (fx * fx + fy * fy))
    a = np.fft.irfft2(np.fft.rfft2(rng.random((h, w))) * g, s=(h, w))
    return (a - a.min()) / max(a.max() - a.min(), 1e-12)


def _image_tiles(exposure, stock, push, seed):
    grain = image.default_grain_px(stock, push)
    h, w = exposure.shape
    grid, _, _ = image.tile_grid(w, h, grain)
    params = image.image_tile_params(stock, grain, grid, 1.0, image.effective_push(stock, push), seed)
    tiles = [np.ascontiguousarray(exposure[t.y_start:t.y_start + t.th, t.x_start:t.x_start + t.tw]) for t in grid]
    return params, tiles


def _crystal_set(rng, stock, w_um, h_um):
    """A host crystal set: a jittered lattice with the stock's density and attributes, so that
    crystals keep about r_min apart."""
    depth, r, mean, width, aspect, sens = SETS[stock]
    step = 1.2 * r
    n = [max(int(v / step), 1) for v in (w_um, h_um, depth)]
    gz, gy, gx = np.meshgrid(*(np.arange(k) for k in n[::-1]), indexing="ij")
    cell = np.array([w_um / n[0], h_um / n[1], depth / n[2]])
    pos = (np.stack([gx, gy, gz], -1).reshape(-1, 3) + 0.5 + rng.uniform(-0.12, 0.12, (gx.size, 3))) * cell
    m = pos.shape[0]
    rad = np.clip(np.exp(rng.normal(math.log(mean), width, m)), 0.15, 0.48 * r)
    dims = np.stack([rad, rad, np.maximum(rad / aspect, 0.05) if stock == "t-max" else rad], -1)
    if stock == "t-max":
        tilt, phi = rng.uniform(-0.17, 0.17, m), rng.uniform(0.0, 2.0 * np.pi, m)
        quat = np.stack([np.cos(phi) * np.sin(tilt / 2), np.sin(phi) * np.sin(tilt / 2), np.zeros(m), np.cos(tilt / 2)], -1)
    else:
        quat = rng.normal(size=(m, 4))
    quat /= np.linalg.norm(quat, axis=1, keepdims=True)
    return pos, dims, quat, np.maximum(rng.normal(sens, 0.15, m), 0.1)


def _gradient_inputs(case, seed):
    """The crystals, their development and the loss of a gradient case (host arrays)."""
    rng = np.random.default_rng([seed, 5])
    px = 1.0 / image.default_grain_px(case["stock"])
    w_um, h_um = case["w"] * px, case["h"] * px
    crystals = _crystal_set(rng, case["stock"], w_um, h_um)
    n = crystals[0].shape[0]
    developed = (rng.random(n) < 0.3).astype(np.uint8)
    clump = rng.integers(1, 7, n)
    boost = np.where(clump > 1, 1.15 + 0.18 * (clump - 1), 1.0)
    expansion = np.where(developed, 1.15 * boost, 0.0)
    sigma = rng.uniform(0.2, 0.3, n).astype(np.float32)
    target = rng.uniform(0.6, 1.0, (case["h"], case["w"])).astype(np.float32)
    return w_um, h_um, crystals, developed, expansion, sigma, target


def _stage_inputs(case, seed):
    rng = np.random.default_rng([seed, 6])
    w, h = case["w"], case["h"]
    gray = np.round(_photo(rng, h, w, 9.0) * 255.0).astype(np.uint8)
    gray[: h // 16] = 0  # a letterboxed frame: the camera gate
    gray[h - h // 16:] = 0
    rgb = np.stack([np.round(_photo(rng, h // 2, w // 2, 7.0) * 255.0).astype(np.uint8) for _ in range(3)], -1)
    grain = image.default_grain_px(case["stock"])
    grid, step, pad = image.tile_grid(w, h, grain)
    dens = [(0.05 + rng.gamma(2.0, 0.04, (t.th, t.tw))).astype(np.float32) for t in grid]
    return gray, np.ascontiguousarray(rgb), grain, grid, step, pad, dens


def prepare(case, seed):
    kind, stock = case["kind"], case.get("stock")
    rng = np.random.default_rng([seed, 1])
    s = {"kind": kind, "case": case, "engine": fg.get_gpu_engine()}
    if kind == "tile":
        grain = image.default_grain_px(stock, case["push"])
        s["params"] = fg.tile_params(stock, 1.0 / grain, case["w"], case["h"], 1.0, case["push"], seed * 7919 + 1)
        s["tile"] = _photo(rng, case["h"], case["w"], max(case["h"], case["w"]) / 12).astype(np.float32)
    elif kind in ("image", "album"):
        params, tiles = [], []
        if kind == "image":
            exposure = _photo(rng, case["h"], case["w"], 32.0).astype(np.float32)
            params, tiles = _image_tiles(exposure, stock, case["push"], seed)
        else:
            sizes = np.random.default_rng([case["images"], case["side"]])  # the album's sizes are the case's
            for k in range(case["images"]):
                h, w = (int(round(math.exp(v))) for v in sizes.uniform(math.log(64), math.log(case["side"]), 2))
                push = float(sizes.choice([0.0, 0.0, 1.0, 2.5]))
                exposure = _photo(rng, h, w, max(h, w) / 16).astype(np.float32)
                p, t = _image_tiles(exposure, STOCKS[k % 3], push, seed * 131 + k)
                params += p
                tiles += t
        s["batch"] = fg.Batch(params, s["engine"])
        s["tiles"] = tiles
    elif kind == "film":
        planes = [_photo(rng, case["h"], case["w"], 12.0) for _ in range(3)]
        s["pixels"] = np.ascontiguousarray(np.round(np.stack(planes, -1) * 255.0).astype(np.uint8))
        s["options"] = film.FilmRenderOptions(preset=stock, grain_size_px=image.default_grain_px(stock, case["push"]),
                                              color=case["color"], supersample=case["ss"], push=case["push"], seed=seed)
    elif kind == "emulsion":
        s["config"] = fg.EmulsionConfig.preset(stock, case["um"], case["um"])
        s["tile"] = _photo(rng, 128, 128, 10.0).astype(np.float32)
        s["seed"] = seed
    elif kind == "expose":
        s["config"] = fg.EmulsionConfig.preset(stock, case["um"], case["um"])
        s["emulsion"] = fg.VirtualEmulsionLayer.from_crystals(s["config"], *_crystal_set(rng, stock, case["um"], case["um"]),
                                                              engine=s["engine"])
        s["tile"] = _photo(rng, case["px"], case["px"], case["px"] / 12).astype(np.float32)
        s["zero"] = np.zeros(len(s["emulsion"]), np.uint32)
        s["seed"] = seed
    elif kind == "gradient":
        w_um, h_um, crystals, developed, expansion, sigma, target = _gradient_inputs(case, seed)
        config = fg.EmulsionConfig.preset(stock, w_um, h_um)
        s["emulsion"] = fg.VirtualEmulsionLayer.from_crystals(config, *crystals, engine=s["engine"])
        s["emulsion"].set_development(developed, expansion)
        s.update(sigma=sigma, target=target, seed=seed,
                 scan=fg.ScanConfig(case["w"], case["h"], case["spp"], fg.ScanMode.NegativeTransmittance, 0.25))
    elif kind == "fast":
        grain = image.default_grain_px(stock, case["push"])
        exposure = _photo(rng, case["h"], case["w"], 24.0).astype(np.float32)
        grid, _, _ = image.tile_grid(case["w"], case["h"], grain)
        s["params"] = [fast.tile_params_fast(stock, 1.0 / grain, t.tw, t.th, 1.0, case["push"], image.tile_seed(seed, t))
                       for t in grid]
        s["tiles"] = [np.ascontiguousarray(exposure[t.y_start:t.y_start + t.th, t.x_start:t.x_start + t.tw]) for t in grid]
    else:
        s["inputs"] = _stage_inputs(case, seed)
    return s


def run(state):
    kind, case, engine = state["kind"], state["case"], state["engine"]
    if kind == "tile":
        return fg.render_tile(state["tile"], state["params"], engine)
    if kind in ("image", "album"):
        b = state["batch"]
        b.set_exposure(state["tiles"])
        b.run()
        stats = b.wait()
        return {"density": b.density(), **{k: stats[k] for k in ("crystals", "photons", "hits", "scan_hits", "developed", "clumps")}}
    if kind == "film":
        report, out = film.render_film(state["pixels"], state["options"], engine)
        return {"image": out, "crystals": report.total_crystals, "developed": report.developed_crystals,
                "clumps": report.total_clumps}
    if kind == "emulsion":
        em = fg.VirtualEmulsionLayer.synthesize(state["config"], 42, engine)  # the demonstrations' patch seed
        fg.expose_emulsion(em, state["tile"], fg.ExposureConfig(6.0, 0.12, 1.3, 48), state["seed"] + 1)
        rep = fg.develop_emulsion(em, fg.DevelopmentConfig(4, 1.15, 1.18, 0.85))
        scan, img = fg.scan_emulsion(em, fg.ScanConfig(case["px"], case["px"], case["spp"], fg.ScanMode.PositivePrint, 0.40),
                                     state["seed"] + 2)
        counts = em.latent_counts()
        em.close()
        return {"scan": scan, "image": img, "counts": counts, "developed": rep.developed_crystals, "clumps": rep.total_clumps}
    if kind == "expose":
        em = state["emulsion"]
        em.set_latent_counts(state["zero"])
        fg.expose_emulsion(em, state["tile"], fg.ExposureConfig(6.0, 0.12, 1.3, 48), state["seed"])
        return em.latent_counts()
    if kind == "gradient":
        em, scan, sigma, target = (state[k] for k in ("emulsion", "scan", "sigma", "target"))
        signal, trans = fg.scan_signal(em, scan, state["seed"], sigma, 0.9, 0.45)
        upstream = (signal - target) * np.float32(2.0 / signal.size)
        g_sigma, g_exposure, g_otf = fg.scan_backward(em, scan, state["seed"], upstream, sigma, 0.9, 0.45)
        return {"signal": signal, "transmittance": trans, "g_sigma": g_sigma, "g_exposure": g_exposure, "g_otf": g_otf}
    if kind == "fast":
        return fast.render_tiles_fast(state["params"], state["tiles"], engine)
    gray, rgb, grain, grid, step, pad, dens = state["inputs"]
    w, h = case["w"], case["h"]
    luma = film.panchromatic_luma(rgb, case["stock"], engine)
    up = film.resize_u8(luma, w, h, film.LANCZOS3, engine)
    heff, _ = film.gelatin_psf(gray, engine)
    out, _ = film.film_finish(case["stock"], grain, 1.0, 0.0, True, w, h, grid, step, pad, dens, gray, heff, engine=engine)
    d_norm = image.blend_tiles(w, h, grid, step, pad, dens)
    sharp = image.scanner_otf(d_norm)
    small = image.resize_triangle(sharp, max(w // 2, 1), max(h // 2, 1))
    return {"luma": luma, "up": up, "heff": heff, "out": out, "d_norm": d_norm, "sharp": sharp, "small": small}


# ---- work that a pass cannot do without ----

def _film_work(px, um2, crystals_um2):
    """Exposure in, density out; per photon (six per um^2) its emission, about two segments and five
    absorbing hits, per pixel four scanner rays."""
    return {"bytes": 8.0 * px, "flops": 6.0 * um2 * 500.0 + px * 4.0 * 60.0 + crystals_um2 * um2 * 100.0}


def _per_um2(stock):
    depth, r = SETS[stock][:2]
    return 0.58 * depth / r ** 3


def work(case):
    kind, stock = case["kind"], case.get("stock")
    if kind == "album":
        side = math.sqrt(64 * case["side"])
        return _film_work(case["images"] * side * side, case["images"] * side * side / 3.2, 5.0)
    grain = image.default_grain_px(stock, case.get("push", 0.0))
    if kind in ("tile", "image"):
        px = case["w"] * case["h"]
        return _film_work(px, px / grain ** 2, _per_um2(stock))
    if kind == "film":
        px = case["w"] * case["h"]
        big = px * case["ss"] ** 2 * (3 if case["color"] else 1)
        return {"bytes": px * (6.0 if case["color"] else 4.0), "flops": _film_work(big, big / grain ** 2, _per_um2(stock))["flops"]}
    if kind == "emulsion":
        um2, px = case["um"] ** 2, case["px"] ** 2
        n = _per_um2(stock) * um2
        return {"bytes": 128 * 128 * 4.0 + px * 5.0 + n * 4.0, "flops": um2 * 6.0 * 500.0 + px * case["spp"] * 60.0 + n * 100.0}
    if kind == "expose":
        um2 = case["um"] ** 2
        n = _per_um2(stock) * um2
        return {"bytes": case["px"] ** 2 * 4.0 + n * (48.0 + 8.0), "flops": um2 * 6.0 * 500.0}
    if kind == "gradient":
        px = case["w"] * case["h"]
        n = _per_um2(stock) * px / grain ** 2
        return {"bytes": px * 16.0 + n * (48.0 + 9.0 + 8.0), "flops": px * case["spp"] * 240.0}
    if kind == "fast":
        px = case["w"] * case["h"]
        return {"bytes": px * 8.0, "flops": px * 4.0 * 200.0}
    px = case["w"] * case["h"]
    return {"bytes": px * 40.0, "flops": px * 120.0}


# ---- results in 64 bits ----

def exact(case, seed):
    if case["kind"] == "gradient" and case["stock"] != "tri-x":  # ellipsoids: hits by geometry alone
        return _exact_gradient(case, seed)
    if case["kind"] == "stages":
        return _exact_stages(case, seed)
    return None


def _philox(c0, k0, k1):
    """First two words of Philox-4x32-10 (Salmon et al., SC'11) for counters (c0, 0, 0, 'SC')."""
    mask = (1 << 32) - 1
    c = [c0, torch.zeros_like(c0), torch.zeros_like(c0), torch.full_like(c0, 0x53430000)]
    # 32 x 32 -> 64 bit products from 16-bit halves (torch has signed 64-bit integers only).
    def mul(m, v):
        lo, mid = m * (v & 0xFFFF), m * (v >> 16)
        full_lo = (lo + ((mid & 0xFFFF) << 16))
        return ((mid >> 16) + (full_lo >> 32)) & mask, full_lo & mask
    for _ in range(10):
        h0, l0 = mul(0xD2511F53, c[0])
        h1, l1 = mul(0xCD9E8D57, c[2])
        c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
        k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
    return c[0], c[1]


def _rays(case, seed, w_um, h_um, dev):
    """Scanner ray origins (um): one jittered ray per stratum of each pixel, [h, w, strata]."""
    g = int(round(math.sqrt(case["spp"])))
    px = torch.arange(case["w"], device=dev)[None, :, None]
    py = torch.arange(case["h"], device=dev)[:, None, None]
    st = torch.arange(g * g, device=dev)[None, None, :]
    signed = lambda v: v - (1 << 64) if v >= 1 << 63 else v
    key = seed + px * signed(0x9E3779B97F4A7C15) + py * signed(0xC6A4A7935BD1E995)  # wraps modulo 2^64
    k0, k1 = key & 0xFFFFFFFF, (key >> 32) & 0xFFFFFFFF
    shape = (case["h"], case["w"], g * g)
    u, v = _philox(st.expand(shape).contiguous(), k0.expand(shape), k1.expand(shape))
    ux, uy = (u >> 8).double() * 2.0 ** -24, (v >> 8).double() * 2.0 ** -24
    x = (px.double() + ((st % g).double() + ux) / g) * (w_um / case["w"])
    y = (py.double() + ((st // g).double() + uy) / g) * (h_um / case["h"])
    return x, y


def _exact_gradient(case, seed):
    w_um, h_um, (pos, dims, quat, _), developed, expansion, sigma, target = _gradient_inputs(case, seed)
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    ids = np.flatnonzero(developed)
    up = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)
    e = up(expansion[ids])
    p, d, q, sg = up(pos[ids]), up(dims[ids]) * e[:, None], up(quat[ids]), up(sigma[ids])
    W, H = case["w"], case["h"]
    ox, oy = _rays(case, seed, w_um, h_um, dev)
    x, y, z, w = q.unbind(1)
    rows = (torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w)], 1),
            torch.stack([2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w)], 1),
            torch.stack([2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], 1))
    z0 = SETS[case["stock"]][0] + 0.1
    m = d.max(1).values
    pw, ph = w_um / W, h_um / H
    bx, by = torch.floor((p[:, 0] - m) / pw).long(), torch.floor((p[:, 1] - m) / ph).long()
    nx = int(torch.ceil(2 * m.max() / pw).item()) + 1
    ny = int(torch.ceil(2 * m.max() / ph).item()) + 1

    def chords():
        """(flat ray index, crystal index, chord) of the hits, pixel offset by pixel offset."""
        for j in range(ny):
            for i in range(nx):
                gx, gy = bx + i, by + j
                c = torch.nonzero((gx >= 0) & (gx < W) & (gy >= 0) & (gy < H)).squeeze(1)
                if not c.numel():
                    continue
                cell = gy[c] * W + gx[c]
                for s in range(ox.shape[2]):
                    dx = ox.view(-1, ox.shape[2])[cell, s] - p[c, 0]
                    dy = oy.view(-1, oy.shape[2])[cell, s] - p[c, 1]
                    dz = z0 - p[c, 2]
                    lo = (rows[0][c] * dx[:, None] + rows[1][c] * dy[:, None] + rows[2][c] * dz[:, None]) / d[c]
                    ld = -rows[2][c] / d[c]
                    a, b, k = (ld * ld).sum(1), 2 * (lo * ld).sum(1), (lo * lo).sum(1) - 1
                    disc = b * b - 4 * a * k
                    sq = torch.sqrt(disc.clamp(min=0))
                    t0, t1 = (-b - sq) / (2 * a), (-b + sq) / (2 * a)
                    hit = torch.nonzero((disc >= 0) & (t1 > 0)).squeeze(1)
                    yield cell[hit] * ox.shape[2] + s, c[hit], t1[hit] - t0[hit].clamp(min=0)

    L = torch.zeros(ox.numel(), dtype=torch.float64, device=dev)
    for ray, c, chord in chords():
        L.index_add_(0, ray, sg[c] * chord)
    ray_t = torch.exp(-L)
    T = ray_t.view(H, W, -1).mean(2)
    exposure, width = 0.9, 0.45
    g = math.exp(-1.0 / (2.0 * width * width))
    n = 1.0 + 2.0 * g
    dg = g / width ** 3
    k, dk = (g / n, 1.0 / n, g / n), (dg / n ** 2, -2.0 * dg / n ** 2, dg / n ** 2)

    def taps(a, k, axis):
        lo = torch.cat([a.narrow(axis, 0, 1), a.narrow(axis, 0, a.shape[axis] - 1)], axis)
        hi = torch.cat([a.narrow(axis, 1, a.shape[axis] - 1), a.narrow(axis, a.shape[axis] - 1, 1)], axis)
        return k[0] * lo + k[1] * a + k[2] * hi

    def transpose(a, axis):
        b = k[1] * a
        last = a.shape[axis] - 1
        b.narrow(axis, 0, last).add_(k[0] * a.narrow(axis, 1, last))
        b.narrow(axis, 1, last).add_(k[2] * a.narrow(axis, 0, last))
        b.narrow(axis, 0, 1).add_(k[0] * a.narrow(axis, 0, 1))
        b.narrow(axis, last, 1).add_(k[2] * a.narrow(axis, last, 1))
        return b

    otf = taps(taps(T, k, 1), k, 0)
    signal = exposure * otf
    up_g = (signal - up(target)) * (2.0 / signal.numel())
    d_otf = taps(taps(T, k, 1), dk, 0) + taps(taps(T, dk, 1), k, 0)
    weight = (exposure * transpose(transpose(up_g, 0), 1)).reshape(-1, 1).expand(-1, ox.shape[2]).reshape(-1) / ox.shape[2]
    grad = torch.zeros(len(ids), dtype=torch.float64, device=dev)
    for ray, c, chord in chords():
        grad.index_add_(0, c, -weight[ray] * ray_t[ray] * chord)
    g_sigma = np.zeros(pos.shape[0])
    g_sigma[ids] = grad.cpu().numpy()
    return {"signal": signal.cpu().numpy(), "transmittance": T.cpu().numpy(), "g_sigma": g_sigma,
            "g_exposure": float((up_g * otf).sum()), "g_otf": float(exposure * (up_g * d_otf).sum())}


def _exact_stages(case, seed):
    gray, _, _, grid, step, pad, dens = _stage_inputs(case, seed)
    w, h = case["w"], case["h"]
    # Gelatin PSF inside the camera gate: 90 % of a 3-tap and 10 % of a 7-tap kernel, each pass
    # normalised by its taps inside the gate.
    ys, xs = np.flatnonzero(gray.any(1)), np.flatnonzero(gray.any(0))
    gate = (slice(ys[0], ys[-1] + 1), slice(xs[0], xs[-1] + 1))
    lin = gray[gate].astype(np.float64) / 255.0

    def blur(a, k, axis):
        r = len(k) // 2
        s, ws = np.zeros_like(a), np.zeros(a.shape[axis])
        for i, t in enumerate(k):
            o = i - r
            src = [slice(None), slice(None)]
            dst = [slice(None), slice(None)]
            n = a.shape[axis]
            if abs(o) >= n:
                continue
            dst[axis], src[axis] = slice(max(-o, 0), n - max(o, 0)), slice(max(o, 0), n - max(-o, 0))
            s[tuple(dst)] += t * a[tuple(src)]
            ws[dst[axis]] += t
        return s / (ws[:, None] if axis == 0 else ws[None, :])

    narrow, wide = (0.15, 0.70, 0.15), (0.03, 0.12, 0.20, 0.30, 0.20, 0.12, 0.03)
    heff = np.zeros((h, w))
    heff[gate] = 0.9 * blur(blur(lin, narrow, 1), narrow, 0) + 0.1 * blur(blur(lin, wide, 1), wide, 0)
    # Hann overlap blend.
    ntx, nty = -(-w // step), -(-h // step)

    def hann(t, nt, start, n):
        g = np.arange(start, start + n, dtype=np.float64)
        o = t * step
        wt = np.ones(n)
        if t + 1 < nt:
            u = np.clip((g - (o + step - pad)) / (2.0 * pad), 0.0, 1.0)
            wt = np.where(g >= o + step - pad, 0.5 + 0.5 * np.cos(np.pi * u), wt)
        if t > 0:
            u = np.clip((g - (o - pad)) / (2.0 * pad), 0.0, 1.0)
            wt = np.where(g < o + pad, 0.5 - 0.5 * np.cos(np.pi * u), wt)
        return wt

    acc, wacc = np.zeros((h, w)), np.zeros((h, w))
    for t, d in zip(grid, dens):
        wt = hann(t.ty, nty, t.y_start, t.th)[:, None] * hann(t.tx, ntx, t.x_start, t.tw)[None, :]
        box = (slice(t.y_start, t.y_start + t.th), slice(t.x_start, t.x_start + t.tw))
        acc[box] += wt * d
        wacc[box] += wt
    d_norm = acc / np.maximum(wacc, 1e-5)
    # Scanner OTF (clamp to edge) and the triangle-filter halving.
    pad_x = np.pad(d_norm, ((0, 0), (1, 1)), mode="edge")
    sharp = OTF_TAPS[0] * pad_x[:, :-2] + OTF_TAPS[1] * d_norm + OTF_TAPS[2] * pad_x[:, 2:]
    pad_y = np.pad(sharp, ((1, 1), (0, 0)), mode="edge")
    sharp = OTF_TAPS[0] * pad_y[:-2] + OTF_TAPS[1] * sharp + OTF_TAPS[2] * pad_y[2:]

    def shrink(a, m):  # along axis 0
        n = a.shape[0]
        ratio = n / m
        sr = max(ratio, 1.0)
        out = np.zeros((m,) + a.shape[1:])
        for o in range(m):
            c = (o + 0.5) * ratio
            lo = min(max(int(math.floor(c - sr)), 0), n - 1)
            hi = min(max(int(math.ceil(c + sr)), lo + 1), n)
            k = np.maximum(1.0 - np.abs((np.arange(lo, hi) - (c - 0.5)) / sr), 0.0)
            out[o] = (k / k.sum()) @ a[lo:hi]
        return out

    small = shrink(shrink(sharp, max(h // 2, 1)).T.copy(), max(w // 2, 1)).T
    return {"luma": None, "up": None, "heff": heff, "out": None, "d_norm": d_norm, "sharp": sharp, "small": small}
