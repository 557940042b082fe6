"""The work that users of this framework have it do, as measurable cases.

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges, ``prepare(case, seed)``
makes what a caller holds before the call (a page on the device or in host memory, a mask, a trained
network), ``run(state)`` is one pass through the public entry points, ``work(case)`` the bytes and
operations that pass cannot do without and ``exact(case, seed)`` its 64-bit result where one can be
written down without the library.

Pages are contact-hole arrays as in ``synthetic.py``: jittered discs (square or staggered lattice)
with a Gaussian-blurred edge and read noise, rendered here with plain torch from the seed alone.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from imageprocessor_new_b200 import connected_components_stats, detect_centers, measure_cds, stack, warmstart

DTYPES = {"uint8": torch.uint8, "uint16": torch.uint16, "float32": torch.float32, "float64": torch.float64}

RADIAL = "gaussian,gradient,halfmax"
AREAS = "projection,half_area,half_area_min,half_area_min_avg"
TAILS = "tail_area,tail_area_norm,edge_area,foot_area,foot_area_ratio"


def listed():
    return [
        # One frame of a live camera: a small 8-bit image in host memory, library defaults (triangle
        # threshold, log-quadratic refinement). Latency of one call.
        dict(name="centers camera frame", kind="centers", h=256, w=320, pitch=16.0, d=7.0, sigma=1.0, stagger=False,
             dtype="uint8", threshold="triangle", refine="logquad", host=True, invert=False, area_max=200),
        # A square contact-hole page from a scanner's host buffer, edge refinement.
        dict(name="centers edges 1024", kind="centers", h=1024, w=1024, pitch=32.0, d=14.0, sigma=1.5, stagger=False,
             dtype="uint16", threshold="otsu", refine="edge_gradmoment", host=True, invert=False, area_max=400),
        # The full 8192 page already on the device, log-quadratic refinement of every hole.
        dict(name="centers page 8192", kind="centers", h=8192, w=8192, pitch=24.0, d=12.0, sigma=1.2, stagger=True,
             dtype="uint16", threshold="otsu", refine="logquad", host=False, invert=False, area_max=400),
        # A large panel in row bands with halos (global Otsu, keep rule, dedupe), ragged last band.
        dict(name="centers tiled panel", kind="tiled", h=15000, w=12001, pitch=20.0, d=10.0, sigma=1.0, stagger=False,
             dtype="uint16", refine="weighted", tile_h=4096, overlap=128, area_max=400),
        # Labels, statistics and centroids of a host mask of odd size, as cv2 users call it.
        dict(name="components 3000x2501", kind="components", h=3000, w=2501, pitch=14.0, d=8.0, sigma=1.0,
             stagger=True, connectivity=8),
        # A field too dense to threshold: Gaussian spots 1.4 FWHM apart in floats, peak seeds, every
        # output of a small result (contours, cells, masks).
        dict(name="cds dense spots", kind="cds", h=480, w=641, pitch=5.6, d=4.0, sigma=1.7, stagger=True, spots=True,
             dtype="float64", methods="gaussian,halfmax", seeds="peaks", invert=False, summary=False, area_max=50),
        # The 1024 contact-hole page from host memory with the Gaussian-fit methods and the full result.
        dict(name="cds contacts 1024", kind="cds", h=1024, w=1024, pitch=32.0, d=14.0, sigma=1.5, stagger=False,
             spots=False, dtype="uint16", methods="gaussian,logquad", seeds="threshold", invert=False, summary=False,
             area_max=400),
        # The headline measurement: the 8192 staggered page on the device, Gaussian-FWHM,
        # radial-gradient and half-height CDs of ~116k holes.
        dict(name="cds page 8192", kind="cds", h=8192, w=8192, pitch=24.0, d=12.0, sigma=1.2, stagger=True,
             spots=False, dtype="uint16", methods=RADIAL, seeds="threshold", invert=False, summary=True, area_max=400),
        # Dark holes on a bright 8-bit page: projection widths and the half-height areas.
        dict(name="cds areas 2048", kind="cds", h=2047, w=2050, pitch=24.0, d=12.0, sigma=1.2, stagger=True,
             spots=False, dtype="uint8", methods=AREAS, seeds="threshold", invert=True, summary=True, area_max=400),
        # The tail family's wide windows (light around every hole, down to its foot).
        dict(name="cds tails 1536", kind="cds", h=1536, w=1531, pitch=24.0, d=12.0, sigma=1.2, stagger=True,
             spots=False, dtype="uint16", methods=TAILS, seeds="threshold", invert=False, summary=True, area_max=400),
        # A stack of uneven pages: the cells of every image and their warm-started fits in one launch.
        dict(name="stack warm fits", kind="stack", images=6, h=2048, w=2048, pitch_lo=16.0, pitch_hi=40.0,
             dtype="uint16"),
        # One training step of the warm-start network (forward, backward, AdamW) at its batch size.
        dict(name="warm start training", kind="train", batch=4096),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["centers", "centers", "tiled", "components", "cds", "cds", "areas", "tails", "dense", "stack",
                       "train"])
    dtype = rng.choice(["uint8", "uint16", "uint16", "float32"])
    if kind in ("centers", "tiled", "components"):
        pitch = round(rng.uniform(14.0, 36.0), 2)
        shape = dict(pitch=pitch, d=round(pitch * rng.uniform(0.4, 0.55), 2), sigma=round(rng.uniform(0.8, 1.6), 2),
                     stagger=rng.random() < 0.5)
        if kind == "components":
            return dict(kind=kind, h=_log(rng, 200, 4000), w=_log(rng, 200, 4000), connectivity=rng.choice([4, 8]),
                        **shape)
        if kind == "tiled":
            tile = _log(rng, 512, 4096)
            return dict(kind=kind, h=_log(rng, 1500, 12000), w=_log(rng, 1000, 12000), dtype=dtype.replace("float32", "uint16"),
                        refine=rng.choice(["weighted", "logquad", "auto"]), tile_h=tile, overlap=min(128, tile // 4),
                        area_max=600, **shape)
        dtype = dtype.replace("float32", "uint16")
        invert = rng.random() < 0.3  # dark holes: the estimator that reads edges, not light
        return dict(kind=kind, h=_log(rng, 200, 8000), w=_log(rng, 200, 8000), dtype=dtype,
                    threshold="otsu",  # (the triangle's level passes noise specks on some pages)
                    refine="edge_gradmoment" if invert else rng.choice(["weighted", "logquad", "edge_gradmoment", "auto"]),
                    host=rng.random() < 0.4, invert=invert, area_max=600, **shape)
    if kind == "train":
        return dict(kind=kind, batch=8 * _log(rng, 64, 1024))
    if kind == "stack":
        lo = round(rng.uniform(16.0, 24.0), 2)
        return dict(kind=kind, images=rng.randint(2, 6), h=_log(rng, 512, 2048), w=_log(rng, 512, 2048), pitch_lo=lo,
                    pitch_hi=round(rng.uniform(lo + 4.0, 40.0), 2), dtype="uint16")
    if kind == "dense":
        pitch = round(rng.uniform(5.4, 8.0), 2)
        fwhm = pitch / rng.uniform(1.4, 1.8)
        return dict(kind="cds", h=_log(rng, 160, 900), w=_log(rng, 160, 900), pitch=pitch, d=round(fwhm, 2),
                    sigma=round(fwhm / 2.3548, 3),
                    stagger=True, spots=True, dtype=rng.choice(["float32", "float64"]), methods="gaussian,halfmax",
                    seeds="peaks", invert=False, summary=True, area_max=50)
    pitch = round(rng.uniform(16.0, 26.0 if kind == "tails" else 36.0), 2)
    most = {"cds": 4000, "areas": 2000, "tails": 1500}[kind]
    return dict(kind="cds", h=_log(rng, 200, most), w=_log(rng, 200, most), pitch=pitch,
                d=round(pitch * rng.uniform(0.42, 0.52), 2), sigma=round(rng.uniform(1.0, 1.5), 2),
                stagger=rng.random() < 0.5, spots=False, dtype=dtype,
                methods={"cds": rng.choice([RADIAL, "gaussian,logquad", "gradient,halfmax"]), "areas": AREAS,
                         "tails": TAILS}[kind],
                seeds="threshold", invert=rng.random() < 0.3, summary=True, area_max=900)


# ------------------------------------------------------------------------------------------ inputs

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(1_000_003 * int(seed) + 17)


def _light(h, w, pitch, d, sigma, stagger, spots, gen):
    """Light of the array at every pixel, one per hole: discs with a Gaussian-blurred edge, or Gaussian
    spots. Every lattice site has its own jitter and diameter; a pixel sums the sites around it. Holes
    cut by the page's edge are there with their centres on the page, without jitter, so that a page
    of a case holds the same number of holes whatever the seed."""
    rows, cols = int(h / pitch) + 6, int(w / pitch) + 7
    i = torch.arange(rows, device="cuda", dtype=torch.float32)[:, None]
    j = torch.arange(cols, device="cuda", dtype=torch.float32)[None, :]
    sy = ((i - 1.5) * pitch).expand(rows, cols)
    sx = (j - 2.5) * pitch + ((i % 2) * (0.5 * pitch) if stagger else 0.0 * i)
    edge = torch.minimum(torch.minimum(sx, w - 1 - sx), torch.minimum(sy, h - 1 - sy))
    inner = (edge >= 0.5 * d + 3.0 * sigma + 2.0).float() * (0.1 if spots else 1.0)
    jx = (torch.rand((rows, cols), device="cuda", generator=gen) - 0.5) * inner
    jy = (torch.rand((rows, cols), device="cuda", generator=gen) - 0.5) * inner
    rad = 0.5 * d * (1.0 + 0.1 * (torch.rand((rows, cols), device="cuda", generator=gen) - 0.5) * inner)
    # (Left out: holes that only just reach the edge, which noise would make whole or cut.)
    reach = 2.355 * sigma if spots else 0.5 * d
    there = ((edge >= (-2.0 * d if spots else 0.25 * d)) & ((edge - reach).abs() >= 1.0)).float()
    out = torch.empty((h, w), dtype=torch.float32, device="cuda")
    xs = torch.arange(w, device="cuda", dtype=torch.float32)[None, :]
    near = 2 if spots else 1
    for y0 in range(0, h, 1024):
        ys = torch.arange(y0, min(h, y0 + 1024), device="cuda", dtype=torch.float32)[:, None]
        acc = torch.zeros((ys.shape[0], w), dtype=torch.float32, device="cuda")
        for a in range(-near, near + 1):
            r = torch.floor(ys / pitch).long() + a + 2
            shift = (r % 2).float() * (0.5 * pitch) if stagger else torch.zeros_like(ys)
            for b in range(-near, near + 1):
                c = torch.floor((xs - shift) / pitch).long() + b + 3
                rr, cc = r.expand(c.shape).clamp(0, rows - 1), c.clamp(0, cols - 1)
                dx = xs - (sx[rr, cc] + jx[rr, cc])
                dy = ys - (sy[rr, cc] + jy[rr, cc])
                r2 = dx * dx + dy * dy
                if spots:
                    acc += there[rr, cc] * torch.exp(-0.5 * r2 / (sigma * sigma))
                else:
                    acc += 0.5 * there[rr, cc] * torch.erfc((torch.sqrt(r2) - rad[rr, cc]) / (math.sqrt(2.0) * sigma))
        out[y0:y0 + ys.shape[0]] = acc
    return out


def _page(case, seed, pitch=None, d=None):
    gen = _generator(seed)
    h, w = case["h"], case["w"]
    light = _light(h, w, case["pitch"] if pitch is None else pitch, case["d"] if d is None else d, case["sigma"],
                   case["stagger"], case.get("spots", False), gen)
    noise = torch.randn((h, w), dtype=torch.float32, device="cuda", generator=gen)
    dtype = case["dtype"]
    if case.get("spots"):
        return (20.0 + 50.0 * light + 2.5 * noise).to(DTYPES[dtype])
    level, contrast, read = (60.0, 150.0, 5.0) if dtype == "uint8" else (1000.0, 3000.0, 100.0)
    if case.get("invert"):
        level, contrast = level + contrast, -contrast
    page = level + contrast * light + read * noise
    if dtype.startswith("uint"):
        top = 255 if dtype == "uint8" else 65535
        return page.round_().clamp_(0, top).to(torch.int32).to(DTYPES[dtype])
    return page.to(DTYPES[dtype])


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        gen = _generator(seed)
        b = case["batch"]
        x = torch.randn((b, warmstart.IN), device="cuda", generator=gen).mul_(0.3).add_(0.4).to(torch.bfloat16)
        t = torch.randn((b, warmstart.OUT), device="cuda", generator=gen)
        return dict(kind=kind, net=warmstart.WarmStartNet(seed=int(seed) % (1 << 31)), x=x, xt=x.t().contiguous(), t=t,
                    weights=torch.ones(warmstart.OUT, device="cuda"))
    if kind == "stack":
        n = case["images"]
        images = []
        for i in range(n):
            pitch = case["pitch_lo"] + (case["pitch_hi"] - case["pitch_lo"]) * i / max(1, n - 1)
            images.append(_page(dict(case, sigma=1.2, stagger=i % 2 == 1), 1000 * int(seed) + i, pitch=pitch,
                                d=min(20.0, 0.5 * pitch)))
        return dict(kind=kind, stack=torch.stack([p.to(torch.int32) for p in images]).to(DTYPES[case["dtype"]]),
                    net=warmstart.WarmStartNet.load())
    if kind == "components":
        page = _page(dict(case, dtype="uint16"), seed)
        mask = (page.to(torch.int32) > 2500).to(torch.uint8) * 255
        return dict(kind=kind, mask=mask.cpu().numpy(), connectivity=case["connectivity"])
    page = _page(case, seed)
    if kind == "tiled":
        kw = dict(threshold="otsu", refine=case["refine"], tile_h=case["tile_h"], overlap=case["overlap"],
                  threshold_mode="global", area_max=case["area_max"])
    elif kind == "centers":
        kw = dict(threshold=case["threshold"], refine=case["refine"], invert=case["invert"],
                  area_max=case["area_max"])
    else:
        kw = dict(methods=tuple(case["methods"].split(",")), seeds=case["seeds"], invert=case["invert"],
                  summary_only=case["summary"], area_max=case["area_max"])
    # Host pages: camera and scanner buffers, and the result that carries the image with it.
    host = case.get("host", kind == "cds" and not case["summary"])
    return dict(kind=kind, page=page.cpu().numpy() if host else page, kw=kw)


# --------------------------------------------------------------------------------------- one pass

def _result(res):
    out = {"seeds": res.seeds_xy}
    for name, m in res.measurements.items():
        out[name] = {"centers": m.centers_xy, "contours": m.contours_xy, "metrics": m.metrics,
                     "status": np.ascontiguousarray(m.status).view(np.uint32)}
        if m.geometry and "edge_px" in m.geometry:
            out[name]["edges"] = m.geometry["edge_px"]
        out[name] = {k: v for k, v in out[name].items() if k == "metrics" or v.size}
    if hasattr(res, "cell_labels"):
        out.update(labels=res.cell_labels, areas=res.cell_areas_px2, boxes=res.boxes_xywh, rois=res.rois,
                   masks=res.masks, background=res.background_map, params=res.deblend_model["params"])
    return out


def run(state):
    kind = state["kind"]
    if kind in ("centers", "tiled"):
        return detect_centers(state["page"], backend="gpu", **state["kw"]).centers_xy
    if kind == "components":
        r = connected_components_stats(state["mask"], connectivity=state["connectivity"])
        return {"labels": r.labels, "stats": r.stats, "centroids": r.centroids}
    if kind == "cds":
        return _result(measure_cds(state["page"], backend="gpu", **state["kw"]))
    if kind == "stack":
        sc = stack.stack_cells(state["stack"])
        params, status, iterations, background, fallback = stack.initial_fits(state["stack"], sc, net=state["net"])
        return {"params": params, "status": status, "iterations": iterations, "background": background,
                "fallback": fallback, "boxes": sc.cells.boxes, "labels": sc.cells.voronoi}
    net = state["net"]
    loss = net.train_step(state["x"], state["xt"], state["t"], state["weights"], lr=1e-3)
    return {"loss": loss, "grads": {k: p.g for k, p in net.p.items()}, "weights": {k: p.w for k, p in net.p.items()}}


def work(case):
    kind = case["kind"]
    if kind == "train":
        b = case["batch"]
        params = warmstart.HID * warmstart.IN + warmstart.HID * warmstart.HID + warmstart.OUT * warmstart.HID
        flops = 2.0 * b * (2 * warmstart.HID * warmstart.IN + 3 * warmstart.HID * warmstart.HID
                           + 3 * warmstart.OUT * warmstart.HID)
        # The batch and its transpose, the targets, and the f32 weights with gradients and moments.
        return {"bytes": 2.0 * 2 * b * warmstart.IN + 4.0 * b * warmstart.OUT + 4.0 * 7 * params, "flops": flops}
    size = {"uint8": 1, "uint16": 2, "float32": 4, "float64": 8}
    px = float(case["h"]) * case["w"]
    if kind == "components":
        return {"bytes": px * (1 + 4), "flops": 0.0}
    if kind == "stack":
        px *= case["images"]
        cells = sum(case["h"] * case["w"] / (case["pitch_lo"] + (case["pitch_hi"] - case["pitch_lo"]) * i
                                             / max(1, case["images"] - 1)) ** 2 for i in range(case["images"]))
        # Labels out; per pixel about six Levenberg-Marquardt passes of 83 operations.
        return {"bytes": px * (2 + 4) + 64.0 * cells, "flops": px * 6 * 83 + cells * 0.66e6}
    holes = px / case["pitch"] ** 2
    page = px * size[case["dtype"]]
    if kind in ("centers", "tiled"):
        return {"bytes": page + 16.0 * holes, "flops": 0.0}
    methods = case["methods"].split(",")
    # Fits: about 13 + 5 x 10 Levenberg-Marquardt passes of 83 operations per pixel, then per method.
    flops = px * 63 * 83
    out = 0.0
    for m in methods:
        out += holes * 8 * 12
        if not case["summary"]:
            out += holes * 8 * 3 * 129
        if m in ("gradient", "halfmax"):
            flops += holes * 128 * 10 * (0.75 * case["pitch"]) * 32
        elif m.startswith("half"):
            flops += px * 16 * 16
        elif "tail" in m or "foot" in m or m == "edge_area":
            flops += px * 5.8 * 16 * 32
    if not case["summary"]:
        out += px * (4 + 4 + 8 + 8 + 1)
    return {"bytes": page + out, "flops": flops}


# ----------------------------------------------------------------------------------- 64-bit values

def _components_exact(case, seed):
    """Centroids of the mask's components in OpenCV's numbering, by label propagation in torch."""
    if case["connectivity"] != 8 or case["h"] * case["w"] > 9_000_000:
        return None
    mask = torch.from_numpy(prepare(case, seed)["mask"]).cuda() > 0
    h, w = mask.shape
    n = h * w
    label = torch.where(mask, torch.arange(n, 0, -1, device="cuda").view(h, w).double(), torch.zeros((), device="cuda").double())
    while True:  # the largest index of each component spreads over it
        grown = torch.nn.functional.max_pool2d(label[None, None], 3, 1, 1)[0, 0] * mask
        if torch.equal(grown, label):
            break
        label = grown
    inv = torch.unique(label.long(), return_inverse=True)[1].view(-1)
    k = int(inv.max()) + 1
    ys = torch.arange(h, device="cuda").view(h, 1).expand(h, w).reshape(-1)
    xs = torch.arange(w, device="cuda").view(1, w).expand(h, w).reshape(-1)
    block = (ys // 2) * ((w + 1) // 2) + xs // 2
    first = torch.full((k,), 1 << 62, device="cuda", dtype=torch.int64).scatter_reduce_(0, inv, block, "amin")
    has_zero = not bool(mask.all())
    if has_zero:
        first[0] = -1  # the background is label 0
    count = torch.bincount(inv, minlength=k)
    cx = torch.zeros(k, dtype=torch.int64, device="cuda").index_add_(0, inv, xs).double() / count
    cy = torch.zeros(k, dtype=torch.int64, device="cuda").index_add_(0, inv, ys).double() / count
    order = torch.argsort(first)
    return {"labels": None, "stats": None, "centroids": torch.stack([cx, cy], 1)[order].cpu().numpy()}


def _train_exact(case, seed):
    """The same step in 64 bits: the network reads the batch and its weights as bf16, as it is defined."""
    s = prepare(case, seed)
    w = {k: p.w.double().clone() for k, p in s["net"].p.items()}
    low = {k: w[k].to(torch.bfloat16).double() for k in ("w1", "w2", "w3")}
    x, t, b = s["x"].double(), s["t"].double(), case["batch"]
    z1 = x @ low["w1"].t() + w["b1"]
    h1 = z1.clamp_min(0)
    z2 = h1 @ low["w2"].t() + w["b2"]
    h2 = z2.clamp_min(0)
    y = h2 @ low["w3"].t() + w["b3"]
    dy = 2.0 * (y - t) / b
    dh2 = (dy @ low["w3"]) * (z2 > 0)
    dh1 = (dh2 @ low["w2"]) * (z1 > 0)
    g = {"w1": dh1.t() @ x, "b1": dh1.sum(0), "w2": dh2.t() @ h1, "b2": dh2.sum(0), "w3": dy.t() @ h2, "b3": dy.sum(0)}
    new = {}
    for k in g:
        m, v = 0.1 * g[k], 0.001 * g[k] ** 2
        decay = 1e-4 if k.startswith("w") else 0.0
        new[k] = w[k] - 1e-3 * ((m / 0.1) / ((v / 0.001).sqrt() + 1e-8) + decay * w[k])
    # The biases start at zero, so their first AdamW step is the learning rate times the gradient's sign,
    # which bf16 decides where a gradient is near zero: no value to be near to.
    new.update(b1=None, b2=None, b3=None)
    return {"loss": (((y - t) ** 2).sum() / b).view(1), "grads": g, "weights": new}


def exact(case, seed):
    """Centres and CDs end where a stop rule of the iterative fit leaves them (64 bits throughout): they
    have no value apart from the method itself. Centroids and the network's step have one."""
    if case["kind"] == "components":
        return _components_exact(case, seed)
    if case["kind"] == "train":
        return _train_exact(case, seed)
    return None
