"""The calls whose speed matters to a program that uses this library, as cases.

A case is a dict of plain values.  `prepare` makes what a program holds before
the call (scenes, contexts, networks, sample buffers on the GPU), `run` is one
pass through the public entry points, `work` the bytes and operations that the
pass cannot do without, and `exact` the outputs in 64-bit arithmetic written
out here with torch alone, where they have a closed definition.

Kinds of case:

* render   - pg_render: plain wavefront path tracing (next-event estimation with
             MIS) of the Cornell box or the glossy plates scene.
* train    - pg_render as a guided training pass: guided by every region's
             mixture and recording guiding samples.
* trace    - pg_trace_closest and pg_trace_any over a caller's ray buffer.
* update   - PathGuiding's update from the tracer's record buffer: the first
             pass and one stepwise pass, with parallax, split and merge.
* fit      - pg_fit_regions at fixed iterations, then pg_pack_vmm_theta.
* infer, grad, learn - the surrogate: mixtures at positions, loss and gradient
             of a batch, one online training pass.
* cache    - frames that grow the irradiance cache.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import __graft_entry__ as entry

pkg = entry.load_package()
abi = pkg.abi
guiding = entry.load_submodule("guiding")

SLOTS = 16            # record slots per pixel
CACHE_ENTRIES = 16384
INVALID = -1          # PG_INVALID_REGION as a signed word
BOX = (-2.0, -1.0, -1.5, 2.0, 3.0, 1.5)  # the surrogate's scene box


def listed():
    return [
        # an interactive preview: one sample per pixel of a small window
        {"name": "render_preview", "kind": "render", "scene": "cornell", "detail": 3, "width": 160, "height": 90,
         "spp": 1, "depth": 8},
        # a frame of the Cornell box as the tracer's benchmark renders it
        {"name": "render_cornell", "kind": "render", "scene": "cornell", "detail": 5, "width": 1280, "height": 720,
         "spp": 16, "depth": 8},
        # the plates scene with its million-triangle occluder, full HD
        {"name": "render_plates", "kind": "render", "scene": "plates", "detail": 707, "width": 1920, "height": 1080,
         "spp": 4, "depth": 10},
        # a training pass in the middle of guided rendering, odd image size
        {"name": "train_guided", "kind": "train", "scene": "plates", "detail": 353, "width": 1001, "height": 563,
         "spp": 4, "depth": 10, "splits": 10},
        # a host renderer's own ray buffer: incoherent rays through the occluder
        {"name": "trace_rays", "kind": "trace", "scene": "plates", "detail": 353, "rays": 2000003},
        # the guiding update of a small image over few regions
        {"name": "update_small", "kind": "update", "splits": 6, "pixels": 14400},
        # the guiding update of a full-HD training pass over the default 4096 regions
        {"name": "update_large", "kind": "update", "splits": 12, "pixels": 2073600},
        # the CPU-runnable fit: equal regions, 8 components
        {"name": "fit_plain", "kind": "fit", "regions": 64, "median": 16384, "sigma": 0.0, "components": 8,
         "iterations": 20, "lobes": 4},
        # the batched fit: 4096 uneven regions, 16 components
        {"name": "fit_batched", "kind": "fit", "regions": 4096, "median": 2048, "sigma": 1.0, "components": 16,
         "iterations": 20, "lobes": 6},
        # the surrogate's mixtures for a buffer of shading points
        {"name": "infer_points", "kind": "infer", "positions": 1048573},
        # the surrogate's online training over the records of one pass
        {"name": "learn_pass", "kind": "learn", "records": 1 << 20, "batch": 65536},
        # prepare frames that grow the irradiance cache
        {"name": "cache_frames", "kind": "cache", "scene": "cornell", "detail": 5, "width": 640, "height": 360,
         "frames": 4, "depth": 8},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _image(rng, most):
    """Width and height of an image of up to `most` pixels, odd ones among them."""
    pixels = math.exp(rng.uniform(math.log(160 * 90), math.log(most)))
    aspect = rng.uniform(1.0, 2.0)
    return max(8, int(math.sqrt(pixels * aspect))), max(8, int(math.sqrt(pixels / aspect)))


def draw(rng):
    kind = rng.choice(["render", "render", "train", "trace", "update", "fit", "fit", "infer", "learn", "grad",
                       "cache"])
    if kind in ("render", "train"):
        scene = rng.choice(["cornell", "plates"])
        w, h = _image(rng, 1280 * 720 if kind == "render" else 1001 * 563)
        c = {"kind": kind, "scene": scene, "detail": rng.randint(2, 5) if scene == "cornell" else _log_int(rng, 20, 353),
             "width": w, "height": h, "spp": _log_int(rng, 1, 16 if kind == "render" else 4),
             "depth": rng.randint(3, 10)}
        if kind == "train":
            c["splits"] = rng.randint(4, 12)
        return c
    if kind == "trace":
        scene = rng.choice(["cornell", "plates"])
        return {"kind": kind, "scene": scene,
                "detail": rng.randint(2, 6) if scene == "cornell" else _log_int(rng, 20, 353),
                "rays": _log_int(rng, 1000, 2000003)}
    if kind == "update":
        return {"kind": kind, "splits": rng.randint(3, 12), "pixels": _log_int(rng, 4000, 1000000)}
    if kind == "fit":
        regions = _log_int(rng, 1, 4096)
        median = _log_int(rng, 256, max(257, min(65536, 4000000 // regions)))
        return {"kind": kind, "regions": regions, "median": median, "sigma": round(rng.uniform(0.0, 1.0), 2),
                "components": rng.randint(2, 16), "iterations": rng.randint(5, 20), "lobes": rng.randint(1, 6)}
    if kind == "infer":
        return {"kind": kind, "positions": _log_int(rng, 100, 1048573)}
    if kind == "learn":
        return {"kind": kind, "records": _log_int(rng, 20000, 1 << 20), "batch": 1 << rng.randint(13, 16)}
    if kind == "grad":
        return {"kind": kind, "records": _log_int(rng, 100, 65536)}
    w, h = _image(rng, 640 * 360)
    return {"kind": kind, "scene": "cornell", "detail": rng.randint(3, 5), "width": w, "height": h,
            "frames": rng.randint(1, 4), "depth": rng.randint(3, 8)}


# --- inputs -------------------------------------------------------------------

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _scene(case, seed):
    if case["scene"] == "cornell":
        return pkg.Scene.cornell(case.get("width", 64), case.get("height", 36), ico_level=case["detail"])
    return pkg.Scene.plates(case.get("width", 64), case.get("height", 36), occluder_grid=case["detail"],
                            seed=1 + seed % 1000)


def _sphere(g, *shape):
    d = torch.randn(*shape, 3, device="cuda", generator=g)
    return d / d.norm(dim=-1, keepdim=True)


def _around(g, mu, kappa):
    """One von Mises-Fisher draw per row around mu (n, 3) with kappa (n,)."""
    u = torch.rand(mu.shape[0], device="cuda", generator=g, dtype=torch.float64)
    phi = 2.0 * math.pi * torch.rand(mu.shape[0], device="cuda", generator=g, dtype=torch.float64)
    k, m = kappa.double(), mu.double()
    w = (1.0 + torch.log(u + (1.0 - u) * torch.exp(-2.0 * k)) / k).clamp(-1.0, 1.0)
    s = torch.sqrt((1.0 - w * w).clamp_min(0.0))
    flip = m[:, 0].abs() > 0.9
    a = torch.zeros_like(m)
    a[:, 0] = (~flip).double()
    a[:, 1] = flip.double()
    t = torch.linalg.cross(m, a)
    t = t / t.norm(dim=1, keepdim=True)
    b = torch.linalg.cross(m, t)
    d = (s * torch.cos(phi))[:, None] * t + (s * torch.sin(phi))[:, None] * b + w[:, None] * m
    return (d / d.norm(dim=1, keepdim=True)).float()


def _lobe_directions(g, region, regions, most_lobes, kappa_lo, kappa_hi):
    """A direction per sample from its region's mixture of 1 to most_lobes lobes."""
    lobes = torch.randint(1, most_lobes + 1, (regions,), device="cuda", generator=g)
    mu = _sphere(g, regions, most_lobes)
    kappa = torch.exp(math.log(kappa_lo) + math.log(kappa_hi / kappa_lo) *
                      torch.rand(regions, most_lobes, device="cuda", generator=g))
    out = []
    for part in region.split(1 << 21):  # bounds the float64 temporaries
        pick = (torch.rand(part.shape[0], device="cuda", generator=g) * lobes[part]).long()
        pick = torch.minimum(pick, lobes[part] - 1)
        out.append(_around(g, mu[part, pick], kappa[part, pick]))
    return torch.cat(out)


def _lognormal(g, n, sigma):
    return torch.exp(sigma * torch.randn(n, device="cuda", generator=g))


def _prepare_fit(case, seed):
    g = _generator(seed)
    R = case["regions"]
    counts = torch.exp(math.log(case["median"]) + case["sigma"] * torch.randn(R, device="cuda", generator=g))
    counts = counts.round().clamp(64, 262144).long()
    offsets = torch.zeros(R + 1, dtype=torch.int32, device="cuda")
    offsets[1:] = counts.cumsum(0).int()
    region = torch.repeat_interleave(torch.arange(R, device="cuda"), counts)
    n = region.shape[0]
    dirw = torch.empty(n, 4, device="cuda")
    dirw[:, :3] = _lobe_directions(g, region, R, case["lobes"], 2.0, 2000.0)
    dirw[:, 3] = _lognormal(g, n, 1.0)
    cfg = abi.forced_iterations(case["iterations"], num_initial_components=case["components"])
    theta = torch.zeros(R, abi.VMM_THETA_DTYPE.itemsize // 4, device="cuda")
    return {"ctx": pkg.FitContext(cfg, max_regions=R), "dirw": dirw, "offsets": offsets, "R": R, "theta": theta}


def _region_centres(splits, box):
    """Region boxes as the context makes them: what a tracer's positions fall into."""
    ctx = pkg.FitContext(abi.default_fit_config(), max_regions=1 << splits)
    ctx.set_regions(splits, np.asarray(box, dtype=np.float32))
    boxes = torch.from_numpy(ctx.region_aabbs()).cuda()
    ctx.close()
    return boxes


def _prepare_update(case, seed):
    """A tracer's record buffer: 16 slots per pixel; a path's first vertices
    lie in regions that follow the image, its later ones anywhere; unused and
    dropped slots are INVALID."""
    g = _generator(seed)
    P, splits = case["pixels"], case["splits"]
    R = 1 << splits
    box = (0.0, 0.0, 0.0, 4.0, 4.0, 4.0)
    boxes = _region_centres(splits, box)
    rec = torch.zeros(P * SLOTS, 10, device="cuda")
    flags = rec.view(torch.int32)[:, 9]
    flags.fill_(INVALID)
    popularity = torch.exp(torch.randn(R, device="cuda", generator=g))
    cdf = popularity.cumsum(0) / popularity.sum()
    vertices = torch.randint(0, 9, (P,), device="cuda", generator=g)  # recorded vertices of each pixel's path
    slot = torch.arange(SLOTS, device="cuda")
    used = (slot[None, :] < vertices[:, None]).reshape(-1)
    used &= torch.rand(P * SLOTS, device="cuda", generator=g) < 0.9
    at = used.nonzero()[:, 0]
    n = at.shape[0]
    u = torch.rand(n, device="cuda", generator=g)
    first = (at % SLOTS) < 2
    u = torch.where(first, ((at // SLOTS).float() / P + 0.02 * u).clamp(max=0.999999), u)
    region = torch.searchsorted(cdf, u).clamp(max=R - 1)
    lo, hi = boxes[region, :3], boxes[region, 3:]
    rec[at, 0:3] = lo + torch.rand(n, 3, device="cuda", generator=g) * (hi - lo)
    rec[at, 3:6] = _lobe_directions(g, region, R, 6, 2.0, 2000.0)
    rec[at, 6] = _lognormal(g, n, 1.0)
    rec[at, 7] = torch.rand(n, device="cuda", generator=g) * 0.5 + 0.05
    dist = torch.exp(torch.rand(n, device="cuda", generator=g) * math.log(1000.0)) * 0.1
    rec[at, 8] = torch.where(torch.rand(n, device="cuda", generator=g) < 0.1, torch.zeros_like(dist), dist)
    flags[at] = region.int()
    ctx = pkg.FitContext(abi.default_fit_config(), max_regions=R)
    ctx.set_split_merge()
    theta = torch.zeros(R, abi.VMM_THETA_DTYPE.itemsize // 4, device="cuda")
    return {"ctx": ctx, "records": rec, "n": P * SLOTS, "splits": splits, "box": np.asarray(box, dtype=np.float32),
            "theta": theta, "R": R}


def _guide_states(splits, box, seed):
    """A trained guide as a program restores it: 4 to 12 lobes per region."""
    rng = np.random.default_rng(seed)
    R = 1 << splits
    s = np.zeros(R, dtype=abi.STATE_DTYPE)
    k = rng.integers(4, 13, R)
    on = np.arange(16)[None, :] < k[:, None]
    w = rng.gamma(1.0, size=(R, 16)) * on
    s["weight"] = w / w.sum(1, keepdims=True)
    mu = rng.normal(size=(R, 16, 3))
    mu[..., 1] = np.abs(mu[..., 1])
    mu /= np.linalg.norm(mu, axis=-1, keepdims=True)
    s["mu_x"], s["mu_y"], s["mu_z"] = mu[..., 0], mu[..., 1], mu[..., 2]
    kap = np.exp(rng.uniform(np.log(2.0), np.log(200.0), (R, 16)))
    s["kappa"] = np.where(on, kap, 0.0)
    s["r"] = np.where(on, 1.0 / np.tanh(kap) - 1.0 / kap, 0.0)
    s["norm"] = np.where(on, kap / (2.0 * np.pi * -np.expm1(-2.0 * kap)), 0.0)
    s["e_min2k"] = np.where(on, np.exp(-2.0 * kap), 1.0)
    s["distance"] = np.exp(rng.uniform(np.log(0.5), np.log(10.0), (R, 16)))
    s["dist_sum_w"] = 1.0
    box = np.asarray(box, dtype=np.float64)
    s["parallax_mean"] = box[:3] + (box[3:] - box[:3]) * rng.random((R, 3))
    s["last_parallax_mean"] = s["parallax_mean"]
    s["k"], s["sample_weight"], s["num_samples"], s["total_num_samples"] = k, 1000.0, 1000.0, 1000
    s["flags"] = abi.PG_STATE_FITTED
    return s


def _prepare_render(case, seed):
    sc = _scene(case, seed)
    P = case["width"] * case["height"]
    st = {"scene": sc, "image": torch.zeros(P * 3, device="cuda")}
    fields = dict(spp=case["spp"], max_depth=case["depth"], seed=1 + seed % 100000)
    if case["kind"] == "train":
        box = np.array(sc.get_scene_size(), dtype=np.float32)
        ctx = pkg.FitContext(abi.default_fit_config(), max_regions=1 << case["splits"])
        ctx.set_regions(case["splits"], box)
        ctx.set_states(_guide_states(case["splits"], box, seed))
        st["guide"] = ctx
        st["records"] = torch.zeros(P * SLOTS, 10, device="cuda")
        fields.update(use_guiding=1, record_samples=1)
    st["params"] = abi.render_params(**fields)
    return st


def _prepare_trace(case, seed):
    g = _generator(seed)
    sc = _scene(case, seed)
    n = case["rays"]
    lo = torch.tensor(sc.get_scene_size()[:3], device="cuda")
    hi = torch.tensor(sc.get_scene_size()[3:], device="cuda")
    rays = torch.empty(n, 8, device="cuda")
    rays[:, 0:3] = lo + (hi - lo) * torch.rand(n, 3, device="cuda", generator=g)
    rays[:, 3] = 1e-3
    rays[:, 4:7] = _sphere(g, n)
    rays[:, 7] = 1e6
    return {"scene": sc, "rays": rays, "n": n, "hits": torch.zeros(n, 4, device="cuda"),
            "occluded": torch.zeros(n, dtype=torch.int32, device="cuda")}


# --- the surrogate's model, for its inputs and its exact values

_LAYERS = ((64, 112), (64, 64), (64, 64), (80, 64))


def _theta(seed):
    """Network weights somewhere in training: He-uniform layers, a small
    output layer and spread initial means, a little off the initialisation."""
    rng = np.random.default_rng(seed)
    parts = []
    for i, (o, c) in enumerate(_LAYERS):
        w = rng.uniform(-1.0, 1.0, (o, c)) * math.sqrt(6.0 / (99 if i == 0 else c)) * (0.2 if i == 3 else 1.0)
        if i == 0:
            w[:, 99:] = 0.0
        b = 0.02 * rng.normal(size=o)
        if i == 3:
            m = rng.normal(size=(16, 3))
            c4 = b.reshape(16, 5)
            c4[:, 1:4] += m / np.linalg.norm(m, axis=1, keepdims=True)
            c4[:, 4] += math.log(8.0)
        parts += [w.reshape(-1), b.reshape(-1)]
    return np.concatenate(parts).astype(np.float32)


def _surrogate_records(g, n):
    lo, hi = torch.tensor(BOX[:3], device="cuda"), torch.tensor(BOX[3:], device="cuda")
    rec = torch.zeros(n, 10, device="cuda")
    rec[:, 0:3] = lo + (hi - lo) * torch.rand(n, 3, device="cuda", generator=g)
    lights = lo + (hi - lo) * torch.rand(4, 3, device="cuda", generator=g)
    to = lights[torch.randint(0, 4, (n,), device="cuda", generator=g)] - rec[:, 0:3]
    dist = to.norm(dim=1, keepdim=True).clamp_min(1e-6)
    rec[:, 3:6] = _around(g, to / dist, torch.full((n,), 50.0, device="cuda"))
    rec[:, 6] = _lognormal(g, n, 1.0)
    rec[:, 7] = 1.0
    rec[:, 8] = dist[:, 0]
    return rec


def _prepare_surrogate(case, seed):
    g = _generator(seed)
    kind = case["kind"]
    net = pkg.Surrogate(BOX, batch=case.get("batch", 65536))
    theta = _theta(seed)
    net.set_params(theta)
    st = {"net": net, "theta": theta}
    if kind == "infer":
        n = case["positions"]
        lo, hi = torch.tensor(BOX[:3], device="cuda"), torch.tensor(BOX[3:], device="cuda")
        st["positions"] = lo + (hi - lo) * torch.rand(n, 3, device="cuda", generator=g)
        st["mixtures"] = torch.zeros(n, 16, 5, device="cuda")
    else:
        n = case["records"]
        st["records"] = _surrogate_records(g, n)
        st["grad"] = torch.zeros(abi.MLP_PARAMS, device="cuda")
    st["n"] = n
    return st


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("render", "train"):
        st = _prepare_render(case, seed)
    elif kind == "cache":
        st = {"scene": _scene(case, seed), "seed": 1 + seed % 100000}
    elif kind == "trace":
        st = _prepare_trace(case, seed)
    elif kind == "update":
        st = _prepare_update(case, seed)
    elif kind == "fit":
        st = _prepare_fit(case, seed)
    else:
        st = _prepare_surrogate(case, seed)
    st["case"] = dict(case)
    return st


# --- one pass -----------------------------------------------------------------

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "render":
        state["image"].zero_()
        state["scene"].render(state["params"], state["image"], stats=False)
        return {"image": state["image"]}
    if kind == "train":
        state["image"].zero_()
        state["scene"].render(state["params"], state["image"], guide=state["guide"], records_dev=state["records"],
                              stats=False)
        rec = state["records"]
        return {"image": state["image"], "geometry": rec[:, :6], "weight": rec[:, 6:9],
                "region": rec.view(torch.int32)[:, 9]}
    if kind == "trace":
        state["scene"].trace_closest(state["rays"], state["n"], state["hits"])
        state["scene"].trace_any(state["rays"], state["n"], state["occluded"])
        return {"hits": state["hits"][:, :3], "primitive": state["hits"].view(torch.int32)[:, 3],
                "occluded": state["occluded"]}
    if kind == "update":
        ctx = state["ctx"]
        ctx.set_regions(state["splits"], state["box"])
        ctx.update(state["records"], state["n"], state["theta"])   # the first training pass
        ctx.update(state["records"], state["n"], state["theta"])   # a stepwise one
        return _mixtures(state["theta"])
    if kind == "fit":
        ctx = state["ctx"]
        ctx.fit(state["dirw"], state["offsets"], state["R"], abi.PG_FIT_INIT)
        ctx.pack_vmm_theta(state["R"], state["theta"])
        return _mixtures(state["theta"])
    if kind == "infer":
        state["net"].infer(state["positions"], state["n"], state["mixtures"])
        m = state["mixtures"]
        return {"weight": m[:, :, 0], "mean": m[:, :, 1:4], "kappa": m[:, :, 4]}
    if kind == "grad":
        loss = state["net"].loss_grad(state["records"], state["n"], state["grad"])
        return {"loss": loss, "grad": state["grad"]}
    if kind == "learn":
        loss = state["net"].train(state["records"], state["n"])
        return {"loss": loss, "params": state["net"].params()}
    entries = guiding.prepare_irradiance_cache(state["scene"], frames=case["frames"], max_depth=case["depth"],
                                               seed=state["seed"], cfg=_cache_config())
    table = np.zeros(CACHE_ENTRIES, dtype=abi.IC_ENTRY_DTYPE)  # one shape, however many entries the frames made
    table[:len(entries)] = entries
    flat = table.view(np.float32).reshape(CACHE_ENTRIES, -1)
    return {"count": len(entries), "entries": flat[:, :11], "gradients": flat[:, 12:],
            "updates": table["num_updates"].astype(np.int64)}


def _cache_config():
    cfg = abi.IrradianceCacheConfig()
    pkg.library().pg_default_irradiance_cache_config(ctypes.byref(cfg))
    cfg.capacity = CACHE_ENTRIES
    return cfg


def _mixtures(theta):
    """A packed mixture buffer, field by field."""
    lobes = theta[:, :160].view(-1, 16, 10)
    return {"mean": lobes[:, :, 0:3], "shape": lobes[:, :, 3:6], "placement": lobes[:, :, 6:10],
            "weight": theta[:, 160:176], "position": theta[:, 176:179], "used": theta.view(torch.int32)[:, 179]}


# --- what a pass cannot do without ----------------------------------------------

def _triangles(case):
    return 20 * 4 ** case["detail"] + 12 if case["scene"] == "cornell" else 2 * case["detail"] ** 2 + 8


def _ray_flops(case):
    """Box tests down a four-wide tree and two triangle tests, per ray."""
    return 2 * 40 + max(1.0, math.log(_triangles(case), 4)) * 4 * 18


def work(case):
    kind = case["kind"]
    if kind in ("render", "train", "cache"):
        P = case["width"] * case["height"]
        passes = case["spp"] if kind != "cache" else case["frames"]
        bounces = min(case["depth"], 4)  # a path of these scenes has about that many vertices
        rays = 2.0 * P * passes * bounces
        b = 12.0 * P + 48.0 * _triangles(case) + (40.0 * SLOTS * P if kind == "train" else 0.0)
        return {"bytes": b, "flops": rays * (_ray_flops(case) + 150)}
    if kind == "trace":
        n = case["rays"]
        return {"bytes": n * (32.0 + 16 + 4) + 48.0 * _triangles(case), "flops": 2.0 * n * _ray_flops(case)}
    if kind == "update":
        slots = SLOTS * case["pixels"]
        valid = 0.9 * 4 * case["pixels"]
        # flags of every slot and the valid records, each pass, and the mixtures
        return {"bytes": 2 * (4.0 * slots + 40.0 * valid + 720.0 * 2 ** case["splits"]),
                "flops": 2 * valid * 8 * 20 * 10.0}
    if kind == "fit":
        n = case["regions"] * case["median"] * math.exp(0.5 * case["sigma"] ** 2)
        return {"bytes": 16.0 * n + 720.0 * case["regions"],
                "flops": n * case["iterations"] * case["components"] * 18.0}
    per = 2.0 * sum(o * c for o, c in _LAYERS)
    if kind == "infer":
        return {"bytes": case["positions"] * (12.0 + 320.0), "flops": case["positions"] * per}
    return {"bytes": case["records"] * 40.0 + 4.0 * abi.MLP_PARAMS,
            "flops": case["records"] * (3.0 * per - 2.0 * _LAYERS[0][0] * _LAYERS[0][1])}


# --- 64-bit values ----------------------------------------------------------------

def exact(case, seed):
    kind = case["kind"]
    if kind == "fit":
        return _exact_fit(case, prepare(case, seed))
    if kind in ("infer", "grad", "learn"):
        return _exact_surrogate(case, prepare(case, seed))
    # images, records, hits and cache entries follow from hit or miss decisions at
    # each vertex: there is no 64-bit value that they come near path by path
    return None


def _kappa_of(r):
    return (3.0 * r - r ** 3) / (1.0 - r * r)


def _exact_fit(case, st):
    """MAP-EM for mixtures of von Mises-Fisher lobes (weight prior 0.01, mean
    cosine prior 0 with weight 1, kappa from the mean resultant length)."""
    K, R = case["components"], case["regions"]
    f = st["dirw"].double()
    off = st["offsets"].long()
    n = (off[1:] - off[:-1]).double()
    # spherical Fibonacci means, in single precision
    mu0 = np.zeros((K, 3))
    for i in range(K):
        phi = np.float32(2.0 * math.pi * float(np.float32(i) / np.float32(1.618033988749895)))
        z = np.float32(1.0) - (np.float32(2.0) * np.float32(i) + np.float32(1.0)) / np.float32(K)
        th = np.arccos(z)
        mu0[i] = (np.sin(th) * np.cos(phi), np.sin(th) * np.sin(phi), np.cos(th))
    mu = torch.from_numpy(mu0).cuda()[None].repeat(R, 1, 1)
    kappa = torch.full((R, K), 5.0, dtype=torch.float64, device="cuda")
    weight = torch.full((R, K), 1.0 / K, dtype=torch.float64, device="cuda")
    region = torch.repeat_interleave(torch.arange(R, device="cuda"), off[1:] - off[:-1])
    max_r = 1.0 / math.tanh(50000.0) - 1.0 / 50000.0
    wpn = 1.0 / (float(np.float32(0.01)) * K + 1.0)
    prior = float(np.float32(0.01)) * wpn
    fits = n > 2 * K
    for _ in range(case["iterations"]):
        norm = kappa / (2.0 * math.pi * -torch.expm1(-2.0 * kappa))
        norm = torch.where(kappa > 0, norm, torch.full_like(norm, 1.0 / (4.0 * math.pi)))
        S = torch.zeros(R, K, 4, dtype=torch.float64, device="cuda")
        W = torch.zeros(R, dtype=torch.float64, device="cuda")
        for lo in range(0, f.shape[0], 1 << 20):
            x, r = f[lo:lo + (1 << 20)], region[lo:lo + (1 << 20)]
            cos = (torch.einsum("nkc,nc->nk", mu[r], x[:, :3]) - 1.0).clamp(max=0.0)
            v = weight[r] * norm[r] * torch.exp(kappa[r] * cos)
            p = v.sum(1)
            ok = p > 1e-8
            gam = torch.where(ok[:, None], v * (x[:, 3] / p)[:, None], torch.zeros_like(v))
            S.index_add_(0, r, torch.cat([gam[:, :, None] * x[:, None, :3], gam[:, :, None]], 2))
            W.index_add_(0, r, torch.where(ok, x[:, 3], torch.zeros_like(p)))
        length = S[:, :, :3].norm(dim=2)
        w = S[:, :, 3] / W[:, None] * wpn + prior
        m = torch.where(length[:, :, None] > 0, S[:, :, :3] / length[:, :, None], mu)
        ns = n[:, None] * w
        rp = (length / S[:, :, 3] * ns) / (ns + 1.0)
        rp = torch.where(rp < max_r, rp, torch.full_like(rp, max_r))
        k = _kappa_of(rp)
        k = torch.where(k < 1e-3, torch.zeros_like(k), k)
        keep = fits[:, None]
        mu = torch.where(keep[:, :, None], m, mu)
        kappa = torch.where(keep, k, kappa)
        weight = torch.where(keep, w, weight)
    norm = kappa / (2.0 * math.pi * -torch.expm1(-2.0 * kappa))
    mean = torch.zeros(R, 16, 3, dtype=torch.float64, device="cuda")
    shape = torch.zeros(R, 16, 3, dtype=torch.float64, device="cuda")
    pi = torch.zeros(R, 16, dtype=torch.float64, device="cuda")
    mean[:, :K], pi[:, :K] = mu, weight
    shape[:, :K] = torch.stack([kappa, norm, torch.exp(-2.0 * kappa)], 2)
    return {"mean": mean, "shape": shape, "placement": None, "weight": pi, "position": None, "used": None}


def _unpack(theta):
    out, at = [], 0
    for o, c in _LAYERS:
        out += [theta[at:at + o * c].view(o, c), theta[at + o * c:at + o * c + o]]
        at += o * c + o
    return out


def _outputs(parts, pos):
    """Raw outputs of the network: Fourier features of the position in the box
    (normalised in single precision), three ReLU layers, a linear one."""
    lo = torch.tensor(BOX[:3], device="cuda")
    inv = 1.0 / (torch.tensor(BOX[3:], device="cuda") - lo)
    x = ((pos - lo) * inv).double()
    i = torch.arange(48, device="cuda")
    a = math.pi * (2.0 ** (i // 3).double()) * x[:, i % 3]
    h = torch.cat([torch.stack([torch.sin(a), torch.cos(a)], 2).flatten(1), x,
                   torch.zeros(x.shape[0], 13, dtype=torch.float64, device="cuda")], 1)
    for layer in range(4):
        h = h @ parts[2 * layer].T + parts[2 * layer + 1]
        if layer < 3:
            h = torch.relu(h)
    return h.view(-1, 16, 5)


def _mixture_of(o):
    pi = torch.softmax(o[:, :, 0], 1)
    mu = o[:, :, 1:4] / o[:, :, 1:4].norm(dim=2, keepdim=True)
    return pi, mu, torch.exp(o[:, :, 4].clamp(-4.0, 9.0))


def _loss(parts, rec):
    pi, mu, kappa = _mixture_of(_outputs(parts, rec[:, 0:3]))
    cos = torch.einsum("njc,nc->nj", mu, rec[:, 3:6].double())
    lf = torch.log(kappa / (2.0 * math.pi)) - torch.log(-torch.expm1(-2.0 * kappa)) + kappa * (cos - 1.0)
    w = rec[:, 6].double()
    return -(w * torch.logsumexp(torch.log(pi) + lf, 1)).sum(), w.sum()


def _gradient(theta, rec):
    theta = theta.detach().requires_grad_(True)
    parts = _unpack(theta)
    total = sum(float(r[:, 6].double().sum()) for r in rec.split(1 << 16))
    loss = 0.0
    for r in rec.split(1 << 16):
        part, _ = _loss(parts, r)
        (part / total).backward(retain_graph=True)
        loss += float(part.detach()) / total
    return loss, theta.grad


def _exact_surrogate(case, st):
    theta = torch.from_numpy(st["theta"]).cuda().double()
    if case["kind"] == "infer":
        with torch.no_grad():
            m = [_mixture_of(_outputs(_unpack(theta), p)) for p in st["positions"].split(1 << 16)]
        return {"weight": torch.cat([a[0] for a in m]), "mean": torch.cat([a[1] for a in m]),
                "kappa": torch.cat([a[2] for a in m])}
    if case["kind"] == "grad":
        loss, g = _gradient(theta, st["records"])
        return {"loss": loss, "grad": g}
    m, v, losses = torch.zeros_like(theta), torch.zeros_like(theta), []
    for t, rec in enumerate(st["records"].split(case["batch"]), 1):
        loss, g = _gradient(theta, rec)
        losses.append(loss)
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        theta = theta.detach() - 1e-3 * (m / (1 - 0.9 ** t)) / (torch.sqrt(v / (1 - 0.999 ** t)) + 1e-8)
    return {"loss": sum(losses) / len(losses), "params": theta.cpu().numpy()}
