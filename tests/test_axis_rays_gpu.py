"""Rays whose slab distances are not ordinary numbers, through the warp walk of
pg_trace_closest / pg_trace_any: bit for bit the CPU twin's hits and those of the
one-ray-per-lane walk (pg_trace_closest_counted).  Directions with one and two zero
components of either sign (0 x infinity where the origin lies on a box plane), none
at all, tiny and huge ones; origins on vertex coordinates, far away and infinite;
tmin at the hit's distance and one ulp to either side.  A counted render's image is
the plain render's."""
from __future__ import annotations

import numpy as np
import pytest

from test_trace_gpu import SCENES, dev, host, make_rays, render_gpu, tracer  # noqa: F401

pytestmark = pytest.mark.gpu


def axis_rays(abi, rng, exp, n):
    rays = make_rays(abi, rng, exp, n)
    v = exp["pos"].reshape(-1, 3)
    org, d = rays["org"], rays["dir"]
    for axis in range(3):  # half of the origins' coordinates are a vertex's
        on = rng.random(n) < 0.5
        org[on, axis] = v[rng.integers(0, len(v), int(on.sum())), axis]
    zeros = rng.integers(0, 8, n)  # bit i: component i is zero (7: no direction)
    for axis in range(3):
        z = (zeros >> axis) & 1 == 1
        d[z, axis] = np.where(rng.random(int(z.sum())) < 0.5, 0.0, -0.0).astype(np.float32)
    scale = np.ones(n, dtype=np.float32)
    scale[::13], scale[1::13], scale[2::13] = 1e-33, 1e-41, 1e37
    d *= scale[:, None]
    some = rng.integers(0, n, n // 16)
    d[some, rng.integers(0, 3, len(some))] = rng.choice(
        np.array([1e-42, -1e-38, 1e-30, 3e38, np.inf, -np.inf, np.nan], dtype=np.float32), len(some))
    far = rng.integers(0, n, n // 64)
    org[far, rng.integers(0, 3, len(far))] = rng.choice(np.array([3e38, -1e30, np.inf], dtype=np.float32), len(far))
    return rays


@pytest.mark.parametrize("name", sorted(SCENES))
def test_hits_of_axis_parallel_rays(name, cuda, pkg, abi, tracer):
    torch = cuda
    sc = SCENES[name](pkg)
    exp = sc.export()
    n = 200003
    rays = axis_rays(abi, np.random.default_rng(21), exp, n)
    want = tracer.closest(exp, rays)
    hit = want["prim"] != 0xFFFFFFFF
    assert hit.mean() > 0.05
    # intervals that begin at the hit, just before it and just behind it
    again = rays.copy()
    t = want["t"]
    step = np.random.default_rng(22).integers(-1, 2, n)
    edge = np.where(step < 0, np.nextafter(t, np.float32(0)), np.where(step > 0, np.nextafter(t, np.float32(np.inf)), t))
    again["tmin"] = np.where(hit, edge, rays["tmin"])
    for r in (rays, again):
        d_rays = dev(torch, r)
        hits, counted = (torch.zeros(n * abi.HIT_DTYPE.itemsize, dtype=torch.uint8, device="cuda") for _ in range(2))
        occ, nodes, tris = (torch.full((n,), 7, dtype=torch.int32, device="cuda") for _ in range(3))
        sc.trace_closest(d_rays, n, hits)
        sc.trace_any(d_rays, n, occ)
        sc.trace_closest_counted(d_rays, n, counted, nodes, tris)
        torch.cuda.synchronize()
        w = tracer.closest(exp, r)
        got = host(hits, abi.HIT_DTYPE)
        bad = np.where((got.view(np.uint32).reshape(-1, 4) != w.view(np.uint32).reshape(-1, 4)).any(axis=1))[0]
        assert bad.size == 0, f"{bad.size} hits differ; first {bad[:3]}: {r[bad[:3]]} gpu {got[bad[:3]]} cpu {w[bad[:3]]}"
        assert np.array_equal(host(counted, abi.HIT_DTYPE).view(np.uint32), got.view(np.uint32))
        assert np.array_equal(occ.cpu().numpy().view(np.uint32), tracer.any(exp, r))


@pytest.mark.parametrize("seed", range(4))
def test_counted_render_is_the_plain_one(seed, cuda, pkg, abi):
    sc = pkg.Scene.cornell(1280, 720, ico_level=5)
    a, b = (render_gpu(cuda, sc, abi.render_params(spp=2, max_depth=8, seed=seed, flags=f))[0]
            for f in (0, abi.PG_RENDER_COUNT_WORK))
    assert np.array_equal(a, b)
