"""Leaves of more than four triangles, which the builder makes only at its depth
limit: triangles along the axes at distances that shrink by 36, so each split peels
one off, around a bundle that is left over.  With up to 15 in a leaf the warp walk
takes it in rounds of four; with more the scene's nodes are not packed and rays go
one per lane.  Hits bit for bit the CPU twin's; a frame in waves is the frame one
sample at a time."""
from __future__ import annotations

import numpy as np
import pytest

from test_trace_gpu import dev, host, render_gpu, tracer  # noqa: F401

pytestmark = pytest.mark.gpu

SCENE = """<scene version="0.5.0">
  <sensor type="perspective">
    <float name="fov" value="45"/>
    <transform name="toWorld"><lookAt origin="0, 0, 3" target="0, 0, 0" up="0, 1, 0"/></transform>
  </sensor>
  <shape type="obj"><string name="filename" value="m.obj"/>
    <bsdf type="diffuse"><rgb name="reflectance" value="0.6, 0.5, 0.4"/></bsdf></shape>
  <shape type="sphere"><point name="center" x="0" y="2" z="3"/><float name="radius" value="0.5"/>
    <emitter type="area"><rgb name="radiance" value="5, 5, 5"/></emitter></shape>
</scene>
"""


def deep_scene(pkg, folder, bundle):
    rng = np.random.default_rng(bundle)
    tris = []
    for axis in range(3):
        for i in range(20):
            c = np.zeros(3)
            c[axis] = 1e6 * 36.0 ** -i
            h = 0.2 * c[axis]
            tris.append(c + [[-h, -h, -h], [h, -h, h], [0, h, 0]])
    for _ in range(bundle):
        a, b = rng.uniform(0.2, 1.0, 2)
        tris.append(np.array([[-a, -b, -0.3], [a, -b, 0.3], [rng.uniform(-a, a), b, 0.0]]))
    v = np.array(tris, dtype=np.float32).reshape(-1, 3)
    (folder / "m.obj").write_text("".join(f"v {x!r} {y!r} {z!r}\n" for x, y, z in v.tolist()) +
                                  "".join(f"f {i + 1} {i + 2} {i + 3}\n" for i in range(0, len(v), 3)))
    (folder / "s.xml").write_text(SCENE)
    return pkg.Scene.load(folder / "s.xml", 64, 48)


@pytest.mark.parametrize("bundle", [5, 8, 13, 15, 16, 21])
def test_leaves_at_the_depth_limit(bundle, tmp_path, cuda, pkg, abi, tracer):
    torch = cuda
    sc = deep_scene(pkg, tmp_path, bundle)
    exp = sc.export()
    assert exp["nodes"]["count"].max() == bundle
    rng = np.random.default_rng(3)
    n = 30011
    rays = np.zeros(n, dtype=abi.RAY_DTYPE)
    rays["org"] = rng.normal(size=(n, 3)) * rng.choice([0.3, 3.0, 1e4], size=(n, 1))
    d = rng.normal(size=(n, 3)) * 0.4 - rays["org"]
    rays["dir"] = d / np.linalg.norm(d, axis=1, keepdims=True)
    rays["tmin"] = rng.choice(np.array([0.0, 1e-3, -1.0], dtype=np.float32), n)
    rays["tmax"] = rng.choice(np.array([1e30, 3.0], dtype=np.float32), n)
    want = tracer.closest(exp, rays)
    assert (want["prim"] >= 60).mean() > 0.1 and len(np.unique(want["prim"])) > bundle  # the bundle's among them
    d_rays = dev(torch, rays)
    hits = torch.zeros(n * abi.HIT_DTYPE.itemsize, dtype=torch.uint8, device="cuda")
    occ = torch.full((n,), 7, dtype=torch.int32, device="cuda")
    sc.trace_closest(d_rays, n, hits)
    sc.trace_any(d_rays, n, occ)
    torch.cuda.synchronize()
    assert np.array_equal(host(hits, abi.HIT_DTYPE).view(np.uint32), want.view(np.uint32))
    assert np.array_equal(occ.cpu().numpy().view(np.uint32), tracer.any(exp, rays))
    frames = [render_gpu(torch, sc, abi.render_params(spp=8, max_depth=4, seed=2, flags=f))[0]
              for f in (0, abi.PG_RENDER_TIME_STAGES, abi.PG_RENDER_COUNT_WORK)]
    assert frames[0].any() and np.array_equal(frames[0], frames[1]) and np.array_equal(frames[0], frames[2])
