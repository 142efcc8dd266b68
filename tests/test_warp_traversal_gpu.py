"""The warp-cooperative traversal of a caller's rays (pg_trace_closest, pg_trace_any)
bit for bit against the CPU twin, at the ray counts where warps are partly filled
(one ray, below and above a refill, a warp, a block, every warp's run uneven) and
for the intervals it treats apart: tmin < 0 (traced alone), tmin 0, tmax infinite,
empty, NaN."""
from __future__ import annotations

import numpy as np
import pytest

from test_trace_gpu import SCENES, dev, host, make_rays, tracer  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 7, 9, 32, 33, 127, 129, 4099, 155655])
@pytest.mark.parametrize("name", ["cornell", "plates"])
def test_ray_counts_and_intervals(name, n, cuda, pkg, abi, tracer):
    torch = cuda
    sc = SCENES[name](pkg)
    exp = sc.export()
    rays = make_rays(abi, np.random.default_rng(n), exp, max(n, 64))[-n:].copy()
    rays["tmin"][1::5] = -0.75
    rays["tmin"][2::5] = 0.0
    rays["tmax"][3::7] = np.inf
    rays["tmax"][4::11] = np.nan
    d_rays = dev(torch, rays)
    d_hits = torch.zeros(n * abi.HIT_DTYPE.itemsize, dtype=torch.uint8, device="cuda")
    d_occ = torch.full((n,), 7, dtype=torch.int32, device="cuda")
    sc.trace_closest(d_rays, n, d_hits)
    sc.trace_any(d_rays, n, d_occ)
    torch.cuda.synchronize()
    got, want = host(d_hits, abi.HIT_DTYPE), tracer.closest(exp, rays)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    assert np.array_equal(d_occ.cpu().numpy().view(np.uint32), tracer.any(exp, rays))
