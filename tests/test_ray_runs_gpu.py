"""How a caller's rays are dealt to warps changes no hit: ray counts where the rays per
warp turn (one, five and six, 31 and 32 a warp of the resident ones), with no ray, every
ray, the first of each 32 and every other ray starting behind its origin (tmin < 0,
traced after the others), against the CPU twin."""
from __future__ import annotations

import numpy as np
import pytest

from test_trace_gpu import SCENES, dev, host, make_rays, tracer  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("behind", ["none", "all", "first", "half"])
@pytest.mark.parametrize("per_warp,off", [(0, 1), (0, 5), (1, 0), (1, 1), (5, 0), (5, 1), (31, 0), (31, 1), (32, 1)])
def test_runs(per_warp, off, behind, cuda, pkg, abi, tracer):
    torch = cuda
    warps = 32 * torch.cuda.get_device_properties(0).multi_processor_count
    n = per_warp * warps + off
    sc = SCENES["plates"](pkg)
    exp = sc.export()
    rays = make_rays(abi, np.random.default_rng(n), exp, max(n, 64))[-n:].copy()
    i = np.arange(n)
    neg = {"none": i < 0, "all": i >= 0, "first": i % 32 == 0, "half": i % 2 == 1}[behind]
    rays["tmin"][neg] = -0.5
    d_rays = dev(torch, rays)
    hits = torch.zeros(n * abi.HIT_DTYPE.itemsize, dtype=torch.uint8, device="cuda")
    occ = torch.full((n,), 7, dtype=torch.int32, device="cuda")
    sc.trace_closest(d_rays, n, hits)
    sc.trace_any(d_rays, n, occ)
    torch.cuda.synchronize()
    assert np.array_equal(host(hits, abi.HIT_DTYPE).view(np.uint32), tracer.closest(exp, rays).view(np.uint32))
    assert np.array_equal(occ.cpu().numpy().view(np.uint32), tracer.any(exp, rays))
