"""The launch shape a fit picks by its sizes (one CTA per SM with many samples
kept, or three with fewer) changes no bit: fits with the shape left open against
the same fit with the three-CTA shape asked for, at the region counts where the
rule turns (one and four regions per SM), for region sizes on both sides of it, with
a region that a cluster shares, one that streams through the ring in either shape,
empty and unfitted ones, initialised and updated fits."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SMS = 152


@pytest.mark.parametrize("components", [8, 13])
@pytest.mark.parametrize("regions,size", [(1, 40000), (3, 300), (SMS, 700), (SMS + 1, 60), (SMS + 1, 900),
                                          (4 * SMS, 100), (4 * SMS, 1700), (4 * SMS + 1, 1700)])
def test_open_shape_equals_three_ctas(regions, size, components, cuda, pkg, abi, workloads):
    torch = cuda
    rng = np.random.default_rng(regions + size)
    counts = rng.integers(size // 2, size + size // 2, regions)
    if regions > 2:
        counts[0], counts[1], counts[2] = 0, 7, 30011  # empty, too few to fit, shared by a cluster
    w = workloads.mixture_samples(rng, counts, 1, 4, 2.0, 500.0, 1.0)
    d = torch.from_numpy(w["dirw"]).cuda()
    o = torch.from_numpy(w["offsets"].view(np.int32)).cuda()
    out = []
    for tuning in ({}, {"threads_per_cta": 128}):
        ctx = pkg.FitContext(abi.forced_iterations(6, num_initial_components=components), max_regions=regions)
        ctx.set_tuning(**tuning)
        ctx.fit(d, o, regions, abi.PG_FIT_INIT)
        ctx.fit(d, o, regions, abi.PG_FIT_UPDATE)
        ctx.sync()
        out.append(ctx.states(regions))
        ctx.close()
    assert np.array_equal(out[0].view(np.uint8), out[1].view(np.uint8))
