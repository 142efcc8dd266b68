"""Renders that trace several samples of every pixel in one wave against the same
render one sample at a time (which stage timing runs): images and ray counts equal
bit for bit, for tiny and odd images, one-bounce paths, waves of unequal size
(1024x768 pixels, 11 samples: more paths than a wave holds) and a guide."""
from __future__ import annotations

import numpy as np
import pytest

from test_trace_gpu import render_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,spp,depth", [(1, 1, 3, 4), (5, 3, 7, 1), (33, 17, 16, 8), (161, 91, 2, 64), (1024, 768, 11, 5)])
def test_waves_equal_single_samples(w, h, spp, depth, cuda, pkg, abi):
    sc = pkg.Scene.cornell(w, h, ico_level=3)
    wave, st = render_gpu(cuda, sc, abi.render_params(spp=spp, max_depth=depth, seed=5))
    one, st1 = render_gpu(cuda, sc, abi.render_params(spp=spp, max_depth=depth, seed=5, flags=abi.PG_RENDER_TIME_STAGES))
    assert np.array_equal(wave, one)
    assert (st.extension_rays, st.shadow_rays, st.paths) == (st1.extension_rays, st1.shadow_rays, st1.paths)


def test_guided_wave_equals_single_samples(cuda, pkg, abi):
    torch = cuda
    sc = pkg.Scene.cornell(64, 36, ico_level=3)
    ctx = pkg.FitContext(abi.default_fit_config(), max_regions=64)
    ctx.set_regions(6, np.array(sc.info().aabb, dtype=np.float32))
    rec = torch.zeros(64 * 36 * 16 * 40, dtype=torch.uint8, device="cuda")
    render_gpu(torch, sc, abi.render_params(spp=8, max_depth=8, seed=1, record_samples=1), guide=ctx, records=rec)
    ctx.update(rec, 64 * 36 * 16)
    images = [render_gpu(torch, sc, abi.render_params(spp=6, max_depth=8, seed=2, use_guiding=1, flags=f), guide=ctx)[0]
              for f in (0, abi.PG_RENDER_TIME_STAGES)]
    assert images[0].any() and np.array_equal(images[0], images[1])
    ctx.close()
