"""States whose lanes past their component count hold something (set by a caller):
split and merge by teams of CTAs reads as many lanes as one CTA does - states and
statistics equal bit for bit, without a fit before it that would reset the lanes,
and a lane past the active ones (a multiple of four) changes no component."""
from __future__ import annotations

import numpy as np
import pytest

from test_guide_gpu import dev
from test_split_merge_teams_gpu import lobes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 4, 7, 8, 12, 15])
@pytest.mark.parametrize("sizes", [[1100, 2047, 40, 8100], [40] * 700 + [7500, 8100]], ids=["few", "many"])
def test_lanes_past_the_components(sizes, k, cuda, pkg, abi):
    torch = cuda
    R, o = len(sizes), np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint32)
    rng = np.random.default_rng(k)
    samples = lobes(rng, sum(sizes), 24)
    d, p, off = (dev(torch, a) for a in (samples[0], samples[1], o))
    cfg = abi.default_fit_config()
    cfg.num_initial_components = k
    out = {}
    active = (k + 3) // 4 * 4
    for stale in (False, True):
        for threshold in (0, 0xFFFFFFFF):
            ctx = pkg.FitContext(cfg, max_regions=R)
            sm = abi.default_split_merge_config()
            sm.min_samples_for_splitting = sm.min_samples_for_post_split_fitting = 0
            sm.cluster_threshold = threshold
            ctx.set_split_merge(sm)
            ctx.fit(d, off, R)
            st = ctx.states(R)
            if stale:  # another mixture's components
                for name, v in (("weight", 0.4), ("mu_x", 0.6), ("mu_z", 0.8), ("kappa", 40.0), ("r", 0.975),
                                ("norm", 40.0 / (2 * np.pi)), ("e_min2k", 0.0)):
                    st[name][:, active:] = v
                ctx.set_states(st)
            ctx.split_merge(d, p, off, R)
            ctx.sync()
            out[stale, threshold] = ctx.states(R), ctx.extras(R)
            ctx.close()
    for stale in (False, True):
        for a, b in zip(out[stale, 0], out[stale, 0xFFFFFFFF]):
            assert a.tobytes() == b.tobytes()
    for name in ("chi2_div", "cov"):
        assert np.array_equal(out[True, 0][1][name][:, :k], out[False, 0][1][name][:, :k])
    assert np.array_equal(out[True, 0][1]["em_iterations"], out[False, 0][1]["em_iterations"])
