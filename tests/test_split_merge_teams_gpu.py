"""Regions that a team of CTAs takes over (long ones from the start, others after
many EM iterations) against the same regions on one CTA each, which is what a
cluster_threshold of 2^32 - 1 asks for: states and statistics equal bit for bit.
Sizes around the teams' thresholds, a batch of a team (12 trips of 128 samples)
and a group of chains (32); few regions and more regions than SMs."""
from __future__ import annotations

import numpy as np
import pytest

from test_guide_gpu import dev

pytestmark = pytest.mark.gpu


def lobes(rng, n, k):
    """Directions around k axes of different widths, and their weights and pdfs."""
    axis = rng.normal(size=(k, 3))
    d = axis[rng.integers(0, k, n)] + rng.normal(size=(n, 3)) * rng.choice([0.05, 0.3, 1.0], size=(n, 1))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return np.column_stack([d, rng.uniform(0.1, 4.0, n)]).astype(np.float32), rng.uniform(0.05, 2.0, n).astype(np.float32)


def run(torch, pkg, abi, sizes, samples, K, **knobs):
    R, o = len(sizes), np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint32)
    cfg = abi.default_fit_config()
    cfg.num_initial_components = K
    cfg.rel_ll_threshold = -1e30  # every refit takes all its iterations
    ctx = pkg.FitContext(cfg, max_regions=R)
    sm = abi.default_split_merge_config()
    sm.min_samples_for_splitting = sm.min_samples_for_post_split_fitting = 0
    for k, v in knobs.items():
        setattr(sm, k, v)
    ctx.set_split_merge(sm)
    d, p, off = (dev(torch, a) for a in (samples[0], samples[1], o))
    for _ in range(2):
        ctx.fit(d, off, R)
        ctx.split_merge(d, p, off, R)
    ctx.sync()
    out = ctx.states(R), ctx.extras(R)
    ctx.close()
    return out


@pytest.mark.parametrize("K", [3, 8, 13])
@pytest.mark.parametrize("sizes", [[1, 31, 33, 1023, 1100, 1535, 1536, 1537, 2047, 3100, 4097, 6999, 8100],
                                   [40] * 700 + [7, 96, 2500, 6100, 7500, 8100, 8190]], ids=["few", "many"])
def test_teams_give_the_bits_of_one_cta(sizes, K, cuda, pkg, abi):
    samples = lobes(np.random.default_rng(K), sum(sizes), 24)
    team = run(cuda, pkg, abi, sizes, samples, K)
    alone = run(cuda, pkg, abi, sizes, samples, K, cluster_threshold=0xFFFFFFFF)
    assert team[1]["em_iterations"].max() >= 100  # more than one CTA keeps a region for
    for a, b in zip(team, alone):
        assert a.tobytes() == b.tobytes()
