"""Fits whose launch shape is chosen on the device (both shapes launched, each behind
the kernel before it): calls of alternating sizes queued on one stream without a
wait between them, and a captured graph replayed with other offsets, give the bits of
the three-CTA shape asked for."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("components", [8, 13])
@pytest.mark.parametrize("per_sm", [1, 3])
def test_calls_in_a_row_and_replays(per_sm, components, cuda, pkg, abi, workloads):
    torch = cuda
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    R = per_sm * sms + 7  # between one and four regions per SM
    cfg = abi.forced_iterations(5, num_initial_components=components)
    sets = []
    for size in (40, 2600, 90, 1500):  # below and above the rule's line
        rng = np.random.default_rng(size + R)
        counts = rng.integers(size // 2, size + size // 2, R)
        counts[0], counts[1] = 0, 27000  # empty, shared by a cluster
        w = workloads.mixture_samples(rng, counts, 1, 4, 2.0, 500.0, 1.0)
        sets.append((torch.from_numpy(w["dirw"]).cuda(), torch.from_numpy(w["offsets"].view(np.int32)).cuda()))

    # the same calls with the three-CTA shape (a context's earlier fits decide which
    # regions a cluster shares), its states after each
    def three_ctas(calls):
        ctx = pkg.FitContext(cfg, max_regions=R)
        ctx.set_tuning(threads_per_cta=128)
        out = []
        for d, o in calls:
            ctx.fit(d, o, R, abi.PG_FIT_INIT)
            out.append(ctx.states(R).tobytes())
        ctx.close()
        return out

    # queued without a wait in between
    row = [sets[i] for i in (0, 1, 2, 3, 1, 0, 3, 2, 1)]
    want = three_ctas(row)
    for n in (len(row) - 1, len(row)):  # the last shape is one and the other
        ctx = pkg.FitContext(cfg, max_regions=R)
        stream = torch.cuda.Stream()
        for d, o in row[:n]:
            ctx.fit(d, o, R, abi.PG_FIT_INIT, stream=stream)
        stream.synchronize()
        assert ctx.states(R).tobytes() == want[n - 1]
        ctx.close()

    # one graph over buffers that take every set in turn
    want = three_ctas([sets[0], *sets])
    buf = torch.zeros(max(d.numel() for d, _ in sets), dtype=torch.float32, device="cuda")
    off = torch.zeros(R + 1, dtype=torch.int32, device="cuda")
    buf[:sets[0][0].numel()].copy_(sets[0][0].reshape(-1))
    off.copy_(sets[0][1])
    ctx = pkg.FitContext(cfg, max_regions=R)
    ctx.fit(buf, off, R, abi.PG_FIT_INIT)  # one-time setup
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        ctx.fit(buf, off, R, abi.PG_FIT_INIT, stream=torch.cuda.current_stream())
    for (d, o), ref in zip(sets, want[1:]):
        buf[:d.numel()].copy_(d.reshape(-1))
        off.copy_(o)
        g.replay()
        torch.cuda.synchronize()
        assert ctx.states(R).tobytes() == ref
    ctx.close()
