"""A sort and a guiding update that find too little device memory return an error, and
smaller calls of the same context after them find their buffers again."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LARGE, SMALL = 24 << 20, 5000  # 16 B of sort buffers a record: 403 MB
ROOM = 250 << 20


def test_small_calls_after_a_failed_large_one(cuda, pkg, abi):
    torch = cuda
    rng = np.random.default_rng(1)
    rec = np.zeros((SMALL, 10), dtype=np.float32)
    rec[:, :3] = rng.random((SMALL, 3))
    d = rng.normal(size=(SMALL, 3))
    rec[:, 3:6] = d / np.linalg.norm(d, axis=1, keepdims=True)
    rec[:, 6:9] = rng.uniform(0.1, 1.0, (SMALL, 3))
    rec[:, 9] = rng.integers(0, 4, SMALL).astype(np.uint32).view(np.float32)
    small = torch.from_numpy(rec).cuda()
    large = torch.zeros((LARGE, 10), dtype=torch.float32, device="cuda")
    large[:, 9] = -1.0  # no region
    out = torch.zeros((SMALL, 10), dtype=torch.float32, device="cuda")
    off = torch.zeros(5, dtype=torch.int32, device="cuda")

    def context():
        ctx = pkg.FitContext(abi.default_fit_config(), max_regions=4)
        ctx.set_regions(2, np.array([0, 0, 0, 1, 1, 1], dtype=np.float32))
        ctx.sort_samples(small, SMALL, 4, out, off)
        ctx.update(small, SMALL)
        ctx.sync()
        return ctx, (out.cpu().numpy().tobytes(), off.cpu().numpy().tobytes(), ctx.states(4).tobytes())

    ctx, want = context()
    ctx.update(small, SMALL)
    ctx.sync()
    again = ctx.states(4).tobytes()
    ctx.close()
    ctx, got = context()
    assert got == want
    torch.cuda.empty_cache()
    held = []
    try:
        while (free := torch.cuda.mem_get_info()[0]) > ROOM + (64 << 20):
            held.append(torch.empty(min(free - ROOM, 8 << 30), dtype=torch.uint8, device="cuda"))
        for call in (lambda: ctx.sort_samples(large, LARGE, 4, None, off), lambda: ctx.update(large, LARGE)):
            with pytest.raises(pkg.PathGuideError):
                call()
    finally:
        held.clear()
        torch.cuda.empty_cache()
    out.zero_()
    ctx.sort_samples(small, SMALL, 4, out, off)
    ctx.update(small, SMALL)
    ctx.sync()
    assert (out.cpu().numpy().tobytes(), off.cpu().numpy().tobytes()) == want[:2]
    assert ctx.states(4).tobytes() == again
    ctx.close()
