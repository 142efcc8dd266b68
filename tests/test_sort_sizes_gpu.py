"""The record sort on both sides of the count from which slots without a region are
dropped before the passes, for region counts whose ids take one, two and three digits
and for those that a sentinel id would take a digit more: sorted records and offsets
against numpy's stable order, few, most and all slots valid, none at all."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R", [1, 256, 257, 65536])
@pytest.mark.parametrize("n", [4097, 1 << 21, (1 << 21) + 4097])
@pytest.mark.parametrize("share", [0.0, 0.3, 1.0])
def test_offsets_and_order(share, n, R, cuda, pkg, abi):
    torch = cuda
    rng = np.random.default_rng(n + R)
    flags = rng.integers(0, R, n).astype(np.uint32)
    flags[rng.random(n) >= share] = rng.choice(np.array([R, R + 1, 0xFFFFFFFF], dtype=np.uint32))
    words = torch.arange(n, dtype=torch.int32, device="cuda")[:, None].repeat(1, 10)  # a record's words: its slot
    words[:, 9] = torch.from_numpy(flags.view(np.int32)).cuda()
    ctx = pkg.FitContext(abi.default_fit_config(), max_regions=1)
    out = torch.full((n + 1, 10), -7, dtype=torch.int32, device="cuda")
    off = torch.zeros(R + 1, dtype=torch.int32, device="cuda")
    ctx.sort_samples(words, n, R, out, off)
    ctx.sync()
    order = np.flatnonzero(flags < R)
    order = order[np.argsort(flags[order], kind="stable")]
    got = out.cpu().numpy()
    assert np.array_equal(got[:len(order), 0], order) and (got[len(order):] == -7).all()
    assert np.array_equal(got[:len(order), 9].view(np.uint32), flags[order])
    assert np.array_equal(off.cpu().numpy(), np.searchsorted(flags[order], np.arange(R + 1)))
    ctx.close()
