"""The record sort, which drops the slots without a region before its passes:
counts around a tile (4096), none, few and all slots valid, and region counts of
one, two and three digits, against a stable bucketing in index order."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 4095, 4096, 4097, 3 * 4096 + 511, 70001])
@pytest.mark.parametrize("share", [0.0, 0.004, 0.3, 1.0])
@pytest.mark.parametrize("R", [1, 256, 257, 65536, 65537])
def test_sort_keeps_the_valid_slots_in_order(n, share, R, cuda, pkg, abi, workloads):
    torch = cuda
    rng = np.random.default_rng(n + R)
    rec = np.zeros(n, dtype=workloads.RECORD_DTYPE)
    valid = rng.random(n) < share
    rec["flags"] = np.where(valid, rng.integers(0, R, size=n), rng.choice([R, 0xFFFFFFFF], size=n))
    rec["weight"] = np.arange(n, dtype=np.float32)
    order = np.flatnonzero(valid)
    order = order[np.argsort(rec["flags"][order], kind="stable")]
    want_off = np.searchsorted(rec["flags"][order], np.arange(R + 1, dtype=np.uint64))
    ctx = pkg.FitContext(abi.default_fit_config(), max_regions=1)
    d_rec = torch.from_numpy(rec.view(np.uint8).reshape(-1).copy()).cuda()
    d_sorted = torch.zeros(n * 40, dtype=torch.uint8, device="cuda")
    d_off = torch.zeros(R + 1, dtype=torch.int32, device="cuda")
    ctx.sort_samples(d_rec, n, R, d_sorted, d_off)
    ctx.sync()
    np.testing.assert_array_equal(d_off.cpu().numpy().view(np.uint32), want_off)
    assert d_sorted.cpu().numpy()[:order.size * 40].tobytes() == rec[order].tobytes()
    ctx.close()
