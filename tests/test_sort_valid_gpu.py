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


@pytest.mark.parametrize("n", [1, 255, 5000])
def test_records_off_the_8_byte_boundary(n, cuda, pkg, abi, workloads):
    """Sorted copies and updated mixtures do not depend on the buffer's alignment."""
    torch = cuda
    rng = np.random.default_rng(n)
    rec = np.zeros(n, dtype=workloads.RECORD_DTYPE)
    rec["position"] = rng.random((n, 3))
    d = rng.normal(size=(n, 3))
    rec["direction"] = d / np.linalg.norm(d, axis=1, keepdims=True)
    rec["weight"], rec["pdf"], rec["distance"] = rng.random(n), rng.uniform(0.1, 1, n), rng.uniform(0, 2, n)
    rec["flags"] = rng.choice([0, 1, 2, 3, 0xFFFFFFFF], size=n)
    got = []
    for off in (0, 4):
        buf = torch.zeros(n * 40 + 8, dtype=torch.uint8, device="cuda")
        buf[off:off + n * 40] = torch.from_numpy(rec.view(np.uint8).reshape(-1).copy()).cuda()
        ctx = pkg.FitContext(abi.default_fit_config(), max_regions=4)
        ctx.set_regions(2, np.array([0, 0, 0, 1, 1, 1], dtype=np.float32))
        out = torch.zeros(n * 40, dtype=torch.uint8, device="cuda")
        offsets = torch.zeros(5, dtype=torch.int32, device="cuda")
        ctx.sort_samples(buf[off:], n, 4, out, offsets)
        ctx.update(buf[off:], n)
        ctx.sync()
        got.append((out.cpu().numpy().tobytes(), offsets.cpu().numpy().tobytes(), ctx.states(4).tobytes()))
        ctx.close()
    assert got[0] == got[1]
