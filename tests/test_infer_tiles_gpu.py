"""Surrogate inference in tiles of 128 positions: every count and output address
gives, bit for bit, the first rows of one large call (counts around a tile and more
tiles than are in flight; outputs off the 16-byte boundary, which take another way
out of shared memory), and writes nothing past them."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
BOX = np.array([-2.0, -1.0, -1.5, 2.0, 3.0, 1.5], dtype=np.float32)
ROW = 80  # floats of a mixture


@pytest.mark.parametrize("n", [1, 127, 128, 129, 255, 4097, 304 * 128 * 2 + 77])
@pytest.mark.parametrize("off", [0, 1, 2])
def test_rows_do_not_depend_on_the_call(n, off, cuda, pkg, abi):
    torch = cuda
    most = 304 * 128 * 2 + 1000
    rng = np.random.default_rng(3)
    pos = torch.from_numpy((BOX[:3] + (BOX[3:] - BOX[:3]) * rng.random((most, 3))).astype(np.float32)).cuda()
    net = pkg.Surrogate(BOX)
    want = torch.empty(most * ROW, dtype=torch.float32, device="cuda")
    net.infer(pos, most, want)
    out = torch.full((off + n * ROW + 8,), -7.0, dtype=torch.float32, device="cuda")
    net.infer(pos, n, out[off:])
    torch.cuda.synchronize()
    assert torch.equal(out[off:off + n * ROW].view(torch.int32), want[:n * ROW].view(torch.int32))
    assert bool((out[:off] == -7.0).all()) and bool((out[off + n * ROW:] == -7.0).all())
    net.close()
