"""A frame of many samples on a device with little memory left: traced with fewer
samples a wave, the image of the frame with room, and most of what was left still
free afterwards."""
from __future__ import annotations

import numpy as np
import pytest

from test_trace_gpu import render_gpu

pytestmark = pytest.mark.gpu

ROOM = 700 << 20  # below the 885 MB of an eight-sample wave, above the 110 MB of one sample


def test_frame_with_little_memory_left(cuda, pkg, abi):
    torch = cuda
    params = abi.render_params(spp=64, max_depth=4, seed=9)
    scenes = [pkg.Scene.cornell(1280, 720, ico_level=2) for _ in range(2)]
    want, _ = render_gpu(torch, scenes[0], params)
    scenes[0].close()
    render_gpu(torch, scenes[1], abi.render_params(spp=1, max_depth=1, seed=1))  # uploads the scene
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    image = torch.zeros(1280 * 720 * 3, dtype=torch.float32, device="cuda")
    held = []
    try:
        while (free := torch.cuda.mem_get_info()[0]) > ROOM + (64 << 20):
            held.append(torch.empty(min(free - ROOM, 8 << 30), dtype=torch.uint8, device="cuda"))
        assert ROOM // 2 < torch.cuda.mem_get_info()[0] < 885 << 20
        scenes[1].render(params, image)
        torch.cuda.synchronize()
        assert torch.cuda.mem_get_info()[0] > ROOM // 4
    finally:
        held.clear()
        torch.cuda.empty_cache()
    assert np.array_equal(image.cpu().numpy().reshape(want.shape).astype(np.float64), want)
    scenes[1].close()
