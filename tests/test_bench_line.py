"""The bench's line stays short enough to be kept whole: the headline's keys and one
value per other workload on stdout, their blocks on stderr."""
from __future__ import annotations

import json
import sys

from conftest import ROOT

sys.path.insert(0, str(ROOT))
import bench  # noqa: E402


def test_one_short_line(capsys):
    line = {"metric": bench.METRIC, "value": 141632.2, "unit": bench.UNIT, "ms_per_step": 1.9,
            "config": {"workload": bench.WORKLOAD, "note": "x" * 400}, "roofline": {"note": "x" * 600},
            "e2e": {"value": 119000.0, "unit": bench.UNIT}, "clocks": {"sm_mhz": 2070.0}, "gpu_launches": 40}
    blocks = {name: {"value": 12345.678901234 + i, "unit": "Mrays/s", "note": "y" * 2000} for i, name in
              enumerate(bench.BLOCKS)}
    blocks["guided"] = {"rows": ["z" * 6000]}  # no value of its own
    bench.print_line({**line, **blocks})
    out = capsys.readouterr()
    assert len(out.out.splitlines()) == 1 and len(out.out) < 3000
    got = json.loads(out.out)
    assert {k: got[k] for k in line} == line
    assert set(got["workloads"]) == set(bench.BLOCKS) - {"guided"}
    assert [next(iter(json.loads(x))) for x in out.err.splitlines()] == list(bench.BLOCKS)


def test_frame_launches():
    # 16 samples of 1280x720 are two waves of eight, 4 of 1920x1080 one wave, 3 of 4096x4096 three; each the camera
    # kernel, two launches per bounce and the pixel sums
    assert bench.frame_launches(1280 * 720, 16, 8) == 2 * 18
    assert bench.frame_launches(1920 * 1080, 4, 10) == 22
    assert bench.frame_launches(4096 * 4096, 3, 5) == 3 * 12
