"""The launches of pg_split_merge when a CUDA call fails, on the host: its object
file linked with a stand-in for the CUDA runtime (split_merge_launch_harness.cpp).
Whichever call fails, the call returns an error, starts nothing once a shape was
refused, and leaves no side stream that the caller's stream does not wait for."""
from __future__ import annotations

import ctypes
import subprocess
from pathlib import Path

import pytest

import __graft_entry__ as entry
from conftest import ROOT

CALLER, SIDE = 1, (10, 11)


@pytest.fixture(scope="module")
def passes(pkg, tmp_path_factory):
    entry.build()
    build = entry.load_submodule("build")
    so = tmp_path_factory.mktemp("launch") / "launch.so"
    subprocess.run(["g++", "-std=c++17", "-fPIC", "-shared", "-Wl,-Bsymbolic", f"-I{ROOT / 'include'}", f"-I{build.CSRC}",
                    f"-I{Path(build.NVCC).resolve().parents[1] / 'include'}",
                    str(ROOT / "tests" / "split_merge_launch_harness.cpp"), str(build.BUILD / "pg_splitmerge.cu.o"),
                    "-o", str(so)], check=True)
    lib = ctypes.CDLL(str(so))

    def run(calls=1, fail=-1, cluster_size=0, regions=300):
        log, queries = ctypes.create_string_buffer(1 << 14), ctypes.c_int()
        st = lib.split_merge_calls(calls, fail, cluster_size, regions, log, len(log), ctypes.byref(queries))
        return st, [line.split() for line in log.value.decode().splitlines()], queries.value

    return run


def unjoined(log):
    """Side streams with work the caller's stream (or the host) does not wait for."""
    open_, recorded = set(), {}
    for what, *arg in log:
        failed = arg and arg[-1] == "failed"
        if failed:
            arg = arg[:-1]
        n = [int(a) for a in arg]
        if what == "launch" and n[0] in SIDE and not failed:
            open_.add(n[0])
            recorded = {e: s for e, s in recorded.items() if s != n[0]}
        elif what == "record" and not failed:
            recorded[n[0]] = n[1]
        elif what == "wait" and not failed and n[0] == CALLER and n[1] in recorded:
            open_.discard(recorded[n[1]])
        elif what == "sync":
            open_.discard(n[0])
    return open_


@pytest.mark.parametrize("cluster_size", [0, 16, 1])
@pytest.mark.parametrize("regions", [152, 153])  # as many as SMs: teams from the start; more: clusters only
def test_every_call_failing_in_turn(regions, cluster_size, passes):
    st, log, _ = passes(cluster_size=cluster_size, regions=regions)
    assert st == 0 and not unjoined(log)
    side = () if cluster_size == 1 else (SIDE if regions == 152 else SIDE[:1])
    assert {int(x[1]) for x in log if x[0] == "launch"} == {CALLER, *side}
    for fail in range(len(log)):
        st, got, _ = passes(fail=fail, cluster_size=cluster_size, regions=regions)
        assert got[fail][-1] == "failed" and st != 0, got
        assert not unjoined(got), got
        if got[fail][0] in ("occupancy", "attribute"):
            assert not any(x[0] == "launch" for x in got), got


def test_occupancy_is_asked_once_per_context_and_shape(passes):
    assert passes(calls=1)[2] == passes(calls=5)[2] == 2
