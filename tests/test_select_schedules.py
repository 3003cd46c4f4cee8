"""The selection's hand-shakes under schedules that a GPU seldom takes: its device code runs on the host
(native/heap_host.cpp), where the schedule can be chosen."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "ufednl_gb300", "csrc")


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("heap") / "heap_host")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, "-o", exe,
                    os.path.join(HERE, "native", "heap_host.cpp")], check=True)
    return lambda *a: subprocess.run([exe, *map(str, a)], check=True, capture_output=True, text=True, timeout=60).stdout


@pytest.mark.parametrize("nch,hit_at", [(2, 1), (2, 9), (3, 1), (3, 2), (8, 1), (8, 4), (8, 5), (8, 7), (8, 9)])
def test_extraction_and_windows_leave_together(host, nch, hit_at):
    """Chunks 1 .. nch - 1, the first window hit in chunk hit_at (or none): its verdict is step hit_at + 1's,
    and both warps leave there, however late the extracting one reads it."""
    met_x, met_w, stuck = map(int, host("steps", nch, hit_at).split())
    last = min(hit_at + 1, nch)
    assert (met_x, met_w, stuck) == (last, last, 0)


@pytest.mark.parametrize("reverse", [0, 1])
@pytest.mark.parametrize("k,values", [(21, 1000), (22, 5), (85, 1000), (300, 1 << 20), (341, 12)])
def test_lanes_that_run_apart_keep_one_heap(host, k, values, reverse):
    """A warp replaces the root together: each lane in turn runs as far ahead of the others as the code's own
    meetings let it, and the heap and every lane's registers end as one thread's."""
    bad, meetings = map(int, host("lanes", k, 200, values, reverse).split())
    assert bad == 0 and meetings > 0


def test_named_barriers_are_reached_by_whole_warps():
    """bar.sync and bar.arrive are undefined on a warp whose lanes are apart: each stands behind __syncwarp()."""
    lines = [(f, t) for f in sorted(os.listdir(CSRC)) for t in open(os.path.join(CSRC, f)).read().splitlines()]
    at = [n for n, (_, t) in enumerate(lines) if 'asm volatile("bar.sync' in t or 'asm volatile("bar.arrive' in t]
    assert at
    for n in at:
        assert lines[n - 1][1].strip() == "__syncwarp();", lines[n]
