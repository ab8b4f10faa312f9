"""Warp-aligned instructions of the kernels (tcgen05.alloc / ld / st / dealloc, the aligned cluster barrier) are undefined
unless the warp is converged, and a wait on an mbarrier is a loop that every lane may leave on its own.  Read from the
source, since code that happens to converge passes every run."""
import re
from pathlib import Path

import pytest

KERNELS = Path(__file__).resolve().parent.parent / "tinyinfinitrain_b200" / "csrc" / "kernels"
SOURCES = sorted(p for p in KERNELS.glob("*.cu") if "mbar_wait" in p.read_text())
ONE_THREAD = re.compile(r"elect_one\(\)|threadIdx\.x == 0|lane == 0|\btid == 0|\bleader\b")
MEET = re.compile(r"__syncwarp\(|__any_sync\(|__all_sync\(|mbar_wait_warp\(|elect_one\(\)")
ALIGNED = re.compile(r"\btmem_(ld|st)(16|32)\(|\btmem_(de)?alloc(_pair)?\(|\btmem_relinquish")
LANE_WAIT = re.compile(r"\bmbar_wait\(")


def _lines(path):
    """Source lines without comments, with the line number and whether the line lies in a block that one thread runs."""
    text = re.sub(r"/\*.*?\*/", lambda m: "\n" * m.group().count("\n"), path.read_text(), flags=re.S)
    depth, single, out = 0, [], []
    for no, line in enumerate(text.splitlines(), 1):
        line = line.split("//")[0]
        single = [d for d in single if d < depth]
        out.append((no, line, bool(single)))
        if ONE_THREAD.search(line) and "if" in line and line.rstrip().endswith("{"):
            single.append(depth + line.count("{") - line.count("}") - 1)
        depth += line.count("{") - line.count("}")
    return out


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_warps_leave_their_waits_together(path):
    lines = _lines(path)
    for i, (no, line, single) in enumerate(lines):
        if single or not LANE_WAIT.search(line):
            continue
        after = "\n".join(t for _, t, _ in lines[i + 1:i + 8])
        leaves = re.search(r"\b(break|return)\b", line)
        # lanes with different answers have to be brought together before anything else, and none may be gone by then
        assert MEET.search(after) and not leaves, f"{path.name}:{no}: a whole warp waits lane by lane"


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_aligned_instructions_follow_a_meeting_point(path):
    split = 0
    for no, line, single in _lines(path):
        if LANE_WAIT.search(line):
            split = no
        elif MEET.search(line) or "__syncthreads(" in line:
            split = 0
        if ALIGNED.search(line):
            assert not single and not split, f"{path.name}:{no}: reached from the lane-by-lane wait of line {split}"


def test_cluster_barrier_brings_the_warp_together():
    text = (KERNELS / "ptx_sm100.cuh").read_text()
    body = text[text.index("void cluster_sync_all()"):]
    body = body[:body.index("\n}")]
    assert re.search(r"\{\s*__syncwarp\(\);\s*asm volatile\(\"barrier\.cluster\.arrive", body)
    for path in KERNELS.glob("*.cu"):
        assert "barrier.cluster" not in path.read_text(), path.name
