"""Orderings in the device code that no run shows to be missing: the source is
read for them."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ressim_gb300", "csrc")
SOURCES = sorted(p for e in ("cu", "cuh") for p in glob.glob(os.path.join(CSRC, "*." + e)))


def code(path):
    """The source without its comments."""
    with open(path) as f:
        return re.sub(r"//[^\n]*|/\*.*?\*/", "", f.read(), flags=re.S)


@pytest.mark.parametrize("path", SOURCES, ids=[os.path.basename(p) for p in SOURCES])
def test_mbarriers_are_fenced_before_use(path):
    """Between the initialisation of mbarriers (in place, or by a helper
    mbar_init) and the barrier that lets other threads use them stands
    fence.mbarrier_init, and where bulk copies complete on them the fence to
    the asynchronous proxy."""
    src = code(path)
    helper = re.search(r"void mbar_init\([^}]*\}", src)
    if helper:  # its calls are looked at instead
        src = src.replace(helper.group(0), "")
    for m in re.finditer(r"mbarrier\.init\.|\bmbar_init\(", src):
        end = re.compile(r"__syncthreads\(\)|cluster\.sync\(\)").search(src, m.end())
        between = src[m.end():end.start() if end else len(src)]
        assert "fence.mbarrier_init" in between
        if "cp.async.bulk" in src:
            assert "fence.proxy.async" in between


def test_segment_sort_reads_before_it_writes():
    """k_seg_sort (amg.cu) puts a segment back in place, a lane's entries where
    other lanes read theirs: a warp barrier stands between."""
    src = code(os.path.join(CSRC, "amg.cu"))
    body = src[src.index("k_seg_sort(int n"):]
    body = body[:body.index("\n}")]
    read, write = body.rindex("val[p0 + e]"), body.rindex("key[p0 + place[c]] =")
    assert read < body.index("__syncwarp()", read) < write
