"""CPU check of the streamed factorization's POTRF: the consumer threads add the
untouched copy into the diagonal tile (stream_add_rows) and then load its first
128x128 block by asynchronous copies (p128_load).  The two deal out the elements
differently, so threads read what others wrote, and a barrier of all consumers
has to stand between them.  The race is improbable on a GPU (one thread would
have to run most of a tile ahead) and its effect is repaired by the refinement,
so the order is checked here, from the maps of both loops and in the source."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dplasma_b200", "csrc")
NCONS, NBI = 256, 256


def _adder(r, c):
    """thread of stream_add_rows that writes element (r, c): pairs of rows, column after column"""
    return (c * (NBI // 2) + r // 2) % NCONS


def _loads():
    """(thread, row, column) of p128_load's copies of two rows, lower 32-blocks only"""
    for tid in range(NCONS):
        r = (tid & 63) * 2
        for c in range(tid >> 6, 128, 4):
            if r + 2 > (c & ~31):
                yield tid, r, c


def _source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def test_loads_read_other_threads_writes():
    # (thread 64 loads column 1, which threads 128.. write): other warps' elements,
    # so no barrier of a warp would do
    crossing = [(t, r, c) for t, r, c in _loads() if _adder(r, c) // 32 != t // 32]
    assert len(crossing) > 0


def test_maps_are_those_of_the_source():
    add, load = _source("potrf_kernel.cu"), _source("dev_potrf128.cuh")
    assert "for (int e = threadIdx.x; e < a.nbi * per_col; e += NCONS)" in add
    assert "const int c = e / per_col, r = 2 * (e % per_col);" in add
    assert "const int r = (tid & 63) * 2;" in load
    assert "for (int c = tid >> 6; c < 128; c += 4)" in load


def test_barrier_between_the_addition_and_potrf():
    src = _source("potrf_kernel.cu")
    start = src.index("void consumer_warps(")
    body = src[start:src.index("__launch_bounds__", start)]
    add = body.index("stream_add_rows(a, k, k")
    between = body[add:body.index("potrf_task<MIXED", add)]
    assert "named_bar_sync(1, NCONS)" in between
    # the strips' additions end in a barrier (slabs) or in the producer's mbarrier
    strip = body[body.index("stream_add_rows(a, m, k"):]
    assert re.search(r"named_bar_sync\(1, NCONS\);\s*} else {\s*fence_proxy_async\(\);.*?mbar_arrive\(&ctl->prep\)", strip,
                     re.S)
