"""CPU model of the ticket selection of the tile Cholesky (chain_ticket and
draw_ticket in dplasma_b200/csrc/potrf_kernel.cu): one CTA runs every POTRF and
draws other tickets while its next POTRF is more than a grid's width ahead, or
when tickets before it stay undrawn; the others pass over POTRF tickets.  Every
CTA runs its tasks in the order it took them, waiting for each one's
dependencies.  Whatever the interleaving, and with a single resident CTA, every
ticket has to run once, and no CTA may end up waiting for ever."""
import random

import numpy as np
import pytest

from test_block_order import tasks as block_tasks
from test_task_order import SLABS, tasks_blocked

T_POTRF, T_TRSM, T_GEMM = 1, 2, 3


class Counts:
    """the completion counters and the rules of wait_deps / all_updates"""

    def __init__(self, mt, S, mixed):
        self.mt, self.S, self.mixed, self.nbs = mt, S, mixed, 2 if mixed else 1
        self.potrf = np.zeros(mt, int)
        self.trsm = np.zeros((mt, mt), int)
        self.upd = np.zeros((mt, mt), int)

    def strips(self, m, k):
        return self.nbs * (SLABS if m == k + 1 else 1)

    def all_updates(self, m, n):
        if self.mixed:
            return -(-n // self.S)
        return 0 if n == 0 else -(-(n - 1) // self.S) + (SLABS if m == n else 1)

    def ready(self, t):
        ty, k, m, n, cnt, bj = t
        if ty == T_POTRF:
            return self.upd[k, k] >= self.all_updates(k, k)
        if ty == T_TRSM:
            return self.upd[m, k] >= self.all_updates(m, k) and self.potrf[k] >= 1
        if self.mixed:
            kl, before = min(k * self.S + self.S, n) - 1, k
        else:
            kl = k + cnt - 1
            before = -(-(n - 1) // self.S) if k == n - 1 else k // self.S
        return (self.trsm[m, kl] >= self.strips(m, kl) and self.trsm[n, kl] >= self.strips(n, kl)
                and self.upd[m, n] >= before)

    def finish(self, t):
        ty, k, m, n = t[:4]
        if ty == T_POTRF:
            self.potrf[k] += 1
        elif ty == T_TRSM:
            self.trsm[m, k] += 1
        else:
            self.upd[m, n] += 1


def run(tl, counts, grid, rng, resident):
    """`resident` of the `grid` CTAs run at a time (a CTA starts when another has
    ended); returns the runs of every ticket"""
    nt, mt = len(tl), counts.mt
    pos = [i for i, t in enumerate(tl) if t[0] == T_POTRF]
    ticket, ran = 0, [0] * nt
    chain = {"next": 0, "carry": -1}
    margin = grid if grid > 1 else 0

    def draw():
        nonlocal ticket
        while True:
            t = ticket
            ticket += 1
            if not (t < nt and tl[t][0] == T_POTRF):
                return t

    def take(is_chain):
        """the next ticket, or None while the chain CTA waits"""
        if not is_chain:
            return draw()
        pp = pos[chain["next"]] if chain["next"] < mt else 1 << 30
        if chain["carry"] < 0:
            go = ticket < pp - margin
            if not go and ticket < pp:
                k = chain["next"]
                if counts.upd[k, k] < counts.all_updates(k, k):
                    go = rng.random() < 0.05            # tickets before it stayed undrawn for a while
                    if not go:
                        return None
            if go:
                chain["carry"] = draw()
        if 0 <= chain["carry"] < pp:
            t, chain["carry"] = chain["carry"], -1
            return t
        chain["next"] += 1
        return pp

    first = True
    waiting, live, queue = {}, [], list(range(grid))
    idle = 0
    while queue or live:
        while queue and len(live) < resident:
            live.append((queue.pop(0), first))
            first = False
        i = rng.randrange(len(live))
        cta, is_chain = live[i]
        t = waiting.get(cta)
        if t is None:
            t = take(is_chain)
            if t is None:
                idle += 1
                assert idle < 200000
                continue
            if t >= nt:
                live.pop(i)
                continue
            waiting[cta] = t
        if counts.ready(tl[t]):
            counts.finish(tl[t])
            ran[t] += 1
            waiting[cta] = None
            idle = 0
        else:
            idle += 1
            assert idle < 200000, "no CTA makes progress"
    return ran


@pytest.mark.parametrize("grid,resident", [(1, 1), (2, 1), (2, 2), (5, 3), (12, 12), (40, 40)])
@pytest.mark.parametrize("P,S,delay,block", [(1, 2, 0, 0), (7, 2, 12, 4), (14, 4, 12, 0), (20, 15, 40, 16)])
def test_fp64_blocks(P, S, delay, block, grid, resident):
    tl = block_tasks(P, S, delay, block)
    for seed in range(3):
        assert run(tl, Counts(P, S, False), grid, random.Random(seed), resident) == [1] * len(tl)


@pytest.mark.parametrize("grid,resident", [(1, 1), (2, 1), (5, 3), (12, 12), (40, 40)])
@pytest.mark.parametrize("mt,S,delay,bw", [(1, 8, 0, 0), (9, 4, 7, 4), (18, 16, 72, 16)])
def test_mixed(mt, S, delay, bw, grid, resident):
    tl = tasks_blocked(S, mt, 2, delay, bw, bw)
    for seed in range(3):
        assert run(tl, Counts(mt, S, True), grid, random.Random(seed), resident) == [1] * len(tl)
