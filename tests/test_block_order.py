"""CPU test of the FP64 factorization's block order: on the P x P grid of
128x128 blocks every task's dependencies (the rules the kernel waits on) are
produced by tasks earlier in the order, and every block receives every panel
once, in increasing order."""
import ctypes

import numpy as np
import pytest

import dplasma_b200 as db

T_POTRF, T_TRSM, T_GEMM = 1, 2, 3


def tasks(P, S, delay, block):
    f = db.lib().dplasma_b200_debug_task_list_blocks
    f.argtypes = [ctypes.c_int] * 4 + [ctypes.c_void_p, ctypes.c_int]
    n = f(P, S, delay, block, None, 0)
    out = np.zeros(n, dtype=np.uint64)
    assert f(P, S, delay, block, out.ctypes.data, n) == n
    return [(int(t) & 0xF, (int(t) >> 4) & 0xFFFF, (int(t) >> 20) & 0xFFFF, (int(t) >> 36) & 0xFFFF,
             (int(t) >> 52) & 0xF, (int(t) >> 56) & 0xF) for t in out]


@pytest.mark.parametrize("P,S,delay,block", [(1, 4, 0, 0), (2, 4, 3, 0), (3, 4, 444, 0), (5, 1, 0, 0), (6, 4, 2, 0),
                                             (16, 4, 148, 0), (33, 4, 148, 8), (40, 3, 10, 5), (24, 8, 444, 0),
                                             (31, 15, 30, 4)])
def test_block_order(P, S, delay, block):
    potrf = np.zeros(P, int)
    trsm = np.zeros((P, P), int)
    upd = np.zeros((P, P), int)        # update tasks done
    panels = np.zeros((P, P), int)     # panels applied, in order

    slabs = 4                          # tasks per link of the chain, 32 rows each
    seen = set()

    def count(m, n):
        return 0 if n == 0 else -(-(n - 1) // S) + (slabs if m == n else 1)

    def strips(m, k):
        return slabs if m == k + 1 else 1

    for i, (ty, k, m, n, cnt, bj) in enumerate(tasks(P, S, delay, block)):
        if bj:
            assert m == k + 1 and (ty, k, bj) not in seen and 1 <= bj <= slabs
            seen.add((ty, k, bj))
        elif ty != T_POTRF:
            assert m != k + 1 or (ty == T_GEMM and k != n - 1), (i, ty, k, m, n)
        if ty == T_POTRF:
            assert panels[k, k] == k and upd[k, k] == count(k, k), (i, k)
            potrf[k] += 1
        elif ty == T_TRSM:
            assert potrf[k] == 1 and upd[m, k] == count(m, k) and panels[m, k] == k, (i, k, m)
            trsm[m, k] += 1
        else:
            assert ty == T_GEMM and 1 <= cnt <= S and k + cnt <= n <= m
            # every panel it reads is solved; the kernel waits for the last one
            for j in range(k, k + cnt):
                assert trsm[m, j] == strips(m, j) and trsm[n, j] == strips(n, j), (i, j, m, n)
            first = -(-(n - 1) // S) if k == n - 1 else k // S
            if bj:
                assert first <= upd[m, n] < first + slabs and panels[m, n] == k
                panels[m, n] += upd[m, n] == first + slabs - 1
            else:
                assert panels[m, n] == k and upd[m, n] == first, (i, k, m, n)
                panels[m, n] += cnt
            upd[m, n] += 1
    assert (potrf == 1).all()
    for m in range(P):
        assert all(trsm[m, k] == strips(m, k) for k in range(m)) and (panels[m, :m + 1] == np.arange(m + 1)).all()
