"""CPU test of the batched kernel's launch shape (bt_choose in
dplasma_b200/csrc/batched.cu): the shape that was fastest on a B200 (148 SMs), at
batches on both sides of where it changes.  A shape of more problems per SM pays
when the batch's work outlasts its largest problem, whatever that one's order."""
import ctypes
import random

import pytest

import dplasma_b200 as db

ONE, FOUR, EIGHT, PAIR = 0, 1, 2, 3       # warps per problem; PAIR: eight, two problems per SM
F64, F32 = 1, 0


def choice(fp64, sizes, sms=148):
    f = db.lib().dplasma_b200_debug_batched_choice
    f.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_int, ctypes.POINTER(ctypes.c_int)]
    return f(fp64, sms, len(sizes), (ctypes.c_int * max(len(sizes), 1))(*sizes))


def uniform(lo, hi, count):
    r = random.Random(hi * count)
    return [r.randint(lo, hi) for _ in range(count)]


@pytest.mark.parametrize("fp64,sizes,best", [
    # one problem per SM and fewer: the lowest latency
    (F64, [8], EIGHT), (F64, [512] * 148, EIGHT), (F32, [256], EIGHT), (F32, uniform(8, 1024, 148), EIGHT),
    # a second problem per SM: not yet worth a shared SM, but for small ones
    (F64, uniform(8, 192, 297), EIGHT), (F64, uniform(8, 256, 400), EIGHT), (F32, uniform(8, 256, 400), EIGHT),
    (F32, uniform(8, 512, 400), EIGHT), (F32, uniform(8, 768, 297), EIGHT), (F32, [64] * 296, FOUR),
    # work for several per SM
    (F64, uniform(64, 256, 1024), FOUR), (F64, uniform(8, 96, 4096), ONE), (F64, uniform(8, 64, 2000), ONE),
    (F64, uniform(32, 512, 4096), EIGHT), (F32, uniform(8, 96, 8192), ONE), (F32, uniform(8, 256, 4096), FOUR),
    (F32, uniform(8, 512, 900), PAIR),
    # many small ones and a few large: the large ones' latency
    (F64, [64] * 500 + [256] * 20, EIGHT), (F32, [32] * 2000 + [512], EIGHT),
    (F32, [16 + i % 33 for i in range(8000)] + [512] * 4, EIGHT),
    # empty problems and none
    (F64, [0] * 40, EIGHT), (F32, [0], EIGHT), (F64, [], EIGHT)])
def test_launch_shape(fp64, sizes, best):
    assert choice(fp64, sizes) == best


def test_every_order_and_batch_has_a_shape():
    for fp64, top in ((F64, 686), (F32, 1024)):
        for n in list(range(1, top, 37)) + [top]:
            for count in (1, 2, 147, 149, 600, 5000):
                assert 0 <= choice(fp64, [n] * count) < (3 if fp64 else 4)
                assert 0 <= choice(fp64, [n] * count, sms=10) < (3 if fp64 else 4)
