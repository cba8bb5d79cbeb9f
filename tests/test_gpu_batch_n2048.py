"""Batches of products of N = 2048: one grouped launch for all of a batch's
transforms of that length (per prime window and table of 64 products), in every
layout, with prime groups and persistent grids.  Every member equals its plain
product."""
import numpy as np
import pytest

import polymul
from polymul import workload as wl

pytestmark = pytest.mark.gpu

WIDTHS = (33, 97, 256, 700, 1300, 2048)


def _products(count, bits=lambda i: 0):
    ctxs, ins, want = [], [], []
    for i in range(count):
        q, a, b = wl.case(2048, WIDTHS[i % len(WIDTHS)], "uniform", seed=500 + i)
        ctx = polymul.Context(2048, WIDTHS[i % len(WIDTHS)], q, prime_bits=bits(i))
        ctxs.append(ctx)
        ins.append((a, b))
        want.append(ctx.run(a, b))
    return ctxs, ins, want


def _check(bt, ins, want):
    for _ in range(2):
        got = bt.run([a for a, _ in ins], [b for _, b in ins])
        for g, w in zip(got, want):
            assert np.array_equal(g, w)


@pytest.mark.parametrize("layout", [0, 1, 2, 3])
def test_one_launch_a_stage(cuda, layout):
    ctxs, ins, want = _products(32)
    with polymul.Batch(ctxs) as bt:
        bt.set_schedule(layout, 1, 0, 0, 0)
        assert bt.info.launches == 3
        _check(bt, ins, want)
    for c in ctxs:
        c.close()


# (layout, order, prime_group, grid, pipe_min_log_n)
@pytest.mark.parametrize("sched", [(0, 0, 5, 0, 0), (1, 1, 0, 1, 0), (1, 1, 16, 2, 11), (2, 1, 3, 1, 12), (2, 1, 0, 0, 11),
                                   (3, 1, 16, 1, 0)])
def test_both_prime_windows_and_more_than_a_table(cuda, sched):
    ctxs, ins, want = _products(70, bits=lambda i: 31 if i % 3 == 0 else 0)
    with polymul.Batch(ctxs) as bt:
        bt.set_schedule(*sched)
        _check(bt, ins, want)
    for c in ctxs:
        c.close()
