"""Batches with products of N = 2^17, whose row tiles are 4096 elements where all
others are 2048: the grouped row pass of that length and the mixed one, where
a persistent block meets tiles of both sizes (one per block, or one per half)
one after the other in the same shared memory.  Every member equals its plain
product, which is checked against the oracle elsewhere."""
import numpy as np
import pytest

import oracle
import polymul
from polymul import workload as wl

pytestmark = pytest.mark.gpu

# N = 2^17 beside every other row length, both prime windows, more tiles of each
# than a persistent grid has blocks.
POINTS = [(1 << 17, 40, 0), (1 << 16, 250, 0), (1 << 14, 600, 0), (1 << 13, 700, 0), (1 << 17, 97, 0), (1 << 12, 300, 0),
          (1 << 15, 130, 0), (1 << 17, 33, 31), (1 << 14, 200, 31), (1 << 12, 64, 31)]

# (layout, order, prime_group, grid, pipe_min_log_n)
SCHEDULES = [(0, 1, 0, 0, 0), (0, 0, 4, 1, 0), (1, 1, 0, 1, 0), (2, 1, 0, 0, 0), (3, 1, 0, 0, 0), (3, 1, 0, 1, 0),
             (3, 0, 1, 1, 0), (3, 0, 2, 1, 16)]


@pytest.fixture(scope="module")
def products(cuda):
    ctxs, ops, want = [], [], []
    for i, (N, W, bits) in enumerate(POINTS):
        q, a, b = wl.case(N, W, "uniform", seed=1700 + i)
        ctx = polymul.Context(N, W, q, prime_bits=bits)
        ctxs.append(ctx)
        ops.append((a, b))
        want.append(ctx.run(a, b))
    q, a, b = wl.case(*POINTS[0][:2], "uniform", seed=1700)
    assert np.array_equal(want[0], oracle.OraclePlan(POINTS[0][0], q).polymul(a, b))
    yield ctxs, ops, want
    for c in ctxs:
        c.close()


@pytest.mark.parametrize("sched", SCHEDULES, ids=lambda s: "L%d-o%d-g%d-p%d-pipe%d" % s)
def test_row_tiles_of_both_sizes(products, sched):
    ctxs, ops, want = products
    with polymul.Batch(ctxs) as bt:
        bt.set_schedule(*sched)
        for _ in range(3):
            got = bt.run([a for a, _ in ops], [b for _, b in ops])
            for g, w in zip(got, want):
                assert np.array_equal(g, w)
