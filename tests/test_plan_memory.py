"""Twiddle tables of the one-block transforms: N = 256 .. 1024 hold two tables of K N
pairs (the forward one in entry order and in the order the kernel reads), as
N < 256 does (forward and inverse), so that what a context holds grows with N
by the tables, the residues and the limbs alone: 16 K + 8 K + 12 L bytes."""
import pytest

import polymul
from polymul import workload as wl


@pytest.mark.parametrize("W", [40, 97, 1000, 2040])
def test_bytes_per_coefficient(W):
    q, _, _ = wl.case(2, W, "zero", seed=W)
    info = {n: polymul.plan_info(1 << n, W, q)[0] for n in range(7, 11)}
    assert len({i.K for i in info.values()}) == 1   # the same basis size throughout
    K, L = info[7].K, q.shape[0]
    for n in (8, 9, 10):
        grown = info[n].device_bytes - info[7].device_bytes
        assert grown == ((1 << n) - 128) * (24 * K + 12 * L)
