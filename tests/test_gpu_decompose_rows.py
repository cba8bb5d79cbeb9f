"""The pipelined decompose's three ways of bringing limbs in: whole 16-byte groups
(L a multiple of 4), raw tiles (other L) and word by word (rows at an odd
offset, or a last tile that is not whole 16-byte groups), with fewer rows than
a tile, one tile a block, and more tiles a block than either ring has slots.
Each operand alone and both in one launch, against the oracle."""
import numpy as np
import pytest

import oracle
import polymul
from polymul import workload as wl

pytestmark = pytest.mark.gpu

CASES = [(2, 65), (4, 65), (4, 97), (64, 130), (128, 1050), (4096, 1747), (16384, 200), (32768, 609), (1 << 18, 40),
         (1 << 18, 70), (1 << 18, 128)]


@pytest.mark.parametrize("N,W", CASES)
def test_limbs_in(cuda, N, W):
    torch = cuda
    q, a, b = wl.case(N, W, "uniform", seed=2 * N + W)
    L = q.shape[0]
    pl = oracle.OraclePlan(N, q, pmax_log2=30)
    want = torch.from_numpy(pl.decompose(a).astype(np.int64)).cuda()
    with polymul.Context(N, W, q) as ctx:
        K = ctx.K
        p = torch.from_numpy(ctx.primes.astype(np.int64))[:, None].cuda()
        first = None
        for off in (0, 1, 0):
            buf = torch.zeros(2 * N * L + 4, dtype=torch.int32, device="cuda")
            buf[off:off + N * L] = torch.from_numpy(a.view(np.int32).reshape(-1)).cuda()
            buf[off + N * L:off + 2 * N * L] = torch.from_numpy(b.view(np.int32).reshape(-1)).cuda()
            at = buf.data_ptr() + 4 * off
            pair = torch.full((2 * K + 1, N), -1, dtype=torch.int32, device="cuda")
            one = torch.full((K + 1, N), -1, dtype=torch.int32, device="cuda")
            two = torch.full((K + 1, N), -1, dtype=torch.int32, device="cuda")
            ctx.stage_decompose(at, pair.data_ptr(), 2)
            ctx.stage_decompose(at, one.data_ptr(), 0)
            ctx.stage_decompose(at + 4 * N * L, two.data_ptr(), 1)
            assert ctx.get_error() == polymul.FPM_OK
            got = one[:K].to(torch.int64) & 0xFFFFFFFF
            assert bool((got < (4 if N > 1024 else 1) * p).all())
            assert torch.equal(got % p, want)
            assert torch.equal(pair[:K], one[:K]) and torch.equal(pair[K:2 * K], two[:K])
            assert bool((pair[2 * K] == -1).all()) and bool((one[K] == -1).all()) and bool((two[K] == -1).all())
            first = pair if first is None else first
            assert torch.equal(pair, first)
