"""The pipelined decompose over its chunk sizes: every share of a chunk per
fold warp (2 to 16 primes), one to three chunks with and without padding, and
tiles with fewer rows than threads.  Residues are exact: congruent to the
oracle's and below 4p (below p where the transform wants canonical input), with
nothing written past the K rows."""
import numpy as np
import pytest

import oracle
import polymul
from polymul import workload as wl

pytestmark = pytest.mark.gpu

CASES = [(N, W) for N in (32, 128, 4096) for W in (40, 97, 200, 300, 480, 700, 868, 940, 1023, 1300, 1600, 1747, 2048)]


@pytest.mark.parametrize("N,W", CASES)
def test_residues_of_every_chunk_size(cuda, N, W):
    torch = cuda
    q, a, _ = wl.case(N, W, "uniform", seed=N + W)
    pl = oracle.OraclePlan(N, q, pmax_log2=30)
    want = pl.decompose(a).astype(np.uint64)
    da = torch.from_numpy(a.view(np.int32)).cuda()
    with polymul.Context(N, W, q) as ctx:
        p = ctx.primes.astype(np.uint64)[:, None]
        out = torch.full((ctx.K + 1, N), -1, dtype=torch.int32, device="cuda")
        ctx.stage_decompose(da.data_ptr(), out.data_ptr(), 0)
        assert ctx.get_error() == polymul.FPM_OK
        got = out.cpu().numpy().view(np.uint32).astype(np.uint64)
        assert (got[ctx.K] == 0xFFFFFFFF).all()
        assert (got[:ctx.K] < (4 if N > 1024 else 1) * p).all()
        assert np.array_equal(got[:ctx.K] % p, want)
