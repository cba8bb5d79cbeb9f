"""The pipelined CRT over limb counts and row alignments: every remainder of L
mod 4 (how a row splits into 16-byte stores), the smallest and largest L, one
to several chunks of primes (odd and even, so tiles start at either operand
slot), one tile and several per block.  Bit-exact against the oracle, and the
same on repeats; words around the result stay untouched."""
import numpy as np
import pytest

import oracle
import polymul
from polymul import workload as wl

pytestmark = pytest.mark.gpu

CASES = [(128, w) for w in (33, 96, 97, 128, 160, 161, 192, 255, 480, 481, 1000, 1024, 1985, 2016, 2048)] + \
        [(4096, 65), (32768, 127), (65536, 96), (65536, 1025)]


@pytest.mark.parametrize("pattern", ["uniform", "max"])
@pytest.mark.parametrize("N,W", CASES)
def test_rows_of_every_limb_count(cuda, N, W, pattern):
    torch = cuda
    q, a, b = wl.case(N, W, pattern, seed=N + 5 * W)
    c_ref, y_ref = oracle.OraclePlan(N, q, pmax_log2=30).polymul(a, b, want_y=True)
    want = torch.from_numpy(c_ref.view(np.int32).reshape(-1)).cuda()
    y = torch.from_numpy(y_ref.view(np.int32)).cuda()
    with polymul.Context(N, W, q) as ctx:
        L = ctx.L
        for off in range(4):
            for _ in range(3):
                buf = torch.full((N * L + 8,), 7, dtype=torch.int32, device="cuda")
                ctx.stage_crt(y.data_ptr(), buf.data_ptr() + 4 * off)
                assert ctx.get_error() == polymul.FPM_OK
                assert torch.equal(buf[off:off + N * L], want)
                assert bool((buf[:off] == 7).all()) and bool((buf[off + N * L:] == 7).all())
