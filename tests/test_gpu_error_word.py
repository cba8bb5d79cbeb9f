"""The host path's error word after a timeout: cleared by the time the call
that reports it returns, whatever the caller's default stream is busy with
(the word is read on the context's own streams, which do not wait for it).

The default stream is kept busy by a spin kernel that ends by itself, the
timeout is made with the library's stall hook; no GPU fault is involved.  Both
forms of the host path: one stream (small operands) and copy streams.
"""
import numpy as np
import pytest

import oracle
import polymul
from polymul import workload as wl

pytestmark = pytest.mark.gpu

SPIN_CYCLES = 1_500_000_000   # 0.75 s or more at 1965 MHz


@pytest.mark.parametrize("N,W", [(4096, 256), (8192, 300)])
def test_a_reported_timeout_is_cleared(cuda, N, W):
    torch = cuda
    q, a, b = wl.case(N, W, "uniform", seed=N + W)
    expect = oracle.OraclePlan(N, q).polymul(a, b)
    with polymul.Context(N, W, q) as ctx:
        assert np.array_equal(ctx.run(a, b), expect)   # allocations, which wait for the whole device
        ctx.set_wait_limit(2_000_000)
        busy = torch.cuda.Event()
        torch.cuda._sleep(SPIN_CYCLES)
        busy.record()
        for mask in (polymul.STALL_DECOMPOSE, polymul.STALL_CRT):
            ctx.inject_stall(mask)
            with pytest.raises(polymul.FpmError) as err:
                ctx.run(a, b)
            assert err.value.code == polymul.FPM_ETIMEOUT
            ctx.inject_stall(0)
            assert np.array_equal(ctx.run(a, b), expect)
        assert not busy.query(), "the default stream went idle before the calls were done"
        torch.cuda.synchronize()
        assert np.array_equal(ctx.run(a, b), expect)
        assert ctx.get_error() == polymul.FPM_OK
