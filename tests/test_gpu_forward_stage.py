"""Forward transforms of both operands alone (stage mode 1) in one block per
prime: both prime windows, aligned and unaligned residues, nothing written
beside them, against the oracle's transform."""
import numpy as np
import pytest

import oracle
import polymul
from polymul import workload as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [30, 31])
@pytest.mark.parametrize("N,W", [(256, 65), (512, 300), (1024, 868), (2048, 40), (2048, 1747)])
def test_forward_of_both_operands(cuda, N, W, bits):
    torch = cuda
    q, a, b = wl.case(N, W, "uniform", seed=3 * N + W)
    pl = oracle.OraclePlan(N, q, pmax_log2=bits)
    res = [pl.decompose(x) for x in (a, b)]
    want = np.concatenate([pl.ntt_forward(r) for r in res])
    with polymul.Context(N, W, q, prime_bits=bits) as ctx:
        n = ctx.K * N
        for off in (0, 1, 3):
            buf = torch.full((2 * n + 8,), 9, dtype=torch.int32, device="cuda")
            buf[off:off + 2 * n] = torch.from_numpy(np.concatenate(res).view(np.int32).reshape(-1)).cuda()
            at = buf.data_ptr() + 4 * off
            ctx.stage_transform(at, at + 4 * n, polymul.MODE_FORWARD)
            assert ctx.get_error() == polymul.FPM_OK
            got = buf.cpu().numpy()
            assert np.array_equal(got[off:off + 2 * n].view(np.uint32).reshape(want.shape), want)
            assert (got[:off] == 9).all() and (got[off + 2 * n:] == 9).all()
