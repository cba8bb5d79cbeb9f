"""The one-launch transforms against the oracle and against the separate passes:
one block per prime (N = 256 .. 2048, products and forward transforms), a
cluster per prime (N = 4096 .. 32768), on both sides of the line where clusters
no longer all fit the GPU, in both prime windows, from aligned and unaligned
residues, and the same on repeats."""
import numpy as np
import pytest

import oracle
import polymul
from polymul import workload as wl

pytestmark = pytest.mark.gpu

CASES = [(N, W, bits) for N in (256, 512, 1024, 2048) for W in (40, 700) for bits in (30, 31)] + \
        [(4096, 64, 30), (4096, 500, 31), (8192, 127, 30), (8192, 600, 31), (16384, 300, 31), (16384, 1070, 30),
         (16384, 1110, 30), (32768, 257, 30), (32768, 400, 31), (32768, 520, 30), (32768, 560, 30)]


@pytest.mark.parametrize("N,W,prime_bits", CASES)
def test_one_launch_transforms(cuda, N, W, prime_bits):
    torch = cuda
    q, a, b = wl.case(N, W, "uniform", seed=N + W)
    pl = oracle.OraclePlan(N, q, pmax_log2=prime_bits)
    _, y = pl.polymul(a, b, want_y=True)
    want = torch.from_numpy(y.view(np.int32)).cuda()
    limbs = torch.from_numpy(np.concatenate([a, b]).view(np.int32)).cuda()
    with polymul.Context(N, W, q, prime_bits=prime_bits) as ctx:
        K = ctx.K
        res = torch.zeros(2 * K * N, dtype=torch.int32, device="cuda")
        ctx.stage_decompose(limbs.data_ptr(), res.data_ptr(), 2)
        for off in (0, 1):
            for _ in range(3):
                buf = torch.full((2 * K * N + 8,), 5, dtype=torch.int32, device="cuda")
                buf[off:off + 2 * K * N] = res
                A = buf.data_ptr() + 4 * off
                ctx.stage_transform(A, A + 4 * K * N, polymul.MODE_PRODUCT)
                assert ctx.get_error() == polymul.FPM_OK
                assert torch.equal(buf[off:off + K * N].view(K, N), want)
                assert bool((buf[:off] == 5).all()) and bool((buf[off + 2 * K * N:] == 5).all())
        if N > 2048:
            # the separate passes (stage modes 2, 3, 4)
            for mode in (2, 3, 4):
                ctx.stage_transform(res.data_ptr(), res.data_ptr() + 4 * K * N, mode)
            torch.cuda.synchronize()
            assert torch.equal(res[:K * N].view(K, N), want)
        elif prime_bits == 30:
            ctx.stage_transform(res.data_ptr(), res.data_ptr() + 4 * K * N, polymul.MODE_FORWARD)
            torch.cuda.synchronize()
            fwd = pl.ntt_forward(pl.decompose(a))
            assert np.array_equal(res[:K * N].view(K, N).cpu().numpy().view(np.uint32), fwd)
