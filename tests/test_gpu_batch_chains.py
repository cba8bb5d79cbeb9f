"""Layout 2 with one-product chains over the branches: products of every transform
form (one block, cluster, separate passes), more and fewer chains than
branches, all and some of the products with chains.  Every member equals its
plain product."""
import numpy as np
import pytest

import polymul
from polymul import workload as wl

pytestmark = pytest.mark.gpu

SIZES = [(64, 40), (512, 100), (2048, 97), (4096, 256), (4096, 70), (8192, 300), (16384, 64), (32768, 350), (65536, 60)]


class DeviceWords:
    """A buffer of the batch as a torch view (used while the batch is open)."""

    def __init__(self, ptr, rows, limbs):
        self.__cuda_array_interface__ = {"shape": (rows, limbs), "typestr": "<i4", "data": (ptr, False), "version": 3}


@pytest.mark.parametrize("take,pipe", [(9, 12), (9, 14), (9, 16), (9, 1), (2, 12), (4, 11)])
def test_chains_equal_plain_products(cuda, take, pipe):
    torch = cuda
    sizes = SIZES[-take:]
    ctxs, ins, want = [], [], []
    for i, (N, W) in enumerate(sizes):
        q, a, b = wl.case(N, W, "uniform", seed=100 + i)
        ctx = polymul.Context(N, W, q)
        ctxs.append(ctx)
        ins.append((a, b))
        want.append(ctx.run(a, b))
    with polymul.Batch(ctxs) as bt:
        bt.set_schedule(2, 1, 0, 0, pipe)
        views = [[torch.as_tensor(DeviceWords(p, c.N, c.L), device="cuda") for p in bt.buffers(i)]
                 for i, c in enumerate(ctxs)]
        for (pa, pb, pc), (a, b) in zip(views, ins):
            pa.copy_(torch.from_numpy(a.view(np.int32)))
            pb.copy_(torch.from_numpy(b.view(np.int32)))
            pc.zero_()
        torch.cuda.synchronize()
        s = torch.cuda.Stream()
        for _ in range(3):
            bt.run_device(s.cuda_stream)
        s.synchronize()
        for (_, _, pc), w in zip(views, want):
            assert np.array_equal(pc.cpu().numpy().view(np.uint32), w)
        got = bt.run([a for a, _ in ins], [b for _, b in ins])
        for g, w in zip(got, want):
            assert np.array_equal(g, w)
    for c in ctxs:
        c.close()
