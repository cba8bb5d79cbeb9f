"""The products this framework is timed on: c = a b mod (X^N + 1, q).

A case is one call of a public entry point on a resident context:

* kind "device": ``Context.run_device`` on device buffers, one exact product;
* kind "host": ``Context.run`` on host arrays (copies in and out inside the
  call), with pageable or pinned buffers;
* kind "batch": ``Batch.run_device``, many products of uneven N and width in
  one tuned CUDA graph.

Every modulus and operand comes from polymul.workload's seeded generators.
Results are whole numbers and exact.
"""
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "fherma-polymult_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import polymul  # noqa: E402
from polymul import workload  # noqa: E402


def _one(kind, N, W, pattern="uniform", pinned=False):
    return {"kind": kind, "N": N, "W": W, "pattern": pattern, "pinned": pinned}


def _batch(count, mix_seed):
    return {"kind": "batch", "count": count, "mix_seed": mix_seed}


def listed():
    return [
        # The smallest calls, where launches and latency are all there is: a
        # toy ring with an odd width, and the widest golden vector of the
        # one-block transform.
        dict(_one("device", 256, 65), name="device_N256_W65"),
        dict(_one("device", 1024, 868), name="device_N1024_W868"),
        # The small benchmark point (256-bit modulus), on device and as one
        # plain call from a program's own pageable arrays.
        dict(_one("device", 4096, 256), name="device_N4096_W256"),
        dict(_one("host", 4096, 256), name="host_N4096_W256"),
        # The narrowest width of the batched mix, one bit short of its limbs.
        dict(_one("device", 8192, 127), name="device_N8192_W127"),
        # An ordinary product of the mix.
        dict(_one("device", 16384, 512), name="device_N16384_W512"),
        # The 868-bit benchmark point with sparse operands (90% zeros).
        dict(_one("device", 32768, 868, "sparse"), name="device_N32768_W868_sparse"),
        # The 1747-bit benchmark point with every coefficient q - 1 (longest
        # carries).
        dict(_one("device", 65536, 1747, "max"), name="device_N65536_W1747_max"),
        # The headline product, on device and end to end from pinned host
        # buffers.
        dict(_one("device", 65536, 2048), name="device_N65536_W2048"),
        dict(_one("host", 65536, 2048, pinned=True), name="host_N65536_W2048"),
        # Past the headline's ring: columns of 128, an odd width.
        dict(_one("device", 1 << 18, 1023), name="device_N262144_W1023"),
        # A tuned batch of uneven products from the batched benchmark's mix.
        dict(_batch(16, 3200), name="batch_mix16"),
    ]


def _primes(N, W):
    """About how many primes the basis of (N, W) holds (primes below 2^30)."""
    return math.ceil((2 * W + math.log2(N) + 21) / 29.99)


def _ops(N, W):
    """Multiply-add operations on words: decompose of both operands, three
    transforms with their butterflies, the pointwise product, the CRT."""
    L, K = workload.limbs_of(W), _primes(N, W)
    return 2 * (3 * K * N * L + 3 * (K * N // 2) * round(math.log2(N)) * 3 + K * N)


def draw(rng):
    limit = _ops(1 << 18, 1023)
    while True:
        what = rng.random()
        if what < 0.1:
            case = _batch(rng.randint(4, 16), rng.randint(1, 1 << 20))
        else:
            kind = "host" if what < 0.25 else "device"
            N = 1 << (rng.randint(12, 16) if kind == "host" else rng.randint(8, 18))
            W = round(math.exp(rng.uniform(math.log(33), math.log(2048))))
            pattern = rng.choice(("uniform", "uniform", "max", "sparse"))
            case = _one(kind, N, W, pattern, kind == "host" and rng.random() < 0.7)
        if work(case)["flops"] <= limit:
            return case


class _Device:
    """A device buffer of rows x limbs words owned by a batch, which lives as
    long as any tensor made from it."""

    def __init__(self, batch, ptr, rows, limbs):
        self.batch = batch
        self.__cuda_array_interface__ = {"shape": (rows, limbs), "typestr": "<i4", "data": (ptr, False), "version": 3}


def _words(x):
    return torch.from_numpy(np.ascontiguousarray(x).view(np.int32))


def _points(case):
    return workload.mix_points(case["count"], case["mix_seed"])


def prepare(case, seed):
    if case["kind"] == "batch":
        points = _points(case)
        contexts = [polymul.Context(N, W, q) for N, W, q in points]
        batch = polymul.Batch(contexts)
        outs = []
        for i, (a, b) in enumerate(workload.mix_operands(points, seed)):
            pa, pb, pc = (torch.as_tensor(_Device(batch, p, *a.shape), device="cuda") for p in batch.buffers(i))
            pa.copy_(_words(a))
            pb.copy_(_words(b))
            outs.append(pc)
        torch.cuda.synchronize()
        batch.tune()
        return {"kind": "batch", "batch": batch, "outs": outs}
    N, W = case["N"], case["W"]
    q, a, b = workload.case(N, W, case["pattern"], seed)
    context = polymul.Context(N, W, q)
    if case["kind"] == "host":
        hold = [_words(a), _words(b), torch.zeros(a.shape, dtype=torch.int32)]
        if case["pinned"]:
            hold = [x.pin_memory() for x in hold]
        return {"kind": "host", "context": context, "hold": hold, "a": hold[0].numpy().view(np.uint32),
                "b": hold[1].numpy().view(np.uint32), "out": hold[2].numpy().view(np.uint32)}
    a, b = _words(a).cuda(), _words(b).cuda()
    return {"kind": "device", "context": context, "a": a, "b": b, "out": torch.zeros_like(a)}


def run(state):
    if state["kind"] == "batch":
        state["batch"].run_device(torch.cuda.current_stream().cuda_stream)
        return state["outs"]
    if state["kind"] == "host":
        state["context"].run(state["a"], state["b"], out=state["out"])
        return state["hold"][2]
    state["context"].run_device(state["a"].data_ptr(), state["b"].data_ptr(), state["out"].data_ptr(),
                                torch.cuda.current_stream().cuda_stream)
    return state["out"]


def work(case):
    sizes = [(N, W) for N, W, _ in _points(case)] if case["kind"] == "batch" else [(case["N"], case["W"])]
    return {"bytes": sum(12 * N * workload.limbs_of(W) for N, W in sizes),
            "flops": sum(_ops(N, W) for N, W in sizes)}


def exact(case, seed):
    """The product by Python integers: each operand's coefficients packed into
    one long integer, multiplied, and folded at X^N = -1."""
    if case["kind"] == "batch" or case["N"] * case["W"] > 4096 * 1024:
        return None
    N = case["N"]
    q, a, b = workload.case(N, case["W"], case["pattern"], seed)
    m = workload.to_int(q)
    width = (2 * case["W"] + N.bit_length()) // 8 + 1

    def packed(rows):
        return int.from_bytes(b"".join(x.to_bytes(width, "little") for x in workload.rows_to_ints(rows)), "little")

    raw = (packed(a) * packed(b)).to_bytes(2 * N * width, "little")
    parts = [int.from_bytes(raw[i * width:(i + 1) * width], "little") for i in range(2 * N)]
    return _words(workload.ints_to_rows([(parts[i] - parts[N + i]) % m for i in range(N)], a.shape[1]))
