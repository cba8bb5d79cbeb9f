"""When the pipelined decompose may bulk-copy whole limb tiles (raw_tiles_aligned,
fherma-polymult_b200/csrc/kernels.h), built with nvcc as a host program: over
bases, ranges and limb counts, a yes means that every 128-row tile starts on a
16-byte boundary and is a multiple of 16 bytes long, as the copies need, and a
range that meets this at an aligned base is a yes.  No GPU is needed; skipped
where nvcc is absent."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fherma-polymult_b200", "csrc")

PROGRAM = r"""
#include "kernels.h"
#include <algorithm>
#include <cstdio>
using namespace fpm;

int main() {
    long bad = 0, yes = 0;
    for (int L = 1; L <= 64; ++L)
        for (uint64_t base : {0ull, 4ull, 8ull, 12ull, 16ull})
            for (uint32_t n0 = 0; n0 < 300; n0 += n0 < 8 ? 1 : n0 < 120 ? 56 : 5)
                for (uint32_t n1 = n0 + 1; n1 < n0 + 300; ++n1) {
                    bool ok = true;
                    for (uint32_t r = n0; r < n1; r += 128) {
                        const uint64_t at = base + 4ull * r * L, bytes = 4ull * L * std::min(128u, n1 - r);
                        ok = ok && at % 16 == 0 && bytes % 16 == 0;
                    }
                    const bool got = raw_tiles_aligned(base, n0, n1, L);
                    yes += got;
                    if (got && !ok) ++bad;
                    if (base % 16 == 0 && ok && !got) ++bad;
                }
    std::printf("%ld yes, %ld failures\n", yes, bad);
    return bad != 0 || yes == 0;
}
"""


def test_raw_tiles_aligned(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    src = tmp_path / "raw.cu"
    src.write_text(PROGRAM)
    exe = tmp_path / "raw"
    subprocess.run([nvcc, "-std=c++17", "--expt-relaxed-constexpr", "-Wno-deprecated-gpu-targets", "-I", CSRC,
                    "-I", os.path.join(CSRC, "..", "..", "include"), str(src), "-o", str(exe)], check=True,
                   capture_output=True, timeout=300)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout[-2000:]
