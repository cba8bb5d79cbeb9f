"""Shared memory of the mixed-geometry row pass (fherma-polymult_b200/csrc/
ntt_passes.cuh), built with nvcc as a host program: a block holds one 256-thread
tile of any row length, or a 128-thread tile in each half, and three blocks
fit an SM (228 KB, 1 KB of it reserved per block), as many as the kernel's
registers are sized for.  No GPU is needed; skipped where nvcc is absent."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fherma-polymult_b200", "csrc")

PROGRAM = r"""
#include "ntt_passes.cuh"
#include <cstdio>
using namespace fpm;

static int bad = 0;

template <int LS>
void tile(uint32_t max_log_s) {
    if (LS > static_cast<int>(max_log_s)) return;
    const uint32_t bytes = mixed_row_bytes(max_log_s);
    const size_t room = row_threads<LS>() == 256 ? bytes : bytes / 2;
    if (row_threads<LS>() != 256 && row_threads<LS>() != 128) ++bad, std::printf("S = 2^%d: %d threads\n", LS, row_threads<LS>());
    if (row_bar_offset<LS>() > room) ++bad, std::printf("S = 2^%d: %zu of %zu bytes\n", LS, row_bar_offset<LS>(), room);
}

int main() {
    for (uint32_t m = 6; m <= 11; ++m) {
        tile<6>(m), tile<7>(m), tile<8>(m), tile<9>(m), tile<10>(m), tile<11>(m);
        const uint32_t bytes = mixed_row_bytes(m);
        if ((bytes / 2) % 1024) ++bad, std::printf("halves of %u bytes\n", bytes);
        if (3 * (bytes + 32 + 1024) > 228 * 1024) ++bad, std::printf("rows up to 2^%u: %u bytes a block\n", m, bytes);
    }
    std::printf("%d failures\n", bad);
    return bad != 0;
}
"""


def test_tiles_fit(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    src = tmp_path / "rows.cu"
    src.write_text(PROGRAM)
    exe = tmp_path / "rows"
    subprocess.run([nvcc, "-std=c++17", "--expt-relaxed-constexpr", "-Wno-deprecated-gpu-targets", "-I", CSRC, str(src),
                    "-o", str(exe)], check=True, capture_output=True, timeout=300)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout[-2000:]
    assert "0 failures" in out.stdout
