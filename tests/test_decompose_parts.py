"""When a decompose cuts its tiles by primes (decompose_parts, fherma-polymult_b200/
csrc/kernels.h), built with nvcc as a host program: parts cover every chunk in
whole runs of 4 piece primes, fit the SMs, and a count of one, which lets the
transform start early, is what every (N, K) gets that cannot be cut (among them
N = 2048, K = 49 .. 56 on 148 SMs); no other in 512 .. 2048, K >= 48, is left
whole there.  No GPU is needed; skipped where nvcc is absent."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fherma-polymult_b200", "csrc")

PROGRAM = r"""
#include "kernels.h"
#include <cstdio>
using namespace fpm;

static int bad = 0;
#define CHECK(c, ...) do { if (!(c)) { ++bad; std::printf(__VA_ARGS__); std::printf("\n"); } } while (0)

int main() {
    for (uint32_t N = 2; N <= (1u << 18); N *= 2)
        for (int K = 1; K <= 160; ++K)
            for (uint32_t operands = 1; operands <= 2; ++operands)
                for (int sms : {1, 16, 132, 148}) {
                    const uint32_t tiles = (N + 127) / 128, chunks = dec_wide_chunks(K), whole = dec_wide_piece(K);
                    CHECK(4 * whole * chunks >= static_cast<uint32_t>(K) && whole % 2 == 0 && whole <= 16, "K %d", K);
                    const DecParts c = decompose_parts(N, K, tiles, operands, sms);
                    CHECK(c.piece >= 2 && c.piece % 2 == 0 && whole % c.piece == 0, "N %u K %d piece %u", N, K, c.piece);
                    if (c.parts == 1) continue;
                    CHECK(N >= 512 && N <= 2048 && K >= 48, "N %u K %d cut", N, K);
                    CHECK(c.parts * c.piece == chunks * whole, "N %u K %d: %u x %u", N, K, c.parts, c.piece);
                    CHECK(c.parts * tiles * operands <= static_cast<uint32_t>(sms), "N %u K %d: %u parts", N, K, c.parts);
                }
    for (uint32_t N = 512; N <= 2048; N *= 2)
        for (int K = 48; K <= 160; ++K)
            CHECK((decompose_parts(N, K, N / 128, 2, 148).parts == 1) == (N == 2048 && K >= 49 && K <= 56), "N %u K %d", N, K);
    std::printf("%d failures\n", bad);
    return bad != 0;
}
"""


def test_decompose_parts(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    src = tmp_path / "parts.cu"
    src.write_text(PROGRAM)
    exe = tmp_path / "parts"
    subprocess.run([nvcc, "-std=c++17", "--expt-relaxed-constexpr", "-Wno-deprecated-gpu-targets", "-I", CSRC, str(src),
                    "-o", str(exe)], check=True, capture_output=True, timeout=300)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout[-2000:]
