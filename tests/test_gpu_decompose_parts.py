"""Tiles cut by primes over idle SMs (and N = 2048, K = 53, which cannot be cut):
residues of one operand and of both, as in test_gpu_decompose_rows, with several
chunks, padding after the last prime, and a guard row."""
import pytest

from test_gpu_decompose_rows import test_limbs_in as limbs_in

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,W", [(512, 900), (512, 2048), (1024, 1300), (1024, 1747), (2048, 768), (2048, 1000), (2048, 2048)])
def test_cut_tiles(cuda, N, W):
    limbs_in(cuda, N, W)
