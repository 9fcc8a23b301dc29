"""MOE_FFN's expert products where there are more tiles than SMs (a CTA walks several tiles, with two accumulators up to 128 rows a run and one beyond) and where the down
product takes 256 rows of its matrix at a time: runs of one and of many rows, experts without any, matrices that end within the second half of a tile, tiles that do not
divide the CTAs.  Reference and tolerance as in the other expert products."""
import pytest

from test_gpu_expert_gemm import test_expert_products as check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts,top,D,ff", [([3, 0, 17, 128] * 15, 1, 520, 520),               # gate and up: 225 tiles, two accumulators; down: 135 of 256 rows
                                             ([3, 0, 17, 129] * 15, 1, 392, 640),               # one accumulator; the last 256 rows hold 8 of the second half
                                             ([1] * 70 + [200], 1, 648, 264),                   # down: 71 runs of three tiles, walked
                                             ([16] * 64, 2, 256, 1160)])
def test_walked_tiles(cuda_backend, counts, top, D, ff):
    check(cuda_backend, counts, top, D, ff)
