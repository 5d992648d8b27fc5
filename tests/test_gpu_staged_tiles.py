"""Wide tiles of staged products: stored by whole lines (results at any alignment, last rows of a tile missing), and long sums (in stretches, or split over a cluster)."""
import pytest

from tests import test_gpu_staged_rows as R

pytestmark = pytest.mark.gpu


# one super-block, so that no cluster takes them: results in fours, in twos and single; one row past a tile, a whole one
@pytest.mark.parametrize("m,n", [(129, 40000), (140, 40002), (256, 40001)])
def test_lines_of_plain_rows(runtime, m, n):
    R.test_staged_linear_against_64_bits(runtime, m, 512, n, False)


@pytest.mark.parametrize("m,inter", [(129, 20000), (256, 20001)])
def test_lines_of_gated_rows(runtime, m, inter):
    R.test_staged_gateup_against_64_bits(runtime, m, 512, inter)


# 100 tiles of 11 steps and 112 of 24, whole, in two and three stretches; 40 of 37, whose steps a cluster splits; 184 of 21 on fewer SMs
@pytest.mark.parametrize("m,k,n", [(200, 5632, 12800), (1000, 12288, 3584), (620, 18944, 2048), (1018, 10752, 5888)])
def test_long_sums(runtime, m, k, n):
    R.test_staged_linear_against_64_bits(runtime, m, k, n, False)


def test_long_gated_sums(runtime):
    R.test_staged_gateup_against_64_bits(runtime, 200, 5632, 6400)
