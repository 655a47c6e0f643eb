"""Rows of 64 Gaussians on grids above 3072 tiles: the oracle's lists, bit for bit, on either side of the lines
in tiles (4096) and in row counts (3.5 million)."""
import pytest

from tests.test_gpu_binning_rows import test_rows_and_lanes as check_lists

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [0.01, 0.04])
@pytest.mark.parametrize("dims,n", [((144, 128, 96), 64767), ((144, 128, 96), 64768), ((128, 128, 128), 54527),
                                    ((128, 128, 128), 54528), ((121, 122, 123), 63), ((152, 144, 96), 5000)])
def test_lists(dims, n, scale, cuda_device):
    check_lists(dims, n, scale, cuda_device)
