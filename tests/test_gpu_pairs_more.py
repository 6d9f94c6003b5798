"""More of tests/test_gpu_pairs.py: sizes and counts on both sides of the lines
between pairs and single radii, NaN barriers in either half of a pair, and
adjoint sweeps of more radii than a lane keeps one sum for."""
import pytest

import test_gpu_pairs as pairs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,nr,batch", [(128, 3, 0), (192, 3, 0), (512, 2, 0), (512, 4, 0), (512, 17, 17), (768, 7, 0),
                                        (1024, 5, 0)])
def test_lines_between_pairs_and_single_radii(N, nr, batch):
    pairs.test_pairs_match_single_radius(N, nr, batch)


@pytest.mark.parametrize("N,nr,batch", [(192, 3, 0), (1024, 3, 0)])
def test_adjoint_lines(N, nr, batch):
    pairs.test_adjoint_pairs_match_single_radius(N, nr, batch)
