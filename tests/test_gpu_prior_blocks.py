"""The MAP objective's prior with blocks of 32, 64, 128 and 256 threads (grids on either side
of where the block doubles on 152 SMs: 9 728, 19 456 and 38 912 voxels), as
test_gpu_prior.py has it and with its tolerance.
"""
import pytest

from test_gpu_prior import test_prior_matches_the_scatter as check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(21, 21, 22), (21, 22, 22), (27, 30, 24), (27, 31, 24), (38, 40, 25), (39, 41, 25)])
@pytest.mark.parametrize("p,all_nb,obj", [(2.0, True, True), (1.0, False, True), (1.4, True, True)])
def test_prior_matches_at_every_block_size(gpu, n, p, all_nb, obj):
    check(gpu, n, p, all_nb, obj)
