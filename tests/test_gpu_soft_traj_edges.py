"""The trajectory sampler's mappings of 24, 48 and 96 coordinates, bit for bit against the oracle at their edges: one chain
(more warps stage J than run chains), and chain counts that leave groups of a warp idle."""
import pytest

import test_gpu_soft_traj_maps as maps

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('M,D', [(16, D) for D in (20, 22, 24, 26, 34, 46, 48, 50)] +
                         [(4, D) for D in (36, 44, 48, 52, 68, 92, 96, 100)])
@pytest.mark.parametrize('R,S', [(1, 9), (5, 6), (33, 7)])
def test_sampler_equals_oracle(M, D, R, S):
    maps.test_sampler_equals_oracle_at_the_mappings_edges(M, D, R, S)
