"""Schedules on both sides of what is staged, bit for bit against the oracle."""
import numpy as np
import pytest

from test_gpu_anneal_group import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('policy', ['arpeggio', 'chord'])
@pytest.mark.parametrize('D,P', [(6, 2), (33, 6), (65, 2), (128, 4)])
@pytest.mark.parametrize('L', [1023, 1024, 1025, 2049, 8192, 8193])
def test_long_schedules(D, P, L, policy):
    rng = np.random.default_rng(L)
    T = rng.integers(50, 900, L)
    c = rng.integers(-200, 200, L) if policy == 'chord' else None
    _check(D, P, 3, 3, T, 60, 'rand', policy, c)
