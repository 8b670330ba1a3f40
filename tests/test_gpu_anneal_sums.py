"""Schedules on both sides of what is staged, running energies beyond 32 bits with stored thresholds (four copies above 90
coordinates, six above 60), and the engine's numbers on its small and large mappings, bit for bit against the oracle."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from test_gpu_anneal_group import NTH, _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('policy', ['arpeggio', 'chord'])
@pytest.mark.parametrize('D,P', [(6, 2), (33, 6), (65, 2), (128, 4)])
@pytest.mark.parametrize('L', [1023, 1024, 1025, 2049, 8192, 8193])
def test_long_schedules(D, P, L, policy):
    rng = np.random.default_rng(L)
    T = rng.integers(50, 900, L)
    c = rng.integers(-200, 200, L) if policy == 'chord' else None
    _check(D, P, 3, 3, T, 60, 'rand', policy, c)


def _same(D, P, B, R, T, q, policy, G, h):
    from arpeggio_b200 import arpeggiofx
    inst, key = np.arange(B, dtype=np.int64) + 3, 0x5151 + (0x77 << 32)
    c = np.arange(len(T)) * 7 - 20 if policy == 'chord' else None
    ref = O.anneal_dd(G, h, P, R, T, q, inst, key, 'rand', policy, c, nthreads=NTH)
    dev = lambda x: torch.from_numpy(np.ascontiguousarray(x, dtype=np.int32)).cuda()
    s, de, st, status = arpeggiofx.anneal(dev(G.transpose(0, 2, 1)), dev(h), P, R, dev(T), q, dev(inst), key, 'rand',
                                          policy, None if c is None else dev(c))
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    for got, want in zip((s, de, st), ref):
        assert np.array_equal(got.cpu().numpy(), want)
    return ref[1]


# fields of the largest size whose pass sums still fit: a use's energy falls by them on about half of its P D spins, six
# copies' beyond 32 bits in the kernel's units (a quarter of what it reports); odd uses are small, so that their sums fit 32
# bits in the same launch
@pytest.mark.parametrize('policy', ['arpeggio', 'chord'])
@pytest.mark.parametrize('B,R', [(3, 6), (40, 33), (230, 31)])
@pytest.mark.parametrize('D,P', [(33, 6), (60, 6), (61, 6), (64, 6), (65, 6), (96, 6), (97, 6), (128, 6), (65, 4), (90, 4),
                                 (91, 4), (96, 4), (97, 4), (128, 4), (128, 2)])
def test_energies_beyond_32_bits(D, P, B, R, policy):
    T = np.array([900, 3000, 500, 410, 300, 700, 200])[:P + 1]
    G = np.full((B, D, D), -2, dtype=np.int32)
    h = np.full((B, D), (2 ** 30 - 1) // D - 2 * (2 * P * D + 2), dtype=np.int32)
    h[1::2] = 300
    h[:, ::3] *= -1
    de = _same(D, P, B, R, T, 60, policy, G, h)
    assert P < 6 or np.abs(de[::2]).max() > 4 * 2 ** 31


@pytest.mark.parametrize('D,P', [(8, 2), (16, 4), (17, 2), (32, 6), (33, 4), (64, 2), (64, 6), (96, 2), (128, 4)])
@pytest.mark.parametrize('B,R', [(3, 5), (90, 9), (700, 9)])
def test_engine_numbers(D, P, B, R):
    from arpeggio_b200 import arpeggiofx
    from test_gpu_anneal_group import _problems
    G, h = _problems(D, B, 2)
    T, c = np.array([900, 700, 500, 410, 300]), np.array([10, -30, 0, 20, 5])
    inst, key = np.arange(B, dtype=np.int64) + 9, 0x4242 + (0x99 << 32)
    ref = O.anneal_chord_hw(G, h, P, R, T, c, 60, inst, key, nthreads=NTH)
    dev = lambda x: torch.from_numpy(np.ascontiguousarray(x, dtype=np.int32)).cuda()
    s, de, st, status = arpeggiofx.anneal_engine(dev(G), dev(h), P, R, dev(T), 60, dev(inst), key, dev(c))
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    for got, want in zip((s, de, st), ref):
        assert np.array_equal(got.cpu().numpy(), want)
