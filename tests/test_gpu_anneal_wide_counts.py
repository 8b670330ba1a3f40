"""Above 64 coordinates the mapping follows the number of anneals a use and in all: two per warp with the last group idle
(31 a use), and one per warp on both sides of each line.  Integers and equal FP32 operations, so equality."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from test_gpu_anneal_group import NTH, _check, _problems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('B,R', [(100, 31), (74, 32), (92, 32), (93, 32), (148, 32), (149, 32), (222, 32), (223, 32),
                                 (149, 64), (222, 64), (223, 64), (80, 33), (300, 28), (300, 29)])
@pytest.mark.parametrize('policy', ['arpeggio', 'chord'])
@pytest.mark.parametrize('D,P', [(65, 2), (96, 4), (97, 2), (128, 4)])
def test_counts(D, P, B, R, policy):
    _check(D, P, B, R, [410, 350, 300, 260], 60, 'rand', policy, [100, 60, 30, 0] if policy == 'chord' else None)


@pytest.mark.parametrize('B,R', [(100, 31), (92, 32), (93, 32), (80, 33)])
@pytest.mark.parametrize('policy', ['arpeggio', 'chord'])
@pytest.mark.parametrize('D,P', [(65, 2), (96, 4), (97, 2), (128, 4)])
def test_counts_float(D, P, B, R, policy):
    from arpeggio_b200 import arpeggiofx
    G, h = (x.astype(np.float32) / np.float32(4096) for x in _problems(D, B, 3))
    inst, key = np.arange(B, dtype=np.int64) + 5, 0x77 + (0x1234 << 32)
    T = np.array([0.1, 0.09, 0.08, 0.07], dtype=np.float32)
    c = np.array([0.03, 0.02, 0.01, 0.0], dtype=np.float32) if policy == 'chord' else None
    ref = O.anneal_dd_f32(G, h, P, R, T, 0.02, inst, key, 'rand', policy, c, nthreads=NTH)
    dev = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()
    s, de, st, status = arpeggiofx.anneal(dev(G.transpose(0, 2, 1)), dev(h), P, R, dev(T), 0.02,
                                          dev(inst.astype(np.int32)), key, 'rand', policy,
                                          None if c is None else dev(c), 'f32')
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    for got, want in zip((s, de, st), ref):
        assert np.array_equal(got.cpu().numpy(), want)
