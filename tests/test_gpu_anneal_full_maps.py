"""The mappings that large batches take, bit for bit against the oracle: anneal counts just above each of the dispatch's
limits, at the edges of each mapping's coordinates, with 32-bit and (a temperature above the stored thresholds' range)
64-bit energies."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from test_gpu_anneal_group import NTH, _check, _problems

pytestmark = pytest.mark.gpu

# (D, P, uses, anneals a use): above 30000 anneals up to 16 coordinates, 10000 up to 32, 37888 up to 64 (four copies and
# fewer); above 64 two per warp past the windows of one per warp
SHAPES = ([(D, P, 910, 33) for D, P in ((1, 2), (8, 2), (15, 4), (16, 2), (16, 6))] +
          [(D, P, 304, 33) for D, P in ((17, 2), (31, 6), (32, 2), (32, 4))] +
          [(D, P, 1149, 33) for D, P in ((33, 2), (40, 4), (48, 2), (48, 4), (49, 2), (63, 4), (64, 2), (64, 4), (64, 6))] +
          [(D, P, 230, 31) for D, P in ((65, 2), (96, 4), (97, 2), (128, 2), (128, 4), (80, 6), (128, 6))])


def _schedule(P, policy, wide):
    T = np.array([410, 350, 300, 260, 230, 200, 180, 150])[:P + 2]
    if wide:
        T[1] = 16384
    c = np.array([100, -60, 30, 0, 20, 10, 0, 0])[:P + 2] if policy == 'chord' else None
    return T, c


@pytest.mark.parametrize('wide', [False, True])
@pytest.mark.parametrize('policy', ['arpeggio', 'chord'])
@pytest.mark.parametrize('D,P,B,R', SHAPES)
def test_integer_maps(D, P, B, R, policy, wide):
    T, c = _schedule(P, policy, wide)
    _check(D, P, B, R, T, 60, 'rand', policy, c)


@pytest.mark.parametrize('policy', ['arpeggio', 'chord'])
@pytest.mark.parametrize('D,P,B,R', SHAPES)
def test_float_maps(D, P, B, R, policy):
    from arpeggio_b200 import arpeggiofx
    G, h = (x.astype(np.float32) / np.float32(4096) for x in _problems(D, B, 3))
    T, c = (None if x is None else x.astype(np.float32) / np.float32(4096) for x in _schedule(P, policy, False))
    inst, key = np.arange(B, dtype=np.int64) + 5, 0x77 + (0x1234 << 32)
    ref = O.anneal_dd_f32(G, h, P, R, T, 0.02, inst, key, 'bal', policy, c, nthreads=NTH)
    dev = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()
    s, de, st, status = arpeggiofx.anneal(dev(G.transpose(0, 2, 1)), dev(h), P, R, dev(T), 0.02,
                                          dev(inst.astype(np.int32)), key, 'bal', policy,
                                          None if c is None else dev(c), 'f32')
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    for got, want in zip((s, de, st), ref):
        assert np.array_equal(got.cpu().numpy(), want)


@pytest.mark.parametrize('D,P,B,R', SHAPES)
def test_chord_rounds_with_a_flip(D, P, B, R):
    from arpeggio_b200 import _lib
    G, h = _problems(D, B, 8)
    T, c = _schedule(P, 'chord', False)
    dev = lambda x: torch.from_numpy(np.ascontiguousarray(x, dtype=np.int32)).cuda()
    s = torch.empty(B, R, P * D, dtype=torch.int8, device='cuda')
    de, n1 = (torch.empty(B, R, dtype=torch.int64, device='cuda') for _ in range(2))
    st = torch.empty(B, R, 2, dtype=torch.int64, device='cuda')
    status = torch.zeros(1, dtype=torch.int32, device='cuda')
    a, p = [dev(x) for x in (G, h, T, c, np.arange(B))], _lib.ptr
    _lib.check(_lib.lib().arp_anneal_chord_dd_n1(p(a[0]), p(a[1]), p(a[2]), p(a[3]), len(T), 60, P, R, D, B, p(a[4]), 3, 4,
                                                 0, p(s), p(de), p(st), p(n1), p(status), _lib.stream_ptr()), 'chord n1')
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    ref = O.anneal_chord_n1(G, h, P, R, T, c, 60, np.arange(B), 3 | (4 << 32), 'rand', nthreads=NTH)
    for got, want in zip((s, de, st, n1), ref):
        assert np.array_equal(got.cpu().numpy(), want)
