"""A flip-test order that repeats a coordinate: the problem is gathered through it as it stands, whatever ran before.
Energies and counters equal the oracle's on the gathered problem; of the spins, those of coordinates named once."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from test_gpu_anneal_group import NTH, _problems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('B,R', [(6, 5), (126, 33), (1149, 33)])
@pytest.mark.parametrize('D', [8, 15, 32, 48, 64, 90, 128])
def test_repeated_coordinates(D, B, R):
    from arpeggio_b200 import _lib
    G, h = _problems(D, B, 4)
    rng = np.random.default_rng(D)
    perm = np.stack([rng.permutation(D) for _ in range(7)])[np.arange(B) % 7]
    perm[1::2, D // 2] = perm[1::2, 0]  # every other order names one coordinate twice
    perm[3::4] = D - 1                  # and every fourth names one alone
    m0 = rng.choice([-2, 0, 2], size=(B, D)).astype(np.int8)
    T, inst, key = [410, 350, 300, 260], np.arange(B), 9 | (7 << 32)
    ws, de, st = O.anneal_dd_warm(G, h, 2, R, T, 0, inst, key, m0, perm, nthreads=NTH)
    dev = lambda x, t=np.int32: torch.from_numpy(np.ascontiguousarray(x, dtype=t)).cuda()
    s = torch.zeros(B, R, 2 * D, dtype=torch.int8, device='cuda')
    gde = torch.empty(B, R, dtype=torch.int64, device='cuda')
    gst = torch.empty(B, R, 2, dtype=torch.int64, device='cuda')
    status = torch.zeros(1, dtype=torch.int32, device='cuda')
    a = [dev(G), dev(h), dev(T), dev(inst), dev(m0, np.int8), dev(perm, np.uint8)]
    p = _lib.ptr
    _lib.check(_lib.lib().arp_anneal_first_accept_warm(p(a[0]), p(a[1]), p(a[2]), len(T), 0, 2, R, D, B, p(a[3]), 9, 7,
                                                       p(a[4]), p(a[5]), p(s), p(gde), p(gst), p(status),
                                                       _lib.stream_ptr()), 'anneal')
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    assert np.array_equal(gde.cpu().numpy(), de)
    assert np.array_equal(gst.cpu().numpy(), st)
    once = (np.stack([np.bincount(x, minlength=D) for x in perm]) == 1)[:, None, None]
    same = s.cpu().numpy().reshape(B, R, 2, D) == ws.reshape(B, R, 2, D)
    assert (same | ~once).all()
