"""Warm-started anneals on every lanes x coordinates mapping, bit for bit against the oracle: anneal counts on both sides
of the dispatch's limits that leave groups of a warp idle, sampled starts, per-problem counts that end inside a warp,
and the narrow blocks a caller may set."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from test_gpu_anneal_group import NTH, _problems

pytestmark = pytest.mark.gpu

FEW = [(3, 5), (100, 33), (126, 33), (600, 9)]  # one anneal per warp (two register bounds), the half mappings
SHAPES = ([(D, B, R) for D in (8, 15, 16) for B, R in FEW + [(910, 33)]] +
          [(D, B, R) for D in (17, 32) for B, R in FEW + [(304, 33)]] +
          [(D, B, R) for D in (33, 48, 49, 50, 64) for B, R in FEW + [(1149, 33)]] +
          [(D, 583, 65) for D in (50, 64)] +
          [(D, B, R) for D in (65, 90, 96, 97, 128) for B, R in [(3, 5), (50, 33), (126, 33), (230, 31)]])


@pytest.mark.parametrize('warps', [0, 1, 4])
@pytest.mark.parametrize('D,B,R', SHAPES)
def test_warm_maps(D, B, R, warps):
    from arpeggio_b200 import _lib
    G, h = _problems(D, B, 6)
    rng = np.random.default_rng(D * 64 + R)
    k = np.arange(B) % 7
    perm = np.stack([rng.permutation(D) for _ in range(7)])[k]
    m0 = rng.choice([-2, 0, 2], size=(7, D))[k]
    cdf = np.sort(rng.integers(0, 1 << 32, size=(7, D, 2), dtype=np.uint32), axis=2)[k]
    ra = np.array([1, 3, 5, R, 4, 2, R - 1])[k]
    T, inst, q = [410, 350, 300, 260, 200], np.arange(B) + 3, 11
    dev = lambda x, t=np.int32: torch.from_numpy(np.ascontiguousarray(x, dtype=t)).cuda()
    a = [dev(G), dev(h), dev(T), dev(inst), dev(m0, np.int8), dev(cdf.view(np.int32)), dev(perm, np.uint8), dev(ra)]
    p = _lib.ptr
    L = _lib.lib()
    _lib.check(L.arp_anneal_tune(D, 2, 2, 0, warps), 'tune')
    try:
        for kind in ('mix', 'sampled', 'counted'):
            s = torch.full((B, R, 2 * D), 9, dtype=torch.int8, device='cuda')
            de = torch.empty(B, R, dtype=torch.int64, device='cuda')
            st = torch.empty(B, R, 2, dtype=torch.int64, device='cuda')
            status = torch.zeros(1, dtype=torch.int32, device='cuda')
            head = (p(a[0]), p(a[1]), p(a[2]), len(T), q, 2, R, D, B, p(a[3]), 21, 8, p(a[4]))
            outs = (p(s), p(de), p(st), p(status), _lib.stream_ptr())
            wr = R // 2 if kind == 'mix' else R
            if kind == 'mix':
                rc = L.arp_anneal_first_accept_warm_mix(*head, p(a[6]), wr, *outs)
            else:
                rc = L.arp_anneal_first_accept_warm_sampled(*head, p(a[5]), p(a[6]), wr,
                                                            p(a[7]) if kind == 'counted' else None, *outs)
            _lib.check(rc, kind)
            torch.cuda.synchronize()
            assert int(status.item()) == 0
            ref = O.anneal_dd_warm(G, h, 2, R, T, q, inst, 21 | (8 << 32), m0, perm, nthreads=NTH, warm_r=wr,
                                   cdf=None if kind == 'mix' else cdf, ra=ra if kind == 'counted' else None)
            for got, want in zip((s, de, st), ref):
                assert np.array_equal(got.cpu().numpy(), want), kind
    finally:
        _lib.check(L.arp_anneal_tune(D, 2, 2, 0, 0), 'tune')
