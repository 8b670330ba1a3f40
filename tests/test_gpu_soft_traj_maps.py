"""The trajectory sampler's lane mappings bit for bit against the oracle: spin counts at the edges of each mapping, chain
counts that leave groups of a warp (and warps of a block) idle, and an exploration field other than h0."""
import os

import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu
NTH = max(1, min(16, os.cpu_count() or 1))


@pytest.mark.parametrize('M,D', [(16, D) for D in (2, 14, 16, 18, 30, 32, 34, 62, 64)] +
                         [(4, D) for D in (4, 28, 32, 36, 64, 68, 124, 128)])
@pytest.mark.parametrize('R,S', [(1, 9), (5, 6), (33, 7)])
def test_sampler_equals_oracle_at_the_mappings_edges(M, D, R, S):
    from arpeggio_b200 import _lib
    B, nb = 3, 2 if M == 16 else 1
    N = nb * D
    rng = np.random.default_rng(1000 * D + R)
    J = rng.normal(size=(B, N, N)).astype(np.float32) * np.float32(0.2 / np.sqrt(N))
    J = (J + J.transpose(0, 2, 1)) / 2
    J[:, np.arange(N), np.arange(N)] = 0
    h0, hf = (rng.normal(size=(B, N)).astype(np.float32) * np.float32(0.3) for _ in range(2))
    scale, c0 = rng.uniform(1, 3, B).astype(np.float32), rng.uniform(5, 9, B).astype(np.float32)
    T = rng.uniform(0.05, 0.4, (B, S)).astype(np.float32)
    s0 = np.where(rng.random((B, N)) < 0.5, 1, -1).astype(np.int8) if R == 5 else None
    inst = np.arange(B, dtype=np.uint32) + 9
    key = 0xABCDEF0123
    dev = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()
    ins = [dev(J), dev(hf), dev(h0), dev(scale), dev(c0), dev(T), None if s0 is None else dev(s0)]
    m0, m1 = (torch.empty(B, D * nb, device='cuda') for _ in range(2))
    bd, bl = torch.empty(B, device='cuda'), torch.empty(B, D, dtype=torch.int8, device='cuda')
    it = dev(inst.view(np.int32))
    _lib.check(_lib.lib().arp_soft_trajectory(*[_lib.ptr(x) for x in ins], 0.01, S, R, D, M, B, _lib.ptr(it),
                                              key & 0xFFFFFFFF, key >> 32, _lib.ptr(m0), _lib.ptr(m1), _lib.ptr(bd),
                                              _lib.ptr(bl), _lib.stream_ptr()), 'soft_trajectory')
    torch.cuda.synchronize()
    want = O.soft_trajectory(J, hf, h0, scale, c0, T, s0, 0.01, S, R, D, M, inst, key, nthreads=NTH)
    for got, w in zip((m0, m1, bd, bl), want):
        assert np.array_equal(got.cpu().numpy(), w)
