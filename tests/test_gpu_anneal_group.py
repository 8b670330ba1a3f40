"""Anneals with several anneals per warp, bit for bit against the oracle: coordinate counts at the edges of
every lanes x coordinates mapping, anneal counts that leave groups of a warp idle, batches on both sides of the
dispatch's anneal counts, and schedules and coefficients on both sides of the 32-bit energies' range."""
import os

import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu
NTH = max(1, min(16, os.cpu_count() or 1))


def _problems(D, B, seed, gmax=4096, distinct=7):
    """B integer problems (the first `distinct` repeated): symmetric G with a dominant diagonal, h of its size."""
    rng = np.random.default_rng(seed)
    n = min(B, distinct)
    A = rng.normal(size=(n, 2 * D, D)) / np.sqrt(2 * D)
    Q = np.einsum('bki,bkj->bij', A, A)
    s = np.abs(Q).max((1, 2))
    G = np.rint(Q / s[:, None, None] * gmax).astype(np.int32)
    h = np.rint(rng.uniform(-1, 1, size=(n, D)) * gmax).astype(np.int32)
    k = np.arange(B) % n
    return G[k], h[k]


def _check(D, P, B, R, T, q, start, policy, c=None, gmax=4096, seed=0):
    from arpeggio_b200 import arpeggiofx
    G, h = _problems(D, B, seed, gmax)
    inst = np.arange(B, dtype=np.int64) + 77
    key = 0x1234567 + (0x9ABC << 32)
    ref = O.anneal_dd(G, h, P, R, T, q, inst, key, start, policy, c, nthreads=NTH)
    dev = lambda x: torch.from_numpy(np.ascontiguousarray(x, dtype=np.int32)).cuda()
    s, de, st, status = arpeggiofx.anneal(dev(G.transpose(0, 2, 1)), dev(h), P, R, dev(T), q, dev(inst), key, start,
                                          policy, None if c is None else dev(c))
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    for got, want in zip((s, de, st), ref):
        assert np.array_equal(got.cpu().numpy(), want)


SHAPES = ([(D, 2) for D in (1, 8, 15, 16, 17, 32, 33, 48, 49, 63, 64, 65, 96, 97, 128)] +
          [(D, 4) for D in (16, 33, 64, 96, 127)] + [(D, 6) for D in (16, 31, 64, 65, 128)])


@pytest.mark.parametrize('policy', ['arpeggio', 'chord'])
@pytest.mark.parametrize('D,P', SHAPES)
def test_every_mapping_equals_the_oracle(D, P, policy):
    """One anneal per warp (a few uses), and the many-per-warp mappings (a batch above the dispatch's count) with an
    anneal count that leaves lanes of the last group idle; 13 sweeps less one pass, so that the last Philox quad
    and the last sweep are cut short."""
    rng = np.random.default_rng(D * 8 + P)
    T = rng.integers(50, 900, 13 * P - 1)
    c = rng.integers(-200, 200, len(T)) if policy == 'chord' else None
    _check(D, P, 3, 5, T, 60, 'bal', policy, c)
    _check(D, P, 126, 33, T[:5 * P - 1], 60, 'rand', policy, None if c is None else c[:5 * P - 1])


@pytest.mark.parametrize('policy', ['arpeggio', 'chord'])
@pytest.mark.parametrize('D,P', SHAPES)
def test_every_float_mapping_equals_the_oracle(D, P, policy):
    """The FP32 rule is one rounding per operation in a fixed order, so every mapping gives the oracle's bits."""
    from arpeggio_b200 import arpeggiofx
    rng = np.random.default_rng(D * 8 + P)
    T = rng.uniform(0.02, 0.3, 7 * P - 1).astype(np.float32)
    c = rng.uniform(-0.1, 0.1, len(T)).astype(np.float32) if policy == 'chord' else None
    for B, R, start in ((3, 5, 'bal'), (126, 33, 'rand')):
        G, h = (x.astype(np.float32) / np.float32(4096) for x in _problems(D, B, 3))
        inst, key = np.arange(B, dtype=np.int64) + 5, 0x77 + (0x1234 << 32)
        ref = O.anneal_dd_f32(G, h, P, R, T, 0.02, inst, key, start, policy, c, nthreads=NTH)
        dev = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()
        s, de, st, status = arpeggiofx.anneal(dev(G.transpose(0, 2, 1)), dev(h), P, R, dev(T), 0.02,
                                              dev(inst.astype(np.int32)), key, start, policy,
                                              None if c is None else dev(c), 'f32')
        torch.cuda.synchronize()
        assert int(status.item()) == 0
        for got, want in zip((s, de, st), ref):
            assert np.array_equal(got.cpu().numpy(), want)


def test_two_and_four_anneals_per_warp_at_64_coordinates():
    for B in (1148, 1149):  # 33 B on both sides of the two-per-warp mapping's upper count, 8 x 148 x 32
        _check(64, 2, B, 33, [410] * 8, 0, 'rand', 'arpeggio')


@pytest.mark.parametrize('name,T,gmax,D', [
    ('largest stored threshold', [16383] * 10, 4096, 40), ('above it', [16384] * 10, 4096, 40),
    ('a negative temperature', [500, -300, 500, 410], 4096, 40), ('longest staged schedule', [410] * 1024, 4096, 6),
    ('longer', [410] * 1025, 4096, 6), ('energies beyond 32 bits', [1 << 20] * 9, 1 << 18, 128),
    ('energies at the 32-bit bound', [3000] * 9, 16000, 128)])
@pytest.mark.parametrize('policy', ['arpeggio', 'chord'])
def test_schedules_and_coefficients_at_the_range_of_the_32_bit_path(name, T, gmax, D, policy):
    _check(D, 2, 3, 6, T, 17, 'rand', policy, gmax=gmax)


def test_an_unaligned_coupling_equals_the_aligned_one():
    """G one int32 past a 16-byte boundary is staged by 4-byte loads; D = 5 has rows that are never aligned."""
    from arpeggio_b200 import arpeggiofx
    for D in (5, 64):
        G, h = _problems(D, 3, 1)
        dev = lambda x: torch.from_numpy(np.ascontiguousarray(x, dtype=np.int32)).cuda()
        T, inst = dev([410] * 20), dev(np.arange(3))
        Ga = dev(G)
        buf = torch.empty(Ga.numel() + 1, dtype=torch.int32, device='cuda')
        Gu = buf[1:].view_as(Ga)
        Gu.copy_(Ga)
        a = arpeggiofx.anneal(Ga, dev(h), 2, 9, T, 0, inst, 5)
        b = arpeggiofx.anneal(Gu, dev(h), 2, 9, T, 0, inst, 5)
        assert all(torch.equal(x, y) for x, y in zip(a[:3], b[:3]))
