"""The readout's block sizes give the same bits: each use of a batch above the small-block count against the same use in
small batches (256-thread blocks), hard and soft, at the edges of the sizes' ranges."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('nt,nr,R,P,M', [(1, 1, 1, 2, 16), (8, 16, 32, 2, 4), (8, 17, 33, 2, 16), (9, 32, 12, 4, 16),
                                         (16, 33, 64, 2, 16), (17, 32, 32, 2, 16), (32, 33, 64, 2, 4), (32, 64, 5, 6, 16),
                                         (16, 16, 65, 2, 16)])
def test_small_blocks_give_the_same_bits(nt, nr, R, P, M):
    from arpeggio_b200 import _lib
    L, p = _lib.lib(), _lib.ptr
    B, D, NR2 = 1187, 2 * nt, 2 * nr
    g = torch.Generator(device='cuda').manual_seed(nt * 100 + R)
    H = torch.randn(B, NR2, D, generator=g, device='cuda')
    y = torch.randn(B, NR2, generator=g, device='cuda') * 3
    hi = {4: 1, 16: 3}[M]
    xq = (2 * torch.randint(0, hi + 1, (B, D), generator=g, device='cuda') - hi).to(torch.int8)
    sp = (2 * torch.randint(0, 2, (B, R, P * D), generator=g, device='cuda') - 1).to(torch.int8)
    n0 = torch.rand(B, generator=g, device='cuda') + 0.5

    def run(a, b, soft):
        n, nb = b - a, D * (1 if M == 4 else 2)
        lv = torch.zeros(n, D, dtype=torch.int8, device='cuda')
        bits = torch.zeros(n, nb, dtype=torch.int8, device='cuda')
        d, pk = torch.zeros(n, device='cuda'), torch.zeros(n, dtype=torch.int32, device='cuda')
        llr = torch.zeros(n, nb, device='cuda')
        keep = [t[a:b].contiguous() for t in (H, y, xq, sp, n0)]
        ins = [p(t) for t in keep[:4]]
        if soft:
            rc = L.arp_readout_llr_dd(*ins, n, NR2, D, P, R, M, p(keep[4]), 50.0, p(lv), p(bits), p(d), p(pk), p(llr),
                                      _lib.stream_ptr())
        else:
            rc = L.arp_readout_dd(*ins, n, NR2, D, P, R, M, p(lv), p(bits), p(d), p(pk), _lib.stream_ptr())
        _lib.check(rc, 'readout')
        torch.cuda.synchronize()
        return lv, bits, d.view(torch.int32), pk, llr.view(torch.int32)
    for soft in (False, True):
        big = run(0, B, soft)
        for a, b in ((0, 600), (600, B)):
            for x, w in zip(big, run(a, b, soft)):
                assert torch.equal(x[a:b], w)
