"""The map's tile shapes (low tiles with a use per block, tall tiles with several) give the same bits for every use: each
use of a batch above the small-batch count against the same use in batches below it, at the edges of every padded
width, with a last block that holds fewer uses, ragged antenna counts and both output types."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _map(L, H, y, s2, M, quant):
    from arpeggio_b200 import _lib
    B, NR2, D = H.shape
    o = [torch.full((B, D, D), 77, dtype=torch.int32, device='cuda'),
         torch.full((B, D), 77, dtype=torch.int32, device='cuda'), torch.zeros(B, D, dtype=torch.int8, device='cuda'),
         torch.zeros(B, device='cuda'), torch.zeros(B, D, device='cuda')]
    st = torch.zeros(1, dtype=torch.int32, device='cuda')
    p = _lib.ptr
    _lib.check(L.arp_map_dd_soft(p(H), p(y), p(s2), B, NR2, D, M, quant, *[p(t) for t in o], p(st), _lib.stream_ptr()),
               'map')
    torch.cuda.synchronize()
    assert int(st.item()) == 0
    return [t.view(torch.int32) if t.dtype == torch.float32 else t for t in o]


@pytest.mark.parametrize('quant', [0, 1])
@pytest.mark.parametrize('nt,nr', [(1, 1), (4, 9), (8, 8), (9, 70), (16, 16), (16, 33), (17, 17), (24, 36), (31, 64),
                                   (32, 32), (33, 40)])
def test_tall_and_low_tiles_give_the_same_bits(nt, nr, quant):
    from arpeggio_b200 import _lib, channel
    L = _lib.lib()
    B = 447  # above the small-batch count; 447 = 3 mod 4 and odd: the last block holds fewer uses
    d = channel.draw_device(100 + nt, torch.linspace(4, 24, B), B, nt, 16, nr=nr)
    H, y = d['H'], d['y']
    s2 = (d['N0'] / 10).float()
    big = _map(L, H, y, s2, 16, quant)
    for a, b in ((0, 200), (200, 447)):
        part = _map(L, H[a:b].contiguous(), y[a:b].contiguous(), s2[a:b].contiguous(), 16, quant)
        for x, w in zip(big, part):
            assert torch.equal(x[a:b], w)
    if nt % 2 == 0:  # an H 4 bytes past a 16-byte boundary takes 4-byte loads
        buf = torch.empty(H.numel() + 1, device='cuda')
        Hu = buf[1:].view_as(H)
        Hu.copy_(H)
        assert all(torch.equal(x, w) for x, w in zip(big, _map(L, Hu, y, s2, 16, quant)))
