"""The training step's products and sums at the edges of their tiles, against float64.

Bounds, from the arithmetic alone: a product's fp32 accumulation makes at most K + 2 roundings (truncations at worst,
2^-23 each) of sums no larger than |A| |B|, its bf16 store one rounding of 2^-8; a column sum makes at most rows
roundings of 2^-24 of sums no larger than the column's absolute sum."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _bf(shape, g):
    return torch.randn(*shape, generator=g).to(torch.bfloat16).cuda()


# one tile; several items per CTA with B kept (K in one to four k tiles, the last ragged) and reloaded (two column
# tiles; more k tiles than the ring holds); ragged rows; narrow N
@pytest.mark.parametrize('M,N,K', [(128, 16, 16), (130, 48, 48), (19200, 256, 16), (19111, 256, 80), (38001, 256, 256),
                                   (19111, 272, 16), (19111, 64, 528), (19111, 16, 256), (19111, 32, 640)])
@pytest.mark.parametrize('b_mn', [0, 1])
@pytest.mark.parametrize('epi', [0, 2, 3, 4])
def test_products(M, N, K, b_mn, epi):
    from arpeggio_b200 import warm
    g = torch.Generator().manual_seed(M + 3 * N + 7 * K + b_mn)
    A, B = _bf((M, K), g), _bf((K, N) if b_mn else (N, K), g)
    bias, aux = torch.randn(N, generator=g).cuda(), _bf((M, N), g)
    Bd = B.double() if b_mn else B.double().t()
    ref = A.double() @ Bd
    tol = (K + 2) * 2.0 ** -23 * (A.double().abs() @ Bd.abs() + bias.double().abs())
    if epi in (2, 3):
        ref = ref + bias.double()
    if epi == 2:
        ref = torch.relu(ref)
    if epi == 4:
        ref = torch.where(aux.double() > 0, ref, 0)
    if epi in (2, 4):
        tol = tol * 1.01 + 2.0 ** -8 * ref.abs()
    ld = N + 8
    C = torch.full((M + 1, ld), -77.0, dtype=torch.bfloat16 if epi in (2, 4) else torch.float32, device='cuda')
    st = torch.zeros(1, dtype=torch.int32, device='cuda')
    warm.gemm(A, 0, K, B, b_mn, N if b_mn else K, M, N, K, epi, C, ld, bias=bias if epi in (2, 3) else None,
              aux=aux if epi == 4 else None, ld_aux=N, status=st)
    torch.cuda.synchronize()
    assert int(st.item()) == 0
    assert bool(((C[:M, :N].double() - ref).abs() <= tol).all())
    assert bool((C[M] == -77).all()) and bool((C[:, N:] == -77).all())


@pytest.mark.parametrize('M,N,K', [(256, 256, 4096), (256, 16, 4096), (384, 80, 1008), (128, 64, 64)])
def test_accumulate(M, N, K):
    from arpeggio_b200 import warm
    g = torch.Generator().manual_seed(M + N + K)
    A, B = _bf((K, M), g), _bf((K, N), g)
    ref = 1 + A.double().t() @ B.double()
    tol = (K + 2) * 2.0 ** -23 * (1 + A.double().abs().t() @ B.double().abs())
    outs = []
    for ws in (None, torch.empty(80 * M * N + 4, device='cuda'), torch.empty(4, device='cuda'), None):
        C = torch.ones(M, N, device='cuda')
        warm.gemm(A, 1, M, B, 1, N, M, N, K, warm.EPI_ACC, C, N, ws=ws)
        outs.append(C)
    torch.cuda.synchronize()
    assert bool(((outs[0].double() - ref).abs() <= tol).all())
    assert all(torch.equal(outs[0], o) for o in outs[1:])  # the same whatever holds the partials


@pytest.mark.parametrize('rows,cols,ld,off', [(1, 8, 8, 0), (5, 8, 16, 0), (129, 24, 24, 0), (4097, 264, 272, 0),
                                              (65536, 256, 256, 0), (70001, 16, 16, 0), (1000, 20, 20, 0),
                                              (1000, 16, 24, 1), (513, 5, 7, 0)])
def test_column_sums(rows, cols, ld, off):
    from arpeggio_b200 import _lib
    g = torch.Generator().manual_seed(rows + cols)
    flat = _bf((rows * ld + 8,), g)
    X = flat[off:off + rows * ld].view(rows, ld)
    part = torch.empty(600 * max(cols, 8), device='cuda')
    outs = []
    for ws in (None, part):
        out = torch.ones(cols, device='cuda')
        _lib.check(_lib.lib().arp_colsum_bf16_ws(_lib.ptr(X), rows, cols, ld, _lib.ptr(out), _lib.ptr(ws),
                                                 0 if ws is None else 4 * ws.numel(), _lib.stream_ptr()), 'colsum')
        outs.append(out)
    torch.cuda.synchronize()
    ref = 1 + X[:, :cols].double().sum(0)
    tol = (rows + 1) * 2.0 ** -24 * (1 + X[:, :cols].double().abs().sum(0))
    assert bool(((outs[0].double() - ref).abs() <= tol).all())
    assert torch.equal(outs[0], outs[1])


@pytest.mark.parametrize('rows,P', [(16, 2), (1008, 4), (20000, 6)])
def test_one_call_step_is_the_steps_one_by_one(rows, P):
    from arpeggio_b200 import warm
    g = torch.Generator().manual_seed(rows)
    X = _bf((rows, 16), g)
    labels = torch.randint(-1, P + 1, (rows,), generator=g).to(torch.int8).cuda()
    a, b = warm.WarmMLP(P=P, seed=3), warm.WarmMLP(P=P, seed=3)
    for _ in range(3):
        a.train_step(X, labels, rows, lr=2e-3)
        b.reserve(rows, train=True)
        b.forward(X, rows)
        b.backward(X, labels, rows)
        b.adam(1.0 / rows, 2e-3)
    torch.cuda.synchronize()
    for k in ('w', 'wb', 'm', 'v', 'grad', 'w2p', 'correct'):
        assert torch.equal(getattr(a, k), getattr(b, k)), k
    torch.testing.assert_close(a.loss, b.loss, rtol=1e-5, atol=0)  # a sum of float atomics
    assert a.steps == b.steps == 3


@pytest.mark.parametrize('rows,classes,ldl,ldd,off', [(1, 2, 5, 3, 0), (255, 3, 16, 16, 0), (1000, 8, 8, 9, 0),
                                                      (513, 7, 16, 16, 1), (257, 5, 12, 24, 0)])
def test_loss(rows, classes, ldl, ldd, off):
    """Softmax cross-entropy and its gradient against float64: __expf is off by at most 2 + 1.2 |x| units in the last
    place, |x| <= 30 here, the quotient and the difference by one each, the bf16 store by 2^-8."""
    from arpeggio_b200 import _lib
    g = torch.Generator().manual_seed(rows)
    z = (torch.rand(rows, ldl, generator=g) * 30 - 15).cuda()
    lab = torch.randint(-1, classes, (rows,), generator=g).to(torch.int8).cuda()
    flat = torch.full((rows * ldd + 8,), 7.0, dtype=torch.bfloat16, device='cuda')
    d = flat[off:off + rows * ldd].view(rows, ldd)
    loss, hits = torch.zeros(1, device='cuda'), torch.zeros(1, dtype=torch.int32, device='cuda')
    _lib.check(_lib.lib().arp_warm_loss(_lib.ptr(z), ldl, _lib.ptr(lab), rows, classes, _lib.ptr(d), ldd,
                                        _lib.ptr(loss), _lib.ptr(hits), _lib.stream_ptr()), 'loss')
    torch.cuda.synchronize()
    zc, use = z[:, :classes].double(), (lab >= 0)
    pr = torch.softmax(zc, 1)
    hot = torch.nn.functional.one_hot(lab.clamp(min=0).long(), classes).double()
    ref = torch.where(use[:, None], pr - hot, 0)
    assert bool(((d[:, :classes].double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 90 * 2.0 ** -23 * pr).all())
    assert bool((d[:, classes:] == 0).all())
    per = torch.where(use, torch.logsumexp(zc, 1) - (zc * hot).sum(1), 0)
    assert abs(loss.item() - per.sum().item()) <= 1e-5 * (per.abs().sum().item() + rows)
    assert int(hits.item()) == int((use & (zc.argmax(1) == lab)).sum())
    assert bool((flat[off + rows * ldd:] == 7).all()) and bool((flat[:off] == 7).all())
