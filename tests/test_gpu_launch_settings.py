"""Two schedule lengths in turn through one anneal kernel cost the host what one does: the settings of a launch are asked
of the runtime once per layout, not at every change."""
import time

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_alternating_schedules():
    from arpeggio_b200 import _lib
    B, R, D, P, L = 1, 4, 16, 2, _lib.lib()
    z = lambda *s, t=torch.int32: torch.zeros(*s, dtype=t, device='cuda')
    G, h, T, inst, st = z(B, D, D), z(B, D), z(64), z(B), z(1)
    out = z(B, R, P * D, t=torch.int8), z(B, R, t=torch.int64), z(B, R, 2, t=torch.int64)
    ins, ptrs, sp = [_lib.ptr(x) for x in (G, h, T)], [_lib.ptr(x) for x in out], _lib.stream_ptr()

    def call(n):
        _lib.check(L.arp_anneal_first_accept(*ins, n, 0, P, R, D, B, _lib.ptr(inst), 1, 2, 0, *ptrs, _lib.ptr(st), sp),
                   'anneal')

    def host_us(lengths):
        best = 1e9
        for _ in range(20):
            torch.cuda.synchronize()
            t = time.perf_counter()
            for i in range(60):
                call(lengths[i % len(lengths)])
            best = min(best, (time.perf_counter() - t) / 60 * 1e6)
        torch.cuda.synchronize()
        return best

    host_us((64, 48))
    same, turns = host_us((64,)), host_us((64, 48))
    assert turns < 1.5 * same, (same, turns)
