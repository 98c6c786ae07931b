"""
The quotients by multiplication of the mixed-radix FFT passes (FastDiv) as the device computes them.
"""
import pytest

pytestmark = pytest.mark.gpu


def test_quotients_on_the_device():
    import torch as t
    from pyrecon_b200 import _lib as L
    count = 1 << 16
    out = t.empty((count, 2), dtype=t.int32, device='cuda')
    q = t.arange(count, dtype=t.int32, device='cuda')
    for d in range(1, 2049):
        L.call('prc_debug_quotients', d, count, L.ptr(out), L.stream_of(out.device))
        quotient = t.div(q, d, rounding_mode='floor')
        assert t.equal(out, t.stack([quotient, q - quotient * d], dim=1)), d
    for d, n in [(0, 1), (2049, 1), (2, 0), (2, count + 1)]:
        assert L.load().prc_debug_quotients(d, n, L.ptr(out), L.stream_of(out.device)) == L.PRC_ERR_ARG
