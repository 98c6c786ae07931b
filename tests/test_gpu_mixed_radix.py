"""
The mixed-radix shared-memory passes at the lengths where a tile's lines change (16, 8 or fewer), with odd axes, primes and
axes of a few cells, against numpy's FP64 transform; and the quotients by multiplication that they index with.
"""
import ctypes

import numpy as np
import pytest

from _util import maxrel

# strided passes take 16 lines up to 232 points in FP32 and 116 in FP64; 606 and 1018 = 2 x 509 fewer than 8 in FP64;
# 121 and 509 begin with a prime above 8
SHAPES = [(232, 234, 18), (234, 232, 22), (116, 118, 30), (118, 116, 25), (5, 3, 466), (3, 7, 235), (2, 3, 2),
          (49, 121, 231), (6, 606, 50), (1018, 2, 10), (509, 3, 4), (4, 509, 6)]


def test_quotients_by_multiplication():
    q = np.arange(1 << 16, dtype='u8')
    for d in range(2, 2049):
        m = np.uint64(0xffffffff // d + 1)
        assert np.array_equal((q * m) >> np.uint64(32), q // np.uint64(d))


@pytest.mark.gpu
@pytest.mark.parametrize('nmesh', SHAPES)
@pytest.mark.parametrize('dtype', ['f4', 'f8'])
def test_mixed_radix_passes(nmesh, dtype):
    import torch as t
    import pyrecon_b200
    from pyrecon_b200 import _lib as L
    boxsize = [1000., 1100., 900.]
    noise = np.random.default_rng(37).standard_normal(nmesh).astype(dtype)
    spectrum = np.fft.rfftn(noise.astype('f8'))
    tol = 1e-5 if dtype == 'f4' else 1e-12     # as the other transforms of these kernels against numpy
    mesh = pyrecon_b200.RealMesh(t.from_numpy(noise).cuda(), boxsize=boxsize, boxcenter=0., nmesh=nmesh, dtype=dtype)
    complex_mesh = mesh.to_complex()
    assert maxrel(t.view_as_real(complex_mesh.value).cpu().numpy(), np.stack([spectrum.real, spectrum.imag], axis=-1)) < tol
    assert maxrel(complex_mesh.to_real().value.cpu().numpy(), noise) < tol
    k = [2 * np.pi * np.fft.fftfreq(n, d=b / n) for n, b in zip(nmesh, boxsize)]
    k[2] = k[2][:nmesh[2] // 2 + 1]
    k = np.meshgrid(*k, indexing='ij')
    k2 = sum(x ** 2 for x in k)
    k2[0, 0, 0] = 1.
    lib, v = L.load(), t.from_numpy(noise).cuda()
    psi = t.empty((3,) + tuple(nmesh), dtype=v.dtype, device='cuda')
    ws = t.empty(lib.prc_zeldovich_psi_workspace_bytes(L.i3(nmesh), v.element_size()), dtype=t.uint8, device='cuda')
    L.call('prc_zeldovich_psi_' + L.suffix(dtype), L.ptr(v), L.i3(nmesh), L.d3(boxsize),
           *[ctypes.c_void_p(p.data_ptr()) for p in psi], 1, L.ptr(ws), ws.numel(), L.stream_of(v.device))
    scale = 0.
    refs = []
    for a in range(3):
        ka = k[a].copy()
        if nmesh[a] % 2 == 0:                  # the symmetrised multiplier: zero on the Nyquist index
            index = [slice(None)] * 3
            index[a] = nmesh[a] // 2
            ka[tuple(index)] = 0.
        dk = spectrum * ka / k2
        dk[0, 0, 0] = 0.
        refs.append(np.fft.irfftn(1j * dk, s=nmesh, axes=(0, 1, 2)))
        scale = max(scale, np.abs(refs[-1]).max())
    for a in range(3):
        assert np.abs(psi[a].cpu().numpy() - refs[a]).max() < tol * scale
