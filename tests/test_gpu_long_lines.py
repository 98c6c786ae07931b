"""
FP64 transforms of 1024-point lines, the longest of the register-resident kernels: on the y and x axes their tile of 128-byte
rows does not fit twice in shared memory.  Against numpy's FP64 transform; the local-line-of-sight iteration (its Hessian
pass) against FP32.
"""
import ctypes

import numpy as np
import pytest

from _util import maxrel

pytestmark = pytest.mark.gpu

SHAPES = [(64, 1024, 64), (1024, 64, 64), (8, 1024, 18), (1024, 1024, 8), (16, 16, 2048)]


@pytest.mark.parametrize('nmesh', SHAPES)
@pytest.mark.parametrize('dtype', ['f4', 'f8'])
def test_transforms_of_1024_points(nmesh, dtype):
    import torch as t
    import pyrecon_b200
    noise = np.random.default_rng(47).standard_normal(nmesh).astype(dtype)
    spectrum = np.fft.rfftn(noise.astype('f8'))
    tol = 1e-5 if dtype == 'f4' else 1e-12     # as the other transforms of these kernels against numpy
    mesh = pyrecon_b200.RealMesh(t.from_numpy(noise).cuda(), boxsize=1000., boxcenter=0., nmesh=nmesh, dtype=dtype)
    complex_mesh = mesh.to_complex()
    assert maxrel(t.view_as_real(complex_mesh.value).cpu().numpy(), np.stack([spectrum.real, spectrum.imag], axis=-1)) < tol
    assert maxrel(complex_mesh.to_real().value.cpu().numpy(), noise) < tol
    mesh.smooth_gaussian(20.)
    k = [2 * np.pi * np.fft.fftfreq(n, d=1000. / n) for n in nmesh]
    k[2] = k[2][:nmesh[2] // 2 + 1]
    g = [np.exp(-0.5 * (20. * x) ** 2) for x in k]
    spectrum *= g[0][:, None, None] * g[1][:, None] * g[2]
    assert maxrel(mesh.value.cpu().numpy(), np.fft.irfftn(spectrum, s=nmesh, axes=(0, 1, 2))) < tol


@pytest.mark.parametrize('nmesh', SHAPES[:3])
def test_iteration_along_1024_points(nmesh):
    """One local-line-of-sight iteration, FP64 against FP32 (whose passes on pairs of columns are other kernels)."""
    import torch as t
    from pyrecon_b200 import _lib as L
    lib = L.load()
    delta = np.random.default_rng(53).standard_normal(nmesh)
    psi = {}
    for dtype in ('f4', 'f8'):
        v = t.from_numpy(delta.astype('f4').astype(dtype)).cuda()
        out = t.empty((3,) + tuple(nmesh), dtype=v.dtype, device='cuda')
        w = t.empty(lib.prc_iterative_fft_workspace_bytes(L.i3(nmesh), v.element_size(), 1), dtype=t.uint8, device='cuda')
        L.call('prc_iterative_fft_' + L.suffix(dtype), L.ptr(v), L.i3(nmesh), L.d3([1000., 1100., 900.]),
               L.d3([1800., 300., 700.]), 0.4, None, 2, *[ctypes.c_void_p(p.data_ptr()) for p in out], 1, L.ptr(w),
               w.numel(), L.stream_of(v.device))
        psi[dtype] = out.cpu().numpy()
    # as test_pairs_of_columns
    for a, b in zip(psi['f4'], psi['f8']):
        assert maxrel(a, b) < 5e-6
