"""
The FP32 passes on pairs of columns (fft_duo.cuh) through the entry points that use them, against the FP64 passes (which
take one column a thread) and numpy's FP64 transform on white noise: every line length on x and on y, widths that end on a single column of a tile
and inside one, boxes of unequal sides, a line of sight off the axes.
"""
import ctypes

import numpy as np
import pytest

from _util import maxrel

pytestmark = pytest.mark.gpu

# lines of 64 to 1024 points; nh = 33, 49, 25, 65 columns (tiles of 8 or 16)
SHAPES = [(64, 512, 64), (1024, 64, 96), (128, 512, 48), (512, 128, 64), (256, 256, 128)]


def _run(kind, nmesh, dtype, delta):
    import torch as t
    from pyrecon_b200 import _lib as L
    lib, sfx = L.load(), L.suffix(dtype)
    v = t.from_numpy(delta.astype(dtype)).cuda()
    st, nm, bs, bc = L.stream_of(v.device), L.i3(nmesh), L.d3([1000., 1100., 900.]), L.d3([1800., 300., 700.])
    los = L.d3(list(np.array([0.3, -0.5, 0.8]) / np.linalg.norm([0.3, -0.5, 0.8])))
    psi = t.empty((3,) + tuple(nmesh), dtype=v.dtype, device='cuda')
    out = [ctypes.c_void_p(psi[i].data_ptr()) for i in range(3)]
    ws = lambda n: t.empty(n, dtype=t.uint8, device='cuda')
    if kind == 'psi':
        w = ws(lib.prc_zeldovich_psi_workspace_bytes(nm, v.element_size()))
        L.call('prc_zeldovich_psi_' + sfx, L.ptr(v), nm, bs, *out, 1, L.ptr(w), w.numel(), st)
    elif kind == 'plane_parallel':
        w = ws(lib.prc_plane_parallel_workspace_bytes(nm, v.element_size()))
        L.call('prc_plane_parallel_fft_' + sfx, L.ptr(v), nm, bs, 0.4, los, *out, 1, L.ptr(w), w.numel(), st)
    else:
        local = kind == 'local'
        w = ws(lib.prc_iterative_fft_workspace_bytes(nm, v.element_size(), int(local)))
        L.call('prc_iterative_fft_' + sfx, L.ptr(v), nm, bs, bc, 0.4, None if local else los, 2, *out, 1, L.ptr(w),
               w.numel(), st)
    return psi.cpu().numpy()


@pytest.mark.parametrize('nmesh', SHAPES)
@pytest.mark.parametrize('kind', ['psi', 'plane_parallel', 'local', 'global'])
def test_pairs_of_columns(kind, nmesh):
    delta = np.random.default_rng(29).standard_normal(nmesh).astype('f4')
    single, double = [_run(kind, nmesh, dtype, delta) for dtype in ('f4', 'f8')]
    # up to 8 transforms one after the other, each some 2^-24 sqrt(log2 cells) of the field's rms, over 6 rms of maximum
    for a, b in zip(single, double):
        assert maxrel(a, b) < 5e-6


@pytest.mark.parametrize('nmesh', SHAPES + [(64, 1024, 64)])
def test_pairs_of_columns_gaussian(nmesh):
    import torch as t
    import pyrecon_b200
    boxsize, radius = np.array([1000., 1100., 900.]), 20.
    noise = np.random.default_rng(31).standard_normal(nmesh).astype('f4')
    mesh = pyrecon_b200.RealMesh(t.from_numpy(noise).cuda(), boxsize=boxsize, boxcenter=0., nmesh=nmesh, dtype='f4')
    mesh.smooth_gaussian(radius)
    k = [2 * np.pi * np.fft.fftfreq(n, d=b / n) for n, b in zip(nmesh, boxsize)]
    k[2] = k[2][:nmesh[2] // 2 + 1]
    g = [np.exp(-0.5 * (radius * x) ** 2) for x in k]
    ref = np.fft.rfftn(noise.astype('f8')) * g[0][:, None, None] * g[1][:, None] * g[2]
    assert maxrel(mesh.value.cpu().numpy(), np.fft.irfftn(ref, s=nmesh, axes=(0, 1, 2))) < 5e-6
