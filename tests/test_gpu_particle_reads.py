"""
The finite-difference shift read-out at the counts where its blocks end: a single particle, around a block, more than
one round of the grid.
"""
import numpy as np
import pytest

from oracle import pipeline

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('mesh_dtype,pos_dtype', [('f8', 'f8'), ('f8', 'f4'), ('f4', 'f4'), ('f4', 'f8')])
@pytest.mark.parametrize('n', [1, 127, 129, 700001])
def test_finite_difference_shifts_bit_exact(mesh_dtype, pos_dtype, n):
    import torch as t
    from pyrecon_b200 import _lib as L
    geom = pipeline.Geometry((14, 9, 33), 1000., 0., dtype=mesh_dtype)
    rng = np.random.default_rng(41)
    mesh = rng.standard_normal(geom.shape).astype(mesh_dtype)
    pos = rng.uniform(-490., 490., (n, 3)).astype(pos_dtype)
    ref = pipeline._Kernels(mesh_dtype).read_finite_difference_cic(mesh, geom.nmesh, geom.boxsize, geom.to_index(pos))
    m, p = t.from_numpy(mesh).cuda(), t.from_numpy(pos).cuda()
    out, flags = t.full_like(p, np.nan), t.zeros(1, dtype=t.int32, device='cuda')
    L.call('prc_read_shifts_phi_' + L.suffix(mesh_dtype), L.ptr(m), L.i3(geom.nmesh), L.d3(geom.boxsize),
           L.d3(geom.boxcenter), L.ptr(p), p.element_size(), n, None, 0.8, None, 0, 0, 0, L.ptr(out),
           out.element_size(), L.ptr(flags), L.stream_of(m.device), None)
    assert int(flags.item()) == 0
    np.testing.assert_array_equal(out.cpu().numpy(), ref.astype(pos_dtype))
