"""
The finite-difference shift read-out and the density contrast from smoothed meshes, at the counts where their blocks and
vectors end: single particles, around a block, more than one round of the grid; meshes with and without a remainder of
four cells, aligned and not.
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


@pytest.mark.parametrize('nmesh', [(1, 1, 2), (5, 3, 7), (8, 4, 4), (90, 110, 131)])
@pytest.mark.parametrize('offset', [0, 1])
@pytest.mark.parametrize('in_dtype,dtype', [('f4', 'f4'), ('f8', 'f4'), ('f4', 'f8'), ('f8', 'f8')])
@pytest.mark.parametrize('randoms', [False, True])
def test_delta_from_meshes(nmesh, offset, in_dtype, dtype, randoms):
    import torch as t
    from pyrecon_b200 import _lib as L
    n, bias, ran_min = int(np.prod(nmesh)), 1.7, 0.3
    size = 3. * n        # a tenth of the mean: some cells are masked
    rng = np.random.default_rng(43)
    d, r = [rng.uniform(0., 2., n + offset).astype(in_dtype) for _ in range(2)]
    dd, dr = [t.from_numpy(a).cuda()[offset:] for a in (d, r)]
    d, r = d[offset:].astype('f8'), r[offset:].astype('f8')
    sums = t.tensor([d.sum(), r.sum()], dtype=t.float64, device='cuda')
    out = t.full((n + offset,), np.nan, dtype=t.float32 if dtype == 'f4' else t.float64, device='cuda')[offset:]
    L.call('prc_delta_from_meshes_' + L.suffix(dtype), L.ptr(dd), L.ptr(dr) if randoms else None, dd.element_size(),
           L.ptr(sums), L.i3(nmesh), bias, ran_min, size, L.ptr(out), L.stream_of(out.device))
    if randoms:
        alpha = d.sum() / r.sum()
        ref = np.where(r > ran_min * r.sum() / size, (d - alpha * r) / (bias * alpha * r), 0.)
    else:
        ref = (d / (d.sum() / n) - 1.) / bias
    # a handful of FP64 roundings of values of order one, divided by r >= 0.1; one rounding to the result's type
    np.testing.assert_allclose(out.cpu().numpy(), ref, rtol=1e-6 if dtype == 'f4' else 1e-12,
                               atol=1e-13 if dtype == 'f8' else 1e-9)
