"""
The marched 19-point sweep and residual (mg_march.cuh) against the C oracle at shapes that cut its tiles and slabs:
rows that end inside a segment, segments of 4 to 32 lanes, fewer rows or planes than a tile, several problems.
"""
import ctypes

import numpy as np
import pytest

from oracle import pipeline
from _util import maxrel

pytestmark = pytest.mark.gpu

# all above the size from which the march runs (1.5 MB of v)
SHAPES = [(80, 70, 72), (61, 67, 100), (7, 130, 512), (300, 5, 268), (64, 64, 128), (5, 1100, 76)]


@pytest.mark.parametrize('nmesh', SHAPES)
@pytest.mark.parametrize('dtype', ['f4', 'f8'])
@pytest.mark.parametrize('los', [None, [0.3, -0.5, 0.8]])
def test_march_matches_oracle(nmesh, dtype, los):
    import torch as t
    from pyrecon_b200 import _lib as L
    boxsize, boxcenter, beta = [800., 600., 1000.], [1600., 100., 300.], 0.4
    if los is not None:
        los = list(np.asarray(los) / np.linalg.norm(los))
    rng = np.random.default_rng(17)
    v, f = [rng.standard_normal(nmesh).astype(dtype) for _ in range(2)]
    lib_o = pipeline._Kernels(dtype)._mesh
    ct = np.ctypeslib.as_ctypes_type(np.dtype(dtype))
    arr = lambda a: np.ascontiguousarray(a, dtype=dtype)
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    nn, b, c = np.array(nmesh, dtype='i8'), arr(boxsize), arr(boxcenter)
    lo = None if los is None else arr(los)
    r_ref, vj = np.empty(nmesh, dtype=dtype), v.copy()
    lib_o.oracle_mg_residual(p(v), p(f), p(r_ref), p(nn), p(b), p(c), ct(beta), None if lo is None else p(lo))
    lib_o.oracle_mg_jacobi(p(vj), p(f), p(nn), p(b), p(c), ct(beta), ct(0.4), ctypes.c_int(2), None if lo is None else p(lo))
    dv, df = t.from_numpy(v).cuda(), t.from_numpy(f).cuda()
    r, scratch = t.empty_like(dv), t.empty_like(dv)
    st, los_arg = L.stream_of(dv.device), L.opt_d3(None if lo is None else list(lo))
    args = [L.i3(nmesh), L.d3(boxsize), L.d3(boxcenter), beta]
    L.call('prc_mg_residual_' + L.suffix(dtype), L.ptr(dv), L.ptr(df), L.ptr(r), *args, los_arg, st)
    L.call('prc_mg_jacobi_' + L.suffix(dtype), L.ptr(dv), L.ptr(df), L.ptr(scratch), *args, 0.4, 2, los_arg, st)
    # as test_multigrid_components: a few roundings of ~20 terms
    tol = 1e-12 if dtype == 'f8' else 2e-5
    assert maxrel(r.cpu().numpy(), r_ref) < tol
    assert maxrel(dv.cpu().numpy(), vj) < tol


@pytest.mark.parametrize('dtype', ['f4', 'f8'])
def test_batched_solve_crossing_to_the_march(dtype):
    """Three problems of (48, 64, 64) together are above the size from which the march runs, each alone is below it in
    FP32: the bits of separate solves, whichever kernel ran."""
    import torch as t
    from pyrecon_b200 import _lib as L
    nmesh, count = (48, 64, 64), 3
    lib, st = L.load(), L.stream_of(t.device('cuda', 0))
    mixed = int(dtype == 'f4')
    td = t.float32 if mixed else t.float64
    gen = t.Generator(device='cuda').manual_seed(5)
    deltas = [t.randn(nmesh, generator=gen, device='cuda', dtype=td) for _ in range(count)]
    tail = [L.i3(nmesh), L.d3([800.] * 3), L.d3([1500.] * 3), 0.4, 0.4, 5, 2, L.opt_d3(None)]

    def solve(ds):
        n = len(ds)
        ws = t.empty(lib.prc_multigrid_batch_workspace_bytes(L.i3(nmesh), 4 if mixed else 8, mixed, n), dtype=t.uint8,
                     device='cuda')
        phis = [t.empty_like(d) for d in ds]
        L.call('prc_multigrid_batch_' + L.suffix(dtype), L.pointer_array(ds), L.pointer_array(phis), n, *tail,
               *([1] if mixed else []), L.ptr(ws), ws.numel(), st)
        t.cuda.synchronize()
        return [x.cpu().numpy() for x in phis]

    together = solve(deltas)
    for d, phi in zip(deltas, together):
        assert np.isfinite(phi).all()
        np.testing.assert_array_equal(phi, solve([d])[0])


@pytest.mark.parametrize('dtype', ['f4', 'f8'])
@pytest.mark.parametrize('nmesh,los', [((40, 48, 32), None), ((80, 40, 56), [0.3, -0.5, 0.8]), ((24, 64, 96), [1., 0., 0.]),
                                       ((20, 12, 24), None), ((12, 12, 28), [0., 0., 1.]), ((96, 24, 12), None)])
def test_coarse_levels_dealt_over_a_cluster(dtype, nmesh, los):
    """V-cycles of the coarse levels in one kernel (planes dealt unevenly, levels that stay in one block, rows of four and of
    two) against every step launched by itself (mg_small_cells = 0), for one problem and two."""
    import torch as t
    from pyrecon_b200 import _lib as L
    lib, st = L.load(), L.stream_of(t.device('cuda', 0))
    mixed = int(dtype == 'f4')
    td = t.float32 if mixed else t.float64
    gen = t.Generator(device='cuda').manual_seed(6)
    deltas = [t.randn(nmesh, generator=gen, device='cuda', dtype=td) for _ in range(2)]
    if los is not None:
        los = list(np.asarray(los) / np.linalg.norm(los))
    tail = [L.i3(nmesh), L.d3([800., 700., 900.]), L.d3([1500.] * 3), 0.4, 0.4, 5, 6, L.opt_d3(los)]

    def solve(ds):
        n = len(ds)
        ws = t.empty(lib.prc_multigrid_batch_workspace_bytes(L.i3(nmesh), 4 if mixed else 8, mixed, n), dtype=t.uint8,
                     device='cuda')
        phis = [t.empty_like(d) for d in ds]
        L.call('prc_multigrid_batch_' + L.suffix(dtype), L.pointer_array(ds), L.pointer_array(phis), n, *tail,
               *([1] if mixed else []), L.ptr(ws), ws.numel(), st)
        t.cuda.synchronize()
        return [x.cpu().numpy() for x in phis]

    n0 = L.launch_count()
    fused = solve(deltas)
    n1 = L.launch_count()
    np.testing.assert_array_equal(fused[1], solve(deltas[1:])[0])
    L.tune_set('mg_small_cells', 0, 0)
    try:
        n2 = L.launch_count()
        steps = solve(deltas)
        assert L.launch_count() - n2 > n1 - n0
    finally:
        L.tune_set('mg_small_cells', 0, -1)
    for a, b in zip(fused, steps):
        assert np.isfinite(a).all()
        assert maxrel(a, b) < (1e-5 if dtype == 'f4' else 1e-12)
