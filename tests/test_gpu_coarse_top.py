"""
Which level the one-launch V-cycle of the coarse multigrid levels starts at, and what its limits leave to launches of single
steps: no sweeps at all, a raised limit.
"""
import numpy as np
import pytest

from _util import maxrel

pytestmark = pytest.mark.gpu


def _solve(dtype, nmesh, los=None, sweeps=5, limit=-1):
    import torch as t
    from pyrecon_b200 import _lib as L
    lib, st = L.load(), L.stream_of(t.device('cuda', 0))
    mixed = int(dtype == 'f4')
    delta = t.randn(nmesh, generator=t.Generator(device='cuda').manual_seed(8), device='cuda',
                    dtype=t.float32 if mixed else t.float64)
    phi = t.full_like(delta, float('nan'))
    ws = t.empty(lib.prc_multigrid_batch_workspace_bytes(L.i3(nmesh), 4 if mixed else 8, mixed, 1), dtype=t.uint8, device='cuda')
    L.tune_set('mg_small_cells', 0, limit)
    n0 = L.launch_count()
    try:
        L.call('prc_multigrid_batch_' + L.suffix(dtype), L.pointer_array([delta]), L.pointer_array([phi]), 1, L.i3(nmesh),
               L.d3([800., 700., 900.]), L.d3([1500.] * 3), 0.4, 0.4, sweeps, 6, L.opt_d3(los), *([1] if mixed else []),
               L.ptr(ws), ws.numel(), st)
        t.cuda.synchronize()
    finally:
        L.tune_set('mg_small_cells', 0, -1)
    return phi.cpu().numpy(), L.launch_count() - n0


@pytest.mark.parametrize('dtype', ['f4', 'f8'])
@pytest.mark.parametrize('nmesh,top', [((32, 32, 32), 16**3), ((40, 40, 40), 20**3), ((48, 48, 48), 12**3),
                                       ((96, 96, 96), 12**3), ((80, 24, 32), 80 * 24 * 32 // 8)])
def test_level_that_the_cluster_starts_at(dtype, nmesh, top):
    """The largest level of at most 13824 cells whose planes its blocks hold: of a cube 16^3, 20^3 or, below a mesh of 3 2^k,
    12^3 (24^3 has 1152 pairs of cells a block, 1024 fit)."""
    launches = {limit: _solve(dtype, nmesh, limit=limit)[1] for limit in (-1, top, top - 1)}
    assert launches[-1] == launches[top] < launches[top - 1]


@pytest.mark.parametrize('dtype', ['f4', 'f8'])
@pytest.mark.parametrize('nmesh,sweeps,limit', [((40, 48, 32), 0, -1), ((40, 48, 32), 1, -1), ((20, 12, 24), 0, -1),
                                                ((64, 16, 16), 5, 1 << 14), ((64, 16, 16), 0, 1 << 14),
                                                ((64, 32, 32), 5, 1 << 16)])
def test_cluster_at_its_limits(dtype, nmesh, sweeps, limit):
    fused, n = _solve(dtype, nmesh, sweeps=sweeps, limit=limit)
    steps, single = _solve(dtype, nmesh, sweeps=sweeps, limit=0)
    assert n < single
    if sweeps == 0:
        assert not fused.any() and not steps.any()
    # as test_coarse_levels_dealt_over_a_cluster
    assert np.isfinite(fused).all() and maxrel(fused, steps) < (1e-5 if dtype == 'f4' else 1e-12)
